"""Where the kernels say that the next one may begin, and wait for one that ran ahead: before anything that a small call would wait for first, and in a warp that has nothing else to do."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "luma_b200" / "csrc"


def test_a_decode_launch_lets_the_next_begin_without_a_load():
    body = re.search(r"void __launch_bounds__\([^)]*\) decode_splitk_kernel\(.*?\n\}\n", (CSRC / "decode_splitk.cu").read_text(), re.S).group(0)
    first = body.index("griddepcontrol.launch_dependents")
    condition = re.search(r"if \(!(\w+)\) asm volatile\(\"griddepcontrol.launch_dependents", body).group(1)
    assert re.search(rf"constexpr bool {condition} = [^;]*;", body[:first]) and " a." not in re.search(rf"constexpr bool {condition} = ([^;]*);", body).group(1)


def test_the_prefill_kernel_waits_for_few_rows_in_the_idle_warp():
    body = (CSRC / "prefill_tcgen05.cu").read_text()
    assert body.count("griddepcontrol.wait") == 1
    set_up = body[body.index("// ------------------------------ set-up"):body.index("// ------------------------------ softmax warpgroups")]
    wait = set_up.index("griddepcontrol.wait")
    assert set_up.index("barrier.cta.arrive 1, 96") < set_up.index("barrier.cta.arrive 2, 320") < wait      # behind what the other warps wait for
    assert re.search(r"if \(!kOnePair && a\.behind_few\) asm volatile\(\"griddepcontrol.wait", set_up)
