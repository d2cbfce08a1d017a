"""The prefill kernel's division of registers between its warpgroups, read from the source (csrc/prefill_tcgen05.cu): every warp of a warpgroup
executes the same setmaxnreg instruction (another one in the same warpgroup is undefined behaviour, whatever its count), and the shares are no more than the
registers that the block was launched with (a request beyond them waits for good)."""
import re
from pathlib import Path

SOURCE = (Path(__file__).resolve().parent.parent / "luma_b200" / "csrc" / "prefill_tcgen05.cu").read_text()


def test_one_setmaxnreg_to_a_warpgroup_and_no_more_than_the_launch_has():
    down = [int(x) for x in re.findall(r'asm volatile\("setmaxnreg\.dec\.sync\.aligned\.u32 (\d+);', SOURCE)]
    up = [int(x) for x in re.findall(r'asm volatile\("setmaxnreg\.inc\.sync\.aligned\.u32 (\d+);', SOURCE)]
    threads = int(re.search(r"constexpr int kThreads = (\d+);", SOURCE).group(1))
    assert len(down) == 1 and len(up) == 1
    launched = 65536 // threads // 8 * 8       # one block to an SM: the compiler's limit, in steps of eight
    assert 128 * down[0] + (threads - 128) * up[0] <= threads * launched
