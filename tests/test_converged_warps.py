"""Loads from tensor memory are instructions of the whole warp: all lanes execute them together. In the prefill kernel's epilogue (csrc/prefill_tcgen05.cu) they stand in loops whose
bodies some lanes leave early, for rows that do not exist, another part's rows or a store that one lane issues; CUDA does not promise that the lanes meet again at a loop's
end. Read from the source: each such load has a __syncwarp() directly before it, or another load that has."""
from pathlib import Path

SOURCE = (Path(__file__).resolve().parent.parent / "luma_b200" / "csrc" / "prefill_tcgen05.cu").read_text()


def test_loads_of_the_epilogue_are_made_by_a_converged_warp():
    lines = [x.strip() for x in SOURCE[SOURCE.index("// epilogue: O_t is final"):SOURCE.index("// ---- host side")].splitlines()]
    loads = [i for i, x in enumerate(lines) if x.startswith("tc_ld32(")]
    assert len(loads) >= 4
    for i in loads:
        assert lines[i - 1].startswith(("__syncwarp();", "tc_ld32(")), lines[i - 1:i + 1]
