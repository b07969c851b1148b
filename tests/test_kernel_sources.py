"""Rules of the kernels' sources that no run shows reliably (CPU)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mestrado_gb300", "csrc")


def test_tensor_memory_is_taken_and_freed_by_converged_warps():
    """tcgen05.alloc and .dealloc are .sync.aligned: every lane of the warp must run them together, and one lane may
    come from a set-up or a wait of its own. A __syncwarp() stands directly before each."""
    seen = 0
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, name)) as f:
            lines = f.read().split("\n")
        for i, line in enumerate(lines):
            if re.search(r'asm volatile\("tcgen05\.(alloc|dealloc)', line):
                seen += 1
                assert lines[i - 1].strip().startswith("__syncwarp();"), f"{name}:{i + 1}"
    assert seen >= 6


def test_the_candidate_tally_is_cleared_a_barrier_before_it_is_set():
    """coarse_cand_select_kernel: a thread that marks the tally while another still clears it loses the mark, and a query
    with missing survivors would not fall back to all centroids."""
    with open(os.path.join(CSRC, "coarse_filter.cu")) as f:
        text = f.read()
    clear = text.index("if (tid < 3) tally[tid] = 0;")
    mark = text.index("tally[2] = 1;")
    assert clear < mark and "__syncthreads" in text[clear:mark]
