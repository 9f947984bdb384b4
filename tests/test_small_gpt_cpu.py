"""dgpt_small_gpt without a GPU: rules on the host, and what can be told from its source."""

import os
import re

import diff_gpt_b200

CSRC = os.path.join(os.path.dirname(diff_gpt_b200.__file__), "csrc")


def test_threads_leave_the_step_loop_by_one_answer():
    """A thread that left by its own reading of `stuck`, which the loading warp may raise at any time, would leave others at a barrier of 256 threads
    for good.  (Not shown by running it: that would hang a GPU.)"""
    kernel = open(os.path.join(CSRC, "small_gpt.cuh")).read().split("small_gpt_kernel(")[1]
    loop = kernel[kernel.index("for (int it = 0; it < p.n_steps; ++it)") : kernel.index("if (stuck && tid == 0)")]
    assert re.findall(r"if \((\w+)\) break;", loop) == ["lost", "lost"]
    assert [line.strip() for line in loop.splitlines() if "stuck" in line] == ["lost = sg_any(stuck);"]
