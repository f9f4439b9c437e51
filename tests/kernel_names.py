"""Names of the kernels that a stretch of code launches, for tests of which launch a call
takes.  Of direct launches only: for a replayed graph the profiler can report the names of
one that has been destroyed."""
import re
from collections import Counter

import pytest


def launched(run):
    """Counter of kernel names ("sweep_rb_pipe_kernel<float>") of what run() launches."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    torch.zeros(1, device="cuda")
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        run()
        torch.cuda.synchronize()
    names = Counter()
    for e in prof.events():
        m = re.match(r"(?:void )?amcfd::(\w+(?:<[^>(]*>)?)\(", e.name)
        if m:
            names[m.group(1)] += 1
    if not names:
        pytest.skip("the profiler reports no kernels here")
    return names
