"""Which kernels of the package a call launches, for tests of what a launcher chooses."""
import re

import torch


def launched(run, pattern):
    """The parts of the launched kernels' names (template arguments included) that ``pattern`` matches, after a first call by itself."""
    run()
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA], acc_events=True) as p:
        run()
        torch.cuda.synchronize()
    found = (re.search(pattern, e.name) for e in p.events())
    return {m.group(0) for m in found if m}
