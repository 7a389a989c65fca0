"""Names of the CUDA kernels that a call launches."""
import re

import torch
from torch.profiler import ProfilerActivity, profile


def launched(call):
    """{kernel without its namespace, return type and arguments, e.g. eriSplitKernel<0,0,0,0,double>: launches}."""
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as p:
        call()
        torch.cuda.synchronize()
    names = {}
    for e in p.events():
        m = re.search(r"(\w+Kernel\w*)(<[^>(]*>)?", e.name)
        if m:
            name = m[1] + (m[2] or "").replace(" ", "")
            names[name] = names.get(name, 0) + 1
    return names
