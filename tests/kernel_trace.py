"""The names of the kernels a call launches, as the CUDA activity trace gives them (launches that find no
work among them)."""
import re


def kernels(fn, library=False):
    """Names without arguments of the kernels fn() launches (library: and those of the sorts and scans); None
    where the trace is not to be had."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    for _ in range(2):  # a process's first trace may come back empty
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            fn()
            torch.cuda.synchronize()
        names = [re.sub(r"^void ", "", e.name).replace("(anonymous namespace)::", "").split("(")[0] for e in p.events()]
        names = [n.replace("bwacuda::", "").strip() for n in names
                 if "bwacuda::" in n or (library and n.startswith("cub::"))]
        if names:
            return names
    return None
