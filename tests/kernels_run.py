"""The names of the kernels that a call launches, from the profiler's activity
records.  The profiler can drop records, so a kernel that is absent here may
have run; one that is present did."""
import time

import torch


def kernels_run(call):
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA], acc_events=True) as prof:
        time.sleep(0.02)
        for _ in range(3):
            call()
        torch.cuda.synchronize()
        time.sleep(0.02)
    return sorted({e.name for e in prof.events() if e.device_type == torch.autograd.DeviceType.CUDA})


def none_of(names, *kernels):
    return not any(k in n for n in names for k in kernels)
