"""Names of the kernels that a call launches, as torch's profiler reports them."""


def kernel_names(torch, call):
    """(names, what the call returned); names is None where the profiler reports no
    kernel at all: a session of a few microseconds may come back empty, and in a
    process of many contexts all of them may."""
    from torch.profiler import ProfilerActivity, profile
    for _ in range(10):
        with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as p:
            out = call()
            torch.cuda.synchronize()
        names = " ".join(e.key for e in p.key_averages())
        if "cfd::" in names:
            return names, out
    return None, out
