"""Names of the kernels a call launches."""
_warm = []


def launched(fn):
    """The kernel names that fn() launches, as one text (profiler activity records)."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    def run(f):
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA, ProfilerActivity.CPU]) as prof:
            f()
            torch.cuda.synchronize()
        return "\n".join(e.name for e in prof.events() if e.device_type == torch.autograd.DeviceType.CUDA)

    if not _warm:  # a process's first profile comes back empty
        x = torch.zeros(1, device="cuda")
        run(lambda: x.add_(1))
        _warm.append(True)
    names = run(fn)
    assert names, "no kernel recorded"
    return names
