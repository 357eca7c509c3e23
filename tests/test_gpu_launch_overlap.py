"""Kernels that read what the kernel right before them wrote, back to back and with other data every time: the same bits as
with a synchronisation after each."""
import pytest

pytestmark = pytest.mark.gpu


def test_each_kernel_sees_the_results_of_the_one_before():
    import torch
    import __graft_entry__ as ge
    ge.load_package()
    from polarai_framework_b200.device_builtins import DeviceBuiltins
    d = DeviceBuiltins()
    g = torch.Generator(device="cuda").manual_seed(1)
    new = lambda *s: torch.empty(s, device="cuda")  # noqa: E731
    base = new(512, 512).uniform_(-1, 1, generator=g)
    kernel, narrow = new(5, 5).uniform_(-1, 1, generator=g), new(512, 10).uniform_(-1, 1, generator=g)

    def step(scale, wait):
        out = {"x": new(512, 512), "conv": new(508, 508), "wide": new(508, 510), "pool": new(254, 254), "flat": new(254, 254),
               "turned": new(512, 512), "few_terms": new(512, 512), "split": new(512, 10), "rows": new(512, 10), "sum": new(512, 10)}
        for call in (lambda: d.fadd(base, scale, base, 0.0, out["x"]), lambda: d.fconv2d(out["x"], kernel, out["conv"]),
                     lambda: d.fpool(out["conv"], (2, 2), (2, 2), out["pool"]), lambda: d.fsoftmax(out["pool"], out["flat"]),
                     lambda: d.fadd(base, -scale, base, 0.0, out["x"]), lambda: d.ftranspose(out["x"], out["turned"]),
                     lambda: d.fconv2d(out["turned"], kernel[:, 1:4].contiguous(), out["wide"]),
                     lambda: d.fmatmul(1, 0, out["turned"], narrow, out["split"]), lambda: d.fmatmul(0, 0, out["turned"], narrow, out["rows"]),
                     lambda: d.fadd(out["split"], 1.0, out["rows"], 1.0, out["sum"]),
                     lambda: d.fmatmul(0, 1, out["sum"], out["rows"], out["few_terms"])):
            call()
            if wait:
                torch.cuda.synchronize()
        return out

    step(1.0, True)
    scales = [0.01 * i for i in range(1, 61)]
    together = [step(s, False) for s in scales]
    torch.cuda.synchronize()
    for s, got in zip(scales, together):
        want = step(s, True)
        for name in want:
            assert torch.equal(got[name], want[name]), (s, name)
