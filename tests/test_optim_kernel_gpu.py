"""The flat clip + Adam kernels: lengths that are no multiple of their vectors, and the guard behind the end (GPU)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4, 1023, 4096 * 1184 + 2])
def test_adam_tail_and_norm(n):
    from scaffold_b200.ops import _lib
    import scaffold_b200.ops.optim  # noqa: F401  (registers the entry points)
    gen = torch.Generator(device="cuda").manual_seed(n % 97)
    p, g, m = (torch.randn(n + 4, generator=gen, device="cuda") for _ in range(3))
    v = torch.rand(n + 4, generator=gen, device="cuda")
    q, mm, vv = (t.double() for t in (p, m, v))
    lib, s = _lib.lib(), _lib.stream_ptr()
    part = torch.zeros(lib.sb_opt_blocks(n), device="cuda")
    norm = torch.zeros(1, device="cuda")
    assert lib.sb_grad_norm(g.data_ptr(), n, part.data_ptr(), norm.data_ptr(), s) == 0
    ref = g[:n].double().norm()
    assert abs(float(norm) - float(ref)) <= 1e-5 * float(ref)
    assert lib.sb_adam_step(p.data_ptr(), g.data_ptr(), m.data_ptr(), v.data_ptr(), n, 1e-2, 0.9, 0.999, 1e-8, 3, 1.0,
                            norm.data_ptr(), 1.0, s) == 0
    gi = g.double() * min(1.0, 1.0 / (float(norm) + 1e-6))
    mm[:n] += (gi[:n] - mm[:n]) * 0.1
    vv[:n] = vv[:n] * 0.999 + gi[:n] ** 2 * 0.001
    q[:n] -= 1e-2 / (1 - 0.9 ** 3) * mm[:n] / ((vv[:n] ** 0.5) / (1 - 0.999 ** 3) ** 0.5 + 1e-8)
    # fp32 arithmetic of a dozen roundings; 1 - 0.999f carries 5e-5 of relative error into the second moment's increment
    torch.testing.assert_close(m.double(), mm, rtol=2e-6, atol=1e-6)
    torch.testing.assert_close(v.double(), vv, rtol=1e-4, atol=1e-6)
    assert torch.equal(p[n:].double(), q[n:])  # nothing behind the end is touched
    assert ((p[:n].double() - q[:n]).abs() <= 2e-6 * q[:n].abs() + 1e-4 * (q[:n] - p[:n].double()).abs() + 5e-6
            * (1 + (mm[:n] / vv[:n] ** 0.5).abs())).all()


@pytest.mark.parametrize("n", [1, 5, 70001])
def test_adam_on_buffers_off_the_vectors_alignment(n):
    """As on aligned ones, but for the multiply-adds that the compiler fuses in one loop and not in the other: each
    moment has two of them and the parameter one more, of terms below 1 (2^-24 each); the step's quotient carries the
    moments' relative errors, 4 roundings of 2^-24, times a step of at most 0.2."""
    from scaffold_b200.ops import _lib
    import scaffold_b200.ops.optim  # noqa: F401  (registers the entry points)
    gen = torch.Generator(device="cuda").manual_seed(n)
    bufs = [torch.rand(n, generator=gen, device="cuda") for _ in range(4)]
    lib, s = _lib.lib(), _lib.stream_ptr()
    outs = []
    for shift in (0, 1):
        own = [torch.full((n + 2,), 7.0, device="cuda") for _ in bufs]
        views = [o[shift:shift + n].copy_(b) for o, b in zip(own, bufs)]
        p, g, m, v = (t.data_ptr() for t in views)
        assert lib.sb_adam_step(p, g, m, v, n, 1e-2, 0.9, 0.999, 1e-8, 3, -1.0, None, 1.0, s) == 0
        torch.cuda.synchronize()
        assert all((o[:shift] == 7).all() and (o[shift + n:] == 7).all() for o in own)
        outs.append([t.clone() for t in views])
    for a, b in zip(*outs):
        torch.testing.assert_close(a, b, rtol=0, atol=2 ** -21)
