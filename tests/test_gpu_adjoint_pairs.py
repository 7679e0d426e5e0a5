"""The double-word solve's two-cells-per-thread kernels where pairs are cut:
odd and even rows, one cell wide to several blocks."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import strata_fdtd_gb300 as S  # noqa: E402


@pytest.mark.parametrize("shape", [(6, 5, 4), (9, 8, 33), (12, 17, 66), (11, 9, 127), (5, 9, 1), (7, 3, 64)])
def test_double_word_pairs_match_fp64_on_odd_rows(shape):
    """Two cells per thread, whole and half pairs, 16-byte and 8-byte rows: the
    double-word trace, loss and both gradients against the FP64 kernels."""
    n = 40
    out = []
    for dtype in ("dw", torch.float64):
        ds = S.DifferentiableSolver(shape, pml_depth=2 if min(shape) > 4 else 1, frequency=20000.0,
                                    probes=[tuple(v // 3 for v in shape), tuple(v - 1 for v in shape)],
                                    dtype=dtype, checkpoint_every=16)
        g = torch.Generator().manual_seed(5)
        theta = torch.rand(shape, generator=g, dtype=torch.float64).cuda().requires_grad_()
        phi = (0.5 * torch.rand(shape, generator=g, dtype=torch.float64)).cuda().requires_grad_()
        target = (1e-3 * torch.rand((n, 2), generator=g, dtype=torch.float64)).cuda()
        loss = ds.loss(theta, target, n, occupancy=phi)
        loss.backward()
        out.append((float(loss.detach()), theta.grad, phi.grad))
    (l0, t0, p0), (l1, t1, p1) = out
    assert l0 == pytest.approx(l1, rel=1e-11)
    # 40 + 40 steps of operations with |error| <= 3 * 2^-48 relative to their operands
    for a, b in ((t0, t1), (p0, p1)):
        assert float((a - b).abs().max()) <= 1e-10 * float(b.abs().max())


@pytest.mark.parametrize("dtype", ["dw", torch.float64, torch.float32])
@pytest.mark.parametrize("shape", [(8, 7, 12), (9, 8, 33), (10, 6, 1), (9, 8, 11)])
def test_injection_in_the_adjoint_kernel_matches_its_own_launch(dtype, shape):
    """Up to four probes are injected by the adjoint kernel, more by a launch
    between two steps.  Probes whose target is their own trace inject exactly
    zero, so three probes and the same three plus such ones give one gradient:
    equal bits, but for FP32 atomics, which flush subnormals (1e-6)."""
    n = 21
    first = (0, 0, 0)
    probes = [first, tuple(v // 2 for v in shape), tuple(v - 1 for v in shape)]
    if dtype == "dw":
        probes[1] = probes[2]  # two on one cell, added in their order
    more = [(1, 1, 0), (2, 0, 0), (3, 3, 0)]
    g = torch.Generator().manual_seed(7)
    theta = torch.rand(shape, generator=g, dtype=torch.float64)
    target = 1e-3 * torch.rand((n, 3), generator=g, dtype=torch.float64)
    grads = []
    for extra in ([], more):
        ds = S.DifferentiableSolver(shape, pml_depth=1, frequency=20000.0, probes=probes + extra,
                                    dtype=dtype, checkpoint_every=8)
        th = theta.to(ds.ext_dtype).cuda().requires_grad_()
        goal = target.to(ds.ext_dtype).cuda()
        if extra:
            goal = torch.cat([goal, ds.forward(th.detach(), n)[0][:, 3:]], 1)
        ds.loss(th, goal, n).backward()
        grads.append(th.grad)
    a, b = grads
    if max(shape) < 20:  # (in 21 steps the long grid's corners hear nothing yet)
        assert float(b.abs().max()) > 0
    if dtype == torch.float32:
        assert float((a - b).abs().max()) <= 1e-6 * float(b.abs().max())
    else:
        assert torch.equal(a, b)


@pytest.mark.parametrize("nz", [200, 201])
def test_double_word_pairs_match_fp64_in_rows_with_an_open_middle(nz):
    """A row of four blocks: warps that apply all decays, those along k only, and
    none.  The waves pass the blocks' edges at 128 and 192; the bound is that of
    the other rows.  (A long grid's ends hear nothing yet: its values there are
    below FP32's range, within the bound's absolute scale.)"""
    shape, n, out = (8, 11, nz), 40, []
    for dtype in ("dw", torch.float64):
        ds = S.DifferentiableSolver(shape, pml_depth=2, frequency=20000.0, source=(4, 5, 127),
                                    probes=[(3, 5, 130), (5, 8, 123), (4, 2, 127)], dtype=dtype,
                                    checkpoint_every=16)
        g = torch.Generator().manual_seed(5)
        theta = torch.rand(shape, generator=g, dtype=torch.float64).cuda().requires_grad_()
        target = (1e-3 * torch.rand((n, 3), generator=g, dtype=torch.float64)).cuda()
        loss = ds.loss(theta, target, n)
        loss.backward()
        out.append((float(loss.detach()), theta.grad))
    (l0, t0), (l1, t1) = out
    assert l0 == pytest.approx(l1, rel=1e-11)
    assert float(t1.abs().max()) > 1e-12
    assert float((t0 - t1).abs().max()) <= 1e-10 * float(t1.abs().max())


@pytest.mark.parametrize("dtype", ["dw", torch.float64, torch.float32])
@pytest.mark.parametrize("n,every", [(24, 8), (21, 8), (8, 8), (3, 8), (1, 1)])
def test_pressures_kept_by_the_forward_pass_give_the_recomputed_gradient(dtype, n, every, monkeypatch):
    """The last segment's pressures from the forward pass, once, and recomputed
    (a second backward pass; a buffer too large to keep): equal bits in FP64 and
    double words, whose sums have a fixed order, and for FP32 within 1e-6."""
    shape, grads = (9, 8, 12), []
    ds = S.DifferentiableSolver(shape, pml_depth=2, frequency=20000.0, probes=[(4, 4, 4), (6, 3, 7)],
                                dtype=dtype, checkpoint_every=every)
    g = torch.Generator().manual_seed(9)
    theta0 = torch.rand(shape, generator=g, dtype=torch.float64).to(ds.ext_dtype).cuda()
    phi0 = 0.5 * torch.rand(shape, generator=g, dtype=torch.float64).to(ds.ext_dtype).cuda()
    target = (1e-3 * torch.rand((n, 2), generator=g, dtype=torch.float64)).to(ds.ext_dtype).cuda()
    for keep in (True, False):
        if not keep:
            monkeypatch.setattr(type(ds), "_STORE_FRACTION", 0.0)
        theta, phi = theta0.clone().requires_grad_(), phi0.clone().requires_grad_()
        loss = ds.loss(theta, target, n, occupancy=phi)
        for again in (True, False):
            grads.append(torch.autograd.grad(loss, (theta, phi), retain_graph=again))
    for a in grads[1:]:
        for x, y in zip(a, grads[0]):
            if dtype == torch.float32:
                assert float((x - y).abs().max()) <= 1e-6 * float(y.abs().max())
            else:
                assert torch.equal(x, y)
