"""The double-word solve's two-cells-per-thread kernels where pairs are cut:
odd and even rows, one cell wide to several blocks."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import strata_fdtd_gb300 as S  # noqa: E402


@pytest.mark.parametrize("shape", [(6, 5, 4), (9, 8, 33), (12, 17, 66), (11, 9, 127), (5, 9, 1), (7, 3, 64),
                                   (8, 11, 201), (8, 11, 200)])
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
