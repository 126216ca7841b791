"""Launch shapes: small and large launches of the same kernels agree.

The plain engine's shapes (leaves per P2M and near-field block, direct or tiled L2L)
add every output's terms in the same order, so a right-hand side alone and inside a
batch that takes the larger shapes must agree bit for bit.  The tensor engine's
near-field items (8, 16 or 32 leaf rows) and translations are compared with the plain
engine at the tolerance of its split products."""
import math

import pytest

pytestmark = pytest.mark.gpu

import isg  # noqa: E402


def _rand(n, U, seed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.complex(torch.randn(n, U, generator=g, device="cuda"), torch.randn(n, U, generator=g, device="cuda"))


# 64 leaves per RHS: 2 x 2-leaf blocks alone, 4 x 4 at 20, 4 x 8 from 65, the largest P2M
# blocks from 257, the tiled L2L from 138 (4352 outputs each)
@pytest.mark.parametrize("nrhs", [17, 20, 47, 65, 257, 305])
def test_plain_shapes_agree_bit_for_bit(nrhs):
    import torch
    s = isg.Solver(4, numrx=24, max_rhs=nrhs, device=0)
    x, g = _rand(nrhs, s.numunk, 1), 3.0 * _rand(1, s.numunk, 2)[0]
    for herm in (False, True):
        y = s.matvec(x, g, hermitian=herm)
        for j in (0, nrhs // 2, nrhs - 1):
            assert torch.equal(y[j], s.matvec(x[j], g, hermitian=herm))
    rx, r = s.aggregate(x), _rand(nrhs, 24, 3)
    xh = s.aggregateh(r)
    for j in (0, nrhs - 1):
        assert torch.equal(rx[j], s.aggregate(x[j]))
        assert torch.equal(xh[j], s.aggregateh(r[j]))


# grids of 4, 8, 16 and 32 leaf rows; items of 8 rows while all of them fit the GPU at once,
# then 16, then 32
@pytest.mark.parametrize("level,nrhs", [(3, 1), (4, 3), (5, 5), (5, 40), (6, 1), (6, 10), (6, 21)])
def test_tensor_near_field_items_match_the_plain_engine(level, nrhs):
    import torch
    s = isg.Solver(level, max_rhs=nrhs, device=0)
    x, g = _rand(nrhs, s.numunk, 4), _rand(nrhs, s.numunk, 5)
    for herm in (False, True):
        for gg in (g, g[0]):
            for order in (isg.ORDER_TREE, isg.ORDER_BLOCKED, isg.ORDER_RASTER):
                a = s.matvec(x, gg, hermitian=herm, order=order, engine=isg.ENGINE_TENSOR)
                b = s.matvec(x, gg, hermitian=herm, order=order)
                # 3xFP16 split products: 2^-22 per term against FP32's 2^-24, both over ~650 terms
                assert torch.linalg.norm(a - b) <= 1e-5 * torch.linalg.norm(b)
    # the dot products of every item reach the solver's scalars
    chi = 0.05 * torch.rand(s.numunk, device="cuda")
    gs, u = ((2 * math.pi) ** 2 * chi).to(torch.complex64), torch.zeros_like(x)
    info = s.bicgs(u, gs, x, engine=isg.ENGINE_TENSOR, tol=1e-5)
    assert all(i["status"] == 0 and i["true_residual"] <= 1e-5 for i in info), info


# L2L items of 8, 16 and 32 parents on parent grids of 4, 8 and 16 rows (64 leaves: at most 16
# parents), M2M of the same grids, the SIMT M2M for the coarse levels up to 140000 outputs
@pytest.mark.parametrize("level,nrhs", [(4, 1), (4, 73), (4, 149), (5, 2), (5, 19), (5, 37), (5, 75), (6, 5), (6, 33)])
def test_tensor_translations_match_the_plain_engine(level, nrhs):
    import torch
    s = isg.Solver(level, max_rhs=nrhs, device=0)
    x = _rand(nrhs, s.numunk, 8)
    for conj in (False, True):
        a, b = s.mlfma(x, conj=conj, engine=isg.ENGINE_TENSOR), s.mlfma(x, conj=conj)
        # the field of a unit input is a sum of ~650 split products of 2^-22 each
        for j in range(nrhs):
            assert torch.linalg.norm(a[j] - b[j]) <= 1e-5 * torch.linalg.norm(b[j])


# row pairs aligned to 16 bytes or not (odd receiver counts), one and two accumulator sets,
# one or two batches of 128
@pytest.mark.parametrize("nrhs,numrx", [(1, 16), (5, 33), (64, 130), (65, 40), (131, 7)])
def test_near_receivers_do_not_depend_on_the_order(nrhs, numrx):
    import torch
    s = isg.Solver(4, numrx=numrx, max_rhs=nrhs, device=0)
    s.set_nearfield_receivers(8.0)
    x, r = _rand(nrhs, s.numunk, 6), _rand(nrhs, numrx, 7)
    xb = s.reorder(x, isg.ORDER_RASTER, isg.ORDER_BLOCKED)
    xt = s.reorder(x, isg.ORDER_RASTER, isg.ORDER_TREE)
    want = s.receive(xb, order=isg.ORDER_BLOCKED)
    assert torch.equal(s.receive(x, order=isg.ORDER_RASTER), want)
    assert torch.equal(s.receive(xt, order=isg.ORDER_TREE), want)
    back = s.receiveh(r, order=isg.ORDER_BLOCKED)
    assert torch.equal(s.receiveh(r, order=isg.ORDER_RASTER), s.reorder(back, isg.ORDER_BLOCKED, isg.ORDER_RASTER))
    assert torch.equal(s.receiveh(r, order=isg.ORDER_TREE), s.reorder(back, isg.ORDER_BLOCKED, isg.ORDER_TREE))
    # <go x, r> = <x, gh r>
    a, b = torch.vdot(want.reshape(-1), r.reshape(-1)), torch.vdot(xb.reshape(-1), back.reshape(-1))
    assert abs(a - b) <= 1e-4 * torch.linalg.norm(want) * torch.linalg.norm(r)
    # a vector that starts 8 bytes past a 16-byte boundary takes the scalar loads
    buf = torch.zeros(nrhs * s.numunk + 1, dtype=torch.complex64, device="cuda")
    buf[1:] = x.reshape(-1)
    assert torch.equal(s.receive(buf[1:].view(nrhs, -1), order=isg.ORDER_RASTER), want)
