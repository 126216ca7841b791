"""The launch-shape autotuner: it picks one of the candidate shapes per level,
and the operator's output does not depend on the choice (the same terms of every
output in the same order)."""
import numpy as np
import pytest

import isg
from _oracle import Oracle, disk_contrast

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", [isg.ENGINE_SIMT, isg.ENGINE_TENSOR])
def test_autotune_keeps_the_operator(engine):
    import torch
    s = isg.Solver(6, numrx=16, max_rhs=8, device=0)
    s.setup_gpu()
    o = Oracle(6, numrx=16)
    g = torch.from_numpy(disk_contrast(o.pos(), radius=4.0, chi=0.4).astype(np.complex64)).cuda()
    rng = np.random.default_rng(3)
    x = torch.from_numpy((rng.normal(size=(8, s.numunk)) + 1j * rng.normal(size=(8, s.numunk))).astype(np.complex64)).cuda()
    before = s.matvec(x, g, engine=engine).cpu().numpy()
    got = s.autotune(8, engine)
    assert all(v in (1, 2, 4, 8, 16, 32, 64) for v in got["m2l_rows"][2:])
    assert all(v in (32, 64) for v in got["l2l_cols"][3:])
    assert all(v in (32, 64) for v in got["m2m_cols"][2:-1])
    assert got["near_pair"] in ((1, 2) if engine == isg.ENGINE_TENSOR else (0,))
    after = s.matvec(x, g, engine=engine).cpu().numpy()
    assert np.linalg.norm(after - before) / np.linalg.norm(before) < 1e-5
    info = s.bicgs(torch.zeros_like(x), g, x, tol=1e-5, engine=engine)
    assert all(i["status"] == 0 and 0 <= i["true_residual"] <= 1e-5 for i in info)


def test_levels_of_the_direct_l2l_keep_the_built_in_columns():
    """Up to 600000 outputs a level L2L has no columns per block to choose: a tuned context
    keeps the built-in 64 for the larger batches that do."""
    s = isg.Solver(6, numrx=16, max_rhs=8, device=0)
    s.setup_gpu()
    for nrhs in (1, 2, 4):
        assert s.autotune(nrhs, isg.ENGINE_SIMT)["l2l_cols"][3:] == [64, 64, 64]


def test_tuned_near_field_items_apply_to_the_operator():
    """The tuner times the near-field kernel that the operator launches: where the launch's
    items are small in any case the choice stays 2, and tuning leaves every bit alone."""
    import torch
    s = isg.Solver(7, numrx=16, max_rhs=12, device=0)
    s.setup_gpu()
    x = torch.randn(12, s.numunk, dtype=torch.complex64, device="cuda", generator=torch.Generator("cuda").manual_seed(5))
    g = torch.full((s.numunk,), 0.3, dtype=torch.complex64, device="cuda")
    before = s.matvec(x, g, engine=isg.ENGINE_TENSOR)
    for nrhs in (1, 2, 4):  # 64 and 128 items of 8 rows, 128 of 16: one per SM
        assert s.autotune(nrhs, isg.ENGINE_TENSOR)["near_pair"] == 2
    s.autotune(12, isg.ENGINE_TENSOR)
    assert torch.equal(s.matvec(x, g, engine=isg.ENGINE_TENSOR), before)
