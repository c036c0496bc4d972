"""Multigrid at the edges of its loops (no cycle, no smoothing before or after,
a tolerance met at once, one patch, a launch's tail) against the CPU oracle, at
every ghost size (needs a B200).  Fields and cycle counts are the oracle's bit
for bit; the error estimate sums in another order: 2^-53 times the number of
cells, rounded up to 1e-12."""
import numpy as np
import pytest

from gpg.abi import GPG_MG, default_params
from gpg.inputs import make_patches

pytestmark = pytest.mark.gpu

LOOPS = [dict(mg_max_iter=0), dict(mg_max_iter=1, mg_npre_smooth=0), dict(mg_max_iter=2, mg_npost_smooth=0),
         dict(mg_max_iter=3, mg_npre_smooth=0, mg_npost_smooth=0, mg_tolerated_error=0.0),
         dict(mg_max_iter=2, mg_npre_smooth=1, mg_npost_smooth=2, mg_tolerated_error=0.0, dh=0.7)]


@pytest.mark.parametrize("rs", [4, 8])
@pytest.mark.parametrize("g", [1, 2, 3, 4, 5])
def test_mg_loops_match_the_oracle(rs, g):
    torch = pytest.importorskip("torch")
    from gpg.lib import solve_device
    from oracle.oracle import run_oracle
    dev = torch.device("cuda:0")
    for n, kw in zip((1, 7, 31, 150, 12), LOOPS):
        d = make_patches(n, g, seed=80 + g, dtype=np.float32 if rs == 4 else np.float64)
        p = default_params(rs, g, GPG_MG, **kw)
        t = {k: torch.from_numpy(d[k].copy()).to(dev) for k in ("rho", "pot_in", "flu")}
        pot, flu, it, err = solve_device(p, t["rho"], t["pot_in"], flu=t["flu"])
        op, of, oi, oe = run_oracle(p, d["rho"], d["pot_in"], flu=d["flu"].copy(), accum_f64=True)
        assert np.array_equal(it.cpu().numpy(), oi), kw
        assert np.array_equal(pot.cpu().numpy(), op), kw
        assert np.array_equal(flu.cpu().numpy(), of), kw
        np.testing.assert_allclose(err.cpu().numpy(), oe, rtol=1e-12, err_msg=str(kw))


@pytest.mark.parametrize("rs", [4, 8])
@pytest.mark.parametrize("g", [1, 2, 3, 4, 5])
def test_launch_sizes_agree(rs, g):
    """Small launches run a kernel with more threads per patch: the same bits for a
    patch solved in a launch of either kind, and the oracle's."""
    torch = pytest.importorskip("torch")
    from gpg.lib import solve_device
    from oracle.oracle import run_oracle
    dev = torch.device("cuda:0")
    d = make_patches(297, g, seed=90 + g, dtype=np.float32 if rs == 4 else np.float64)
    p = default_params(rs, g, GPG_MG)
    t = {k: torch.from_numpy(d[k]).to(dev) for k in ("rho", "pot_in", "flu")}

    def solve(n):
        flu = t["flu"][:n].clone()
        pot, _, it, err = solve_device(p, t["rho"][:n], t["pot_in"][:n], flu=flu)
        return pot, flu, it, err

    want = solve(297)
    for n in (1, 148, 149, 296):
        for a, b in zip(solve(n), want):
            assert torch.equal(a, b[:n])
    op, of, oi, _ = run_oracle(p, d["rho"][:12], d["pot_in"][:12], flu=d["flu"][:12].copy(), accum_f64=True)
    assert np.array_equal(want[0][:12].cpu().numpy(), op)
    assert np.array_equal(want[1][:12].cpu().numpy(), of)
    assert np.array_equal(want[2][:12].cpu().numpy(), oi)
