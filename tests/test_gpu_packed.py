"""FP32 two-row SOR kernels sweep two heights per packed register pair: their
results must be those of the scalar one-row kernel (variant 0) bit for bit,
also where values are zeros of either sign, denormal or not finite, and at
patch counts around a launch's tail (needs a B200)."""
import numpy as np
import pytest

from gpg.abi import GPG_SOR, default_params
from gpg.inputs import make_patches

pytestmark = pytest.mark.gpu


def special_patches(npatch, g):
    d = make_patches(npatch, g, seed=40 + g, dtype=np.float32, fluid=False)
    rho, pin = d["rho"], d["pot_in"]
    rho[0], pin[0] = 0.0, 0.0
    if npatch > 1:
        rho[1], pin[1] = -0.0, -0.0
    if npatch > 2:
        rho[2] *= np.float32(1e-38)
        pin[2] *= np.float32(1e-40)
    if npatch > 3:
        rho[3, 1, 2, 3] = np.nan
    if npatch > 4:
        pin[4, 3, 3, 3] = np.inf
    return rho, pin


@pytest.mark.parametrize("g", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("npatch", [1, 149, 331])
def test_packed_kernels_return_the_scalar_bits(g, npatch):
    torch = pytest.importorskip("torch")
    from gpg.lib import check, library, solve_device
    lib, dev = library(), torch.device("cuda:0")
    rho, pin = (torch.from_numpy(a).to(dev) for a in special_patches(npatch, g))
    p = default_params(4, g, GPG_SOR, gra_acc=0, sor_max_iter=23)
    outs = {}
    try:
        for v in (0, 10, 11, 12, 13, 14, 15, 16):
            check(lib.gpg_set_sor_variant(4, g, v))
            pot, _, it, rs = solve_device(p, rho, pin)
            outs[v] = [pot.view(torch.int32).cpu(), torch.isnan(pot).cpu(), it.cpu(), rs.cpu()]
    finally:
        check(lib.gpg_set_sor_variant(4, g, -1))
    bits0, nan0, it0, rs0 = outs[0]
    for v, (bits, nan, it, rs) in outs.items():
        assert torch.equal(nan, nan0) and torch.equal(it, it0), v
        assert torch.equal(bits[~nan], bits0[~nan0]), v  # a NaN's payload is not specified
        assert torch.equal(torch.nan_to_num(rs, nan=-1.0), torch.nan_to_num(rs0, nan=-1.0)), v


@pytest.mark.parametrize("rs,g,gg", [(4, 1, 1), (4, 2, 2), (4, 3, 1), (4, 4, 2), (4, 5, 1), (8, 1, 1), (8, 4, 2)])
@pytest.mark.parametrize("scheme", [1, 2])
def test_wide_loads_fall_back_off_their_alignment(rs, g, gg, scheme):
    """Density pairs, coarse-potential pairs and 16-byte fluid runs: arrays one
    element off the allocation's alignment give the aligned arrays' bits."""
    torch = pytest.importorskip("torch")
    from gpg.lib import solve_device
    dev = torch.device("cuda:0")
    d = make_patches(37, g, seed=60 + g, gra_ghost=gg, dtype=np.float32 if rs == 4 else np.float64)
    p = default_params(rs, g, scheme, gra_ghost=gg, p5_gradient=int(gg == 2))

    def off(t, k):
        buf = torch.empty(t.numel() + k, dtype=t.dtype, device=dev)
        buf[k:] = t.reshape(-1)
        return buf[k:].view(t.shape)

    t = {k: torch.from_numpy(d[k]).to(dev) for k in ("rho", "pot_in", "flu")}
    want = solve_device(p, t["rho"], t["pot_in"], flu=t["flu"].clone())
    for k in (1, 2, 3):
        got = solve_device(p, off(t["rho"], k), off(t["pot_in"], k), flu=off(t["flu"], k))
        for a, b in zip(got, want):
            assert torch.equal(a, b), k


@pytest.mark.parametrize("g", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("init", [0, 1])
def test_one_row_columns_off_their_alignment(g, init):
    """FP32 lanes of one row and a whole column choose between pair and single
    density loads once for the column: the same bits either way."""
    torch = pytest.importorskip("torch")
    from gpg.lib import check, library, solve_device
    d = make_patches(37, g, seed=80 + g, dtype=np.float32, fluid=False)
    rho, pin = (torch.from_numpy(d[k]).cuda() for k in ("rho", "pot_in"))
    buf = torch.empty(rho.numel() + 1, device="cuda")
    buf[1:] = rho.reshape(-1)
    p = default_params(4, g, GPG_SOR, gra_acc=0, init_mode=init)
    try:
        for v in range(6):
            check(library().gpg_set_sor_variant(4, g, v))
            try:
                want = solve_device(p, rho, pin)
            except Exception:       # more threads than the registers allow
                continue
            got = solve_device(p, buf[1:].view(rho.shape), pin)
            for k in (0, 2, 3):
                assert torch.equal(got[k], want[k]), v
    finally:
        check(library().gpg_set_sor_variant(4, g, -1))
