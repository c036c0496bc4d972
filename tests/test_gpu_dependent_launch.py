"""Solves that read what the solve just before them wrote, launched back to back
(their kernels' starts and ends overlap), in a stream and in a captured graph:
the same bits as with a synchronisation between them (needs a B200)."""
import numpy as np
import pytest

from gpg.abi import GPG_INIT_GUESS, GPG_INIT_ZERO, GPG_MG, GPG_SOR, default_params
from gpg.inputs import make_patches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rs", [4, 8])
@pytest.mark.parametrize("npatch", [3, 300, 5000])
@pytest.mark.parametrize("g", [1, 4, 5])
def test_chained_solves(rs, npatch, g):
    torch = pytest.importorskip("torch")
    from gpg.lib import solve_device
    dev = torch.device("cuda:0")
    dt = np.float32 if rs == 4 else np.float64
    d = make_patches(npatch, g, seed=7 + g, dtype=dt)
    rho, pin, flu0 = (torch.from_numpy(d[k]).to(dev) for k in ("rho", "pot_in", "flu"))
    tdt = rho.dtype
    m = 6 + 2 * g
    guess = torch.zeros((npatch, m, m, m), device=dev, dtype=tdt)
    first = default_params(rs, g, GPG_SOR, gra_ghost=0, gra_acc=0, init_mode=GPG_INIT_ZERO, sor_max_iter=4)
    second = default_params(rs, g, GPG_SOR, init_mode=GPG_INIT_GUESS, sor_max_iter=12)
    mg = default_params(rs, g, GPG_MG, mg_max_iter=2)
    lo = g - 1

    def outputs():
        return [torch.zeros((npatch, 8, 8, 8), device=dev, dtype=tdt)] + \
            [torch.zeros((npatch, 10, 10, 10), device=dev, dtype=tdt) for _ in range(2)] + \
            [torch.zeros(npatch, device=dev, dtype=torch.int32) for _ in range(3)] + \
            [torch.zeros(npatch, device=dev, dtype=torch.float64) for _ in range(3)] + [flu0.clone()]

    def chain(o, wait):
        step = torch.cuda.synchronize if wait else (lambda: None)
        if g == 1:      # the second solve starts from what the first one wrote
            solve_device(first, rho, pin, pot_out=o[0], iters=o[3], resid=o[6])
            step()
            solve_device(second, rho, pin, pot_out=o[1], flu=o[9], guess=o[0], iters=o[4], resid=o[7])
        else:           # the fluid passes through both
            solve_device(first, rho, pin, pot_out=o[0], iters=o[3], resid=o[6])
            step()
            guess[:, lo:lo + 8, lo:lo + 8, lo:lo + 8] = o[0]
            step()
            solve_device(second, rho, pin, pot_out=o[1], flu=o[9], guess=guess, iters=o[4], resid=o[7])
        step()
        solve_device(mg, rho, pin, pot_out=o[2], flu=o[9], iters=o[5], resid=o[8])
        step()

    want = outputs()
    chain(want, True)
    got = outputs()
    chain(got, False)
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a, b)

    again = outputs()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain(again, False)
    for k, t in enumerate(outputs()):
        again[k].copy_(t)
    graph.replay()
    torch.cuda.synchronize()
    for a, b in zip(again, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("npatch", [1, 9, 300, 5000])
@pytest.mark.parametrize("variant", [0, 1])
def test_chained_learned_solves(npatch, variant):
    torch = pytest.importorskip("torch")
    from gpg.linear import LinearGuess
    dev = torch.device("cuda:0")
    d = make_patches(npatch, 1, seed=3, dtype=np.float32)
    rho, pin = (torch.from_numpy(d[k]).to(dev) for k in ("rho", "pot_in"))
    lin = LinearGuess(max_batch=64)
    lin.set_params(0.01 * np.random.default_rng(5).standard_normal(lin.nparams).astype(np.float32))
    lin.set_variant(variant)
    p = default_params(4, 1, GPG_SOR, gra_ghost=0, gra_acc=0, sor_max_iter=6)

    def chain(wait):
        out, src = [], rho  # each solve's density is the potential before it
        for _ in range(4):
            out.append(lin.solve(p, src, pin))
            src = out[-1][0]
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return out

    for a, b in zip(chain(True), chain(False)):
        for k in (0, 2, 3):
            assert torch.equal(a[k], b[k])
    lin.check()
    lin.close()
