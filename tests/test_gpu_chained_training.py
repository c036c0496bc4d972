"""Chains of launches whose kernels' starts and ends overlap, without and with a
synchronisation after each: the same bits.  Every array that a chain hands on
holds a wrong value when the chain begins (needs a B200)."""
import numpy as np
import pytest

from gpg.abi import GPG_INIT_GUESS, GPG_INIT_ZERO, GPG_MG, GPG_SOR, default_params
from gpg.inputs import make_patches

pytestmark = pytest.mark.gpu
CNST = float(np.float32(4 * np.pi * 1e-5))


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("no CUDA device")
    return t


@pytest.mark.parametrize("rs", [4, 8])
@pytest.mark.parametrize("npatch", [3, 300, 5000])
@pytest.mark.parametrize("g", [1, 2, 3])
def test_start_values_handed_from_solve_to_solve(torch, rs, npatch, g):
    """At ghost 1, 2 and 3 an output window of ghost g - 1 has the cells of a start
    value, so each solve reads what the kernel before it wrote."""
    from gpg.lib import solve_device
    d = make_patches(npatch, g, seed=17 + g, gra_ghost=g - 1, dtype=np.float32 if rs == 4 else np.float64, fluid=False)
    rho, pin = (torch.from_numpy(d[k]).cuda() for k in ("rho", "pot_in"))
    kw = dict(gra_ghost=g - 1, gra_acc=0)
    first = default_params(rs, g, GPG_SOR, init_mode=GPG_INIT_ZERO, sor_max_iter=3, **kw)
    next_ = default_params(rs, g, GPG_SOR, init_mode=GPG_INIT_GUESS, sor_max_iter=3, **kw)
    mg = default_params(rs, g, GPG_MG, mg_max_iter=1, **kw)
    m = 6 + 2 * g

    def poisoned():
        return [torch.full((npatch, m, m, m), 1e3 * (k + 1), device="cuda", dtype=rho.dtype) for k in range(6)]

    iters = torch.zeros(npatch, device="cuda", dtype=torch.int32)
    resid = torch.zeros(npatch, device="cuda", dtype=torch.float64)

    def chain(o, wait):
        src = None
        for k, p in enumerate((first, next_, next_, mg, next_, next_)):
            # the density of the multigrid solve is the potential before it
            solve_device(p, src if p is mg else rho, pin, pot_out=o[k], guess=src if p is next_ else None, iters=iters,
                         resid=resid)
            src = o[k]
            if wait:
                torch.cuda.synchronize()

    want, got, again = poisoned(), poisoned(), poisoned()
    chain(want, True)
    chain(got, False)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain(again, False)
    for a, b in zip(again, poisoned()):
        a.copy_(b)
    graph.replay()
    torch.cuda.synchronize()
    for a, b, c in zip(want, got, again):
        assert torch.equal(a, b) and torch.equal(a, c)
        assert not torch.equal(a, want[-1]) or a is want[-1]


@pytest.mark.parametrize("npatch", [1, 5, 40, 300])
def test_network_training(torch, npatch):
    from gpg.net import Net
    d = make_patches(npatch, 1, seed=4, fluid=False)
    rho, pin = (torch.from_numpy(d[k]).cuda() for k in ("rho", "pot_in"))

    def chain(wait):
        net = Net(max_batch=npatch, seed=3)
        out, target = [], pin
        for _ in range(4):     # each step's target is the prediction before it
            loss = torch.full((1,), -1.0, device="cuda")
            guess = torch.full((npatch, 8, 8, 8), 1e3, device="cuda")
            grad = torch.full((net.nparams,), 1e3, device="cuda")
            for call in (lambda: net.train_step(rho, pin, target, CNST, 1e-3, loss=loss),
                         lambda: net.predict(rho, pin, guess, CNST),
                         lambda: net.gradients(rho, pin, guess, CNST, grad=grad),
                         lambda: net.apply_gradient(grad, 1e-3)):
                call()
                if wait:
                    torch.cuda.synchronize()
            target = guess
            out += [loss, guess, grad]
        out.append(torch.from_numpy(net.params()))
        net.check()
        net.close()
        return out

    for a, b in zip(chain(True), chain(False)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("npatch", [1, 64, 300, 3000])
def test_correction_training(torch, npatch):
    from gpg.linear import LinearGuess
    d = make_patches(npatch, 1, seed=4, fluid=False)
    rho, pin = (torch.from_numpy(d[k]).cuda() for k in ("rho", "pot_in"))
    p = default_params(4, 1, GPG_SOR, gra_ghost=0, gra_acc=0, sor_max_iter=4)

    def chain(wait):
        lin = LinearGuess(max_batch=npatch)
        out, src = [], rho
        for _ in range(4):     # features of the solve before, a step on them, a solve with the new weights
            target = torch.full((npatch, 8, 8, 8), 1e3, device="cuda")
            loss = torch.full((1,), -1.0, device="cuda")
            lin.solve(p, src, pin, pot_out=target)
            if wait:
                torch.cuda.synchronize()
            u, t = lin.features(p, rho, pin, target)
            if wait:
                torch.cuda.synchronize()
            lin.train_step(u, t, 1e-3, loss=loss)
            if wait:
                torch.cuda.synchronize()
            src = target
            out += [target, u, t, loss]
        out.append(torch.from_numpy(lin.params()))
        lin.check()
        lin.close()
        return out

    for a, b in zip(chain(True), chain(False)):
        assert torch.equal(a, b)
