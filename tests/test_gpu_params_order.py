"""Parameters set, read or created by a host call, with the kernels before and
after it on a stream that the default stream does not order (needs a B200)."""
import numpy as np
import pytest

from gpg.abi import GPG_SOR, default_params
from gpg.inputs import make_patches

pytestmark = pytest.mark.gpu
CNST = float(np.float32(4 * np.pi * 1e-5))
N = 512


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("no CUDA device")
    return t


def _inputs(torch):
    d = make_patches(N, 1, seed=5, fluid=False)
    return [torch.from_numpy(d[k]).cuda() for k in ("rho", "pot_in")]


class _Net:
    def __init__(self, torch, seed=1):
        from gpg.net import Net
        self.h = Net(max_batch=N, seed=seed)
        self.rho, self.pin = _inputs(torch)
        self.target = self.pin.clone()
        self.torch = torch

    def apply(self, stream):
        out = self.torch.empty((N, 8, 8, 8), device="cuda")
        self.h.predict(self.rho, self.pin, out, CNST, stream=stream)
        return out

    def train(self, stream):
        self.h.train_step(self.rho, self.pin, self.target, CNST, 1e-3, stream=stream)


class _Lin:
    def __init__(self, torch, seed=1):
        from gpg.linear import LinearGuess
        self.h = LinearGuess(max_batch=N)
        self.rho, self.pin = _inputs(torch)
        self.p = default_params(4, 1, GPG_SOR, gra_ghost=0, gra_acc=0, sor_max_iter=2)
        g = torch.Generator(device="cuda").manual_seed(3)
        self.u, self.t = (torch.randn((N, 8, 64), generator=g, device="cuda") for _ in range(2))
        self.torch = torch

    def apply(self, stream):
        out = self.torch.empty((N, 8, 8, 8), device="cuda")
        self.h.solve(self.p, self.rho, self.pin, pot_out=out, stream=stream)
        return out

    def train(self, stream):
        self.h.train_step(self.u, self.t, 1e-3, stream=stream)


@pytest.mark.parametrize("kind", [_Net, _Lin])
def test_set_params_then_another_stream(torch, kind):
    m, side = kind(torch), torch.cuda.Stream()
    rng = np.random.default_rng(2)
    weights = [0.05 * rng.standard_normal(m.h.nparams).astype(np.float32) for _ in range(2)]
    want = []
    for w in weights:
        m.h.set_params(w)
        torch.cuda.synchronize()
        want.append(m.apply(None))
        torch.cuda.synchronize()
    assert not torch.equal(*want)
    for k in range(20):
        m.h.set_params(weights[k % 2])
        got = m.apply(side)
        side.synchronize()
        assert torch.equal(got, want[k % 2])
    m.h.check()
    m.h.close()


@pytest.mark.parametrize("kind", [_Net, _Lin])
def test_get_and_set_params_wait_for_training_steps(torch, kind):
    m, side = kind(torch), torch.cuda.Stream()
    start = m.h.params()
    torch.cuda.synchronize()

    def steps():
        for _ in range(10):
            m.train(side)

    steps()
    got = m.h.params()
    torch.cuda.synchronize()
    assert np.array_equal(got, m.h.params())
    steps()
    m.h.set_params(start)     # nothing of the steps is left, the moments included
    torch.cuda.synchronize()
    assert np.array_equal(m.h.params(), start)
    steps()
    assert np.array_equal(m.h.params(), got)
    m.h.close()


def test_created_net_on_another_stream(torch):
    side = torch.cuda.Stream()
    want = None
    for _ in range(5):
        m = _Net(torch, seed=4)
        got = m.apply(side)
        side.synchronize()
        want = got if want is None else want
        assert torch.equal(got, want)
        m.h.close()
