"""Device memory of the learned starts' handles, and their training at batches
around the number of partial sums that the memory is sized for (needs a B200)."""
import numpy as np
import pytest

from gpg.inputs import make_patches

pytestmark = pytest.mark.gpu
CNST = float(np.float32(4 * np.pi * 1e-5))


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("no CUDA device")
    return t


def _net(n):
    from gpg.net import Net
    return Net(max_batch=n, seed=2)


def _lin(n):
    from gpg.linear import LinearGuess
    m = LinearGuess(max_batch=n)
    m.set_params(0.01 * np.random.default_rng(4).standard_normal(m.nparams).astype(np.float32))
    return m


@pytest.mark.parametrize("make,mib", [(_net, 8), (_lin, 2)])
def test_small_handles_are_small(torch, make, mib):
    """A handle for one patch holds its weights and a patch's work, not a batch's."""
    make(1).close()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    handles = [make(1) for _ in range(8)]
    used = free - torch.cuda.mem_get_info()[0]
    for h in handles:
        h.close()
    assert used <= 8 * mib * 2 ** 20


def _net_step(torch, h, n):
    d = make_patches(n, 1, seed=9, fluid=False)
    rho, pin = (torch.from_numpy(d[k]).cuda() for k in ("rho", "pot_in"))
    grad, loss = torch.empty(h.nparams, device="cuda"), torch.empty(1, device="cuda")
    h.gradients(rho, pin, pin * 1.1, CNST, grad=grad, loss=loss)
    return grad, loss


def _lin_step(torch, h, n):
    g = torch.Generator(device="cuda").manual_seed(n)
    u, t = (torch.randn((n, 8, 64), generator=g, device="cuda") for _ in range(2))
    grad, loss = torch.empty(h.nparams, device="cuda"), torch.empty(1, device="cuda")
    h.gradients(u, t, grad=grad, loss=loss)
    return grad, loss


@pytest.mark.parametrize("make,step,sizes", [(_net, _net_step, (1, 2, 14, 15, 16, 60)),
                                             (_lin, _lin_step, (1, 63, 64, 65, 2368, 2369))])
def test_full_batch_gives_the_larger_handles_bits(torch, make, step, sizes):
    big = make(4096 if make is _lin else 64)
    for n in sizes:
        h = make(n)
        for a, b in zip(step(torch, h, n), step(torch, big, n)):
            assert torch.equal(a, b), n
        h.check()
        h.close()
    big.close()


def test_create_without_memory_leaves_no_error(torch):
    """A handle too large for the device is refused; the next calls work."""
    from gpg.abi import GPG_ERR_OOM
    from gpg.lib import GpgError
    with pytest.raises(GpgError) as e:
        _net(1 << 20)
    assert e.value.status == GPG_ERR_OOM
    h = _net(2)
    _net_step(torch, h, 2)
    torch.cuda.synchronize()
    h.check()
    h.close()
