"""The network's training kernels split a batch into units of 10, 5, 2 or 1
planes of a patch by its size.  A batch whose size is a power of two times
another's scales the loss gradient by a power of two, exactly also in bfloat16,
so its gradient is the mean of its parts' gradients up to the order of the FP32
sums (needs a B200).

Tolerance: FP32 sums over at most 1024 x 1000 cells, of which one accumulator
takes 490 MMA steps and the last stage 148 partial sums; the gradients cancel by
about a factor of ten: 1e-3 in the 2-norm, that of the comparison with the
oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,part", [(2, 1), (64, 32), (128, 32), (512, 128), (1024, 128)])
def test_gradient_of_a_batch_is_the_mean_of_its_parts(n, part):
    torch = pytest.importorskip("torch")
    from gpg.inputs import make_patches
    from gpg.net import Net
    dev = torch.device("cuda:0")
    d = make_patches(n, 1, seed=5, dtype=np.float32, fluid=False)
    rho, pin = (torch.from_numpy(d[k]).to(dev) for k in ("rho", "pot_in"))
    target = pin.mean((1, 2, 3), keepdim=True) * torch.linspace(0.9, 1.1, 512, device=dev).view(1, 8, 8, 8)
    cnst = float(np.float32(4 * np.pi * 1e-5))
    net = Net(max_batch=n, seed=3)

    def run(lo, hi):
        g, loss = torch.full((net.nparams,), float("nan"), device=dev), torch.empty(1, device=dev)
        net.gradients(rho[lo:hi], pin[lo:hi], target[lo:hi].contiguous(), cnst, grad=g, loss=loss)
        return g.double(), loss.double()

    whole, loss = run(0, n)
    again, _ = run(0, n)
    assert torch.equal(whole, again)
    parts = [run(lo, lo + part) for lo in range(0, n, part)]
    mean = torch.stack([g for g, _ in parts]).mean(0)
    assert torch.isfinite(whole).all()
    assert (whole - mean).norm() <= 1e-3 * mean.norm()
    want = torch.stack([q for _, q in parts]).mean()
    assert abs(loss - want) <= 1e-5 * want
    net.check()
    net.close()
