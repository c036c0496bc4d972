"""The learned correction's gradient at patch counts around the kernel's chunk
(64 patches) and split (37 CTAs per block), and with features off the 16-byte
alignment of its vector loads, against the FP64 oracle (needs a B200).

Tolerance: each value is a chain of at most 64 + 64 ceil(n / 2368) FP32
multiply-adds and 37 partial sums, each off by at most 2^-24 of the running
sum of magnitudes: 1e-5 in the 2-norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 2368, 2369])
def test_gradient_at_chunk_edges(n, offset):
    torch = pytest.importorskip("torch")
    from gpg.linear import LinearGuess
    from oracle.lin_oracle import gradients
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(n)
    u, t = (rng.standard_normal((n, 8, 64)).astype(np.float32) for _ in range(2))
    w = (0.1 * rng.standard_normal(4 * 64 * 64)).astype(np.float32)

    def place(a):
        buf = torch.empty(a.size + offset, device=dev)
        buf[offset:] = torch.from_numpy(a.reshape(-1)).to(dev)
        return buf[offset:].view(a.shape)

    lin = LinearGuess(max_batch=n)
    lin.set_params(w)
    grad, loss = torch.full((lin.nparams,), float("nan"), device=dev), torch.empty(1, device=dev)
    lin.gradients(place(u), place(t), grad=grad, loss=loss)
    want_loss, want = gradients(w.astype(np.float64).reshape(4, 64, 64), u.astype(np.float64), t.astype(np.float64))
    want = np.asarray(want).reshape(-1)
    got = grad.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)
    assert abs(loss.item() - want_loss) <= 1e-5 * want_loss
    lin.close()
