"""What KPPSurrogate.gradients keeps between calls and what it gives away."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def L():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from roundabout_b200 import learned

    return learned


def batch(L, B, seed):
    import torch

    g = torch.Generator(device="cuda").manual_seed(seed)
    X = torch.randn(B, L.NINP, device="cuda", generator=g).to(torch.bfloat16)
    return X, X.T.contiguous(), B, torch.randn(B, L.NOUTP, device="cuda", generator=g)


def test_results_are_the_callers(L):
    """The loss and every gradient are tensors of their own, aligned as torch allocates them, and a later call leaves
    them alone."""
    import torch

    s = L.KPPSurrogate(seed=1)
    loss, Y, gW, gb = s.gradients(*batch(L, 256, 1))
    out = [loss, Y, *gW, *gb]
    assert all(t.data_ptr() % 512 == 0 for t in out)
    assert all(t.untyped_storage().nbytes() == t.numel() * 4 for t in out)
    assert len({t.untyped_storage().data_ptr() for t in out}) == len(out)
    kept = [t.clone() for t in out]
    s.gradients(*batch(L, 256, 2))
    assert all(torch.equal(a, b) for a, b in zip(out, kept))
