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


def test_one_workspace_at_a_time(L):
    """A batch of another size is made after the kept one has been given back, and releasing leaves nothing."""
    import torch

    s = L.KPPSurrogate(seed=1)
    row = 8320   # bytes of activations and their gradients per batch row
    small, large = batch(L, 16384, 1), batch(L, 16384 + 8, 2)
    s.gradients(*small)
    base = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    s.gradients(*large)
    # the new workspace in the old one's place, plus the results (Y, and the weights' gradients)
    assert torch.cuda.max_memory_allocated() - base < 0.2 * row * 16384
    s.release_workspace()
    assert base - torch.cuda.memory_allocated() > 0.9 * row * 16384
    s.gradients(*small)


def test_training_leaves_no_workspace(L):
    import torch

    s = L.KPPSurrogate(seed=1)
    X, XT, _, T = batch(L, 16384, 3)
    s.train(X, XT, T, epochs=1, batch=8192)
    before = torch.cuda.memory_allocated()
    s.train(X, XT, T, epochs=1, batch=8192)
    assert torch.cuda.memory_allocated() == before
    s.release_workspace()
    assert torch.cuda.memory_allocated() == before


def test_forward_keeps_its_activations(L):
    """forward(save=True) leaves the hidden layers' activations, its own, and the same outputs as without."""
    import torch

    s = L.KPPSurrogate(seed=1)
    X = batch(L, 256, 4)[0]
    Y = s.forward(X, save=True)
    c = s._cache
    assert torch.equal(c["H1T"], c["H1"].T) and torch.equal(c["H2T"], c["H2"].T)
    z1 = X.float() @ s.Wb[0].float().T + s.b[0]
    z2 = c["H1"].float() @ s.Wb[1].float().T + s.b[1]
    for got, want in ((c["Z1"], z1), (c["Z2"], z2)):
        assert (got - want).abs().max() <= 2e-3 * want.abs().max()   # FP32 sums in another order
    kept = {k: t.clone() for k, t in c.items()}
    s.gradients(*batch(L, 256, 5))
    assert all(torch.equal(c[k], t) for k, t in kept.items())
    assert torch.equal(s.forward(X), Y) and s._cache is None


@pytest.mark.parametrize("n", [0, 1, 255, 256, 257, 5000])
def test_zero(L, n):
    """vphys_mlp_zero: the given lengths, no further, and null buffers left out."""
    import torch

    from roundabout_b200 import _ffi

    a, b = torch.ones(n + 3, device="cuda"), torch.ones(8, device="cuda")
    _ffi.check(_ffi.get_lib().vphys_mlp_zero(a.data_ptr(), n, None, 4, b.data_ptr(), 5, None, 0, None), "vphys_mlp_zero")
    assert not a[:n].any() and (a[n:] == 1).all()
    assert not b[:5].any() and (b[5:] == 1).all()
