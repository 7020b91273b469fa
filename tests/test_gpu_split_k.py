"""The tcgen05 GEMM's split of a long K over a cluster (S = 8, 4 or 2 CTAs per
128-row tile) against a torch FP64 product of the same BF16 operands: K at and
beside the multiples where S changes, ragged in K, M and N, and with padded
outputs.  FP32 sums of BF16 products in blocks: within 1e-5 of the sum of the
products' absolute values (K 2^-24 at K = 16384 is 1e-3; blocked sums and the
tensor core's accumulation stay far below)."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(128, 256, 4096), (256, 256, 4096), (80, 256, 4088), (130, 160, 2048), (1, 16, 2040),
                                   (256, 80, 1024), (77, 240, 1032), (256, 256, 1016), (2300, 48, 4096), (128, 256, 16384)])
def test_split(M, N, K):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from roundabout_b200 import _ffi

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    A = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    B = torch.randn(N, K, generator=g, device="cuda").to(torch.bfloat16)
    ld = N + 4
    out = torch.full((M, ld), float("nan"), device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    P = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    L = _ffi.get_lib()
    runs = []
    for _ in range(2):
        _ffi.check(L.vphys_gemm_tn_bf16(P(A), K, P(B), K, M, N, K, 0.5, None, None, N, 0, P(out), ld, None, N, None, M, P(err),
                                        None), "vphys_gemm_tn_bf16")
        runs.append(out.clone())
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    assert torch.equal(runs[0][:, :N], runs[1][:, :N])   # the sum does not depend on timing
    assert torch.isnan(out[:, N:]).all()
    want = 0.5 * (A.double() @ B.double().T)
    scale = 0.5 * (A.double().abs() @ B.double().abs().T)
    assert ((out[:, :N].double() - want).abs() <= 1e-5 * scale).all()


@pytest.mark.parametrize("rows,cols", [(1, 1), (31, 80), (32, 80), (33, 77), (4096, 80), (50, 800), (50, 766), (33, 767),
                                       (31, 768), (1, 4000), (8, 97), (65, 96), (80000, 97)])
def test_loss_gradient(rows, cols):
    """vphys_mlp_loss: tiles of 32 rows and 96 columns, one tile per block or (80000 x 97) several."""
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from roundabout_b200 import _ffi

    g = torch.Generator(device="cuda").manual_seed(rows * 1000 + cols)
    Y, T = (torch.randn(rows, cols, generator=g, device="cuda") for _ in range(2))
    w = torch.rand(cols, generator=g, device="cuda")
    d32 = torch.empty_like(Y)
    d16 = torch.empty(rows, cols, dtype=torch.bfloat16, device="cuda")
    dt = torch.empty(cols, rows, dtype=torch.bfloat16, device="cuda")
    loss = torch.zeros(1, device="cuda")
    P = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    _ffi.check(_ffi.get_lib().vphys_mlp_loss(P(Y), P(T), P(w), rows, cols, 0.25, P(d32), P(d16), P(dt), P(loss), None),
               "vphys_mlp_loss")
    want = 0.25 * w * (Y - T)
    assert torch.allclose(d32, want, rtol=1e-6, atol=1e-7)
    assert torch.equal(d16, d32.to(torch.bfloat16)) and torch.equal(dt, d16.T.contiguous())
    full = (w.double() * (Y.double() - T.double()) ** 2).sum()
    assert abs(float(loss) - float(full)) <= 1e-5 * float(full)   # positive FP32 terms: about sqrt(5000) roundings, 2e-6


@pytest.mark.parametrize("N,K", [(64, 160), (256, 256), (96, 8)])
@pytest.mark.parametrize("form", ["three outputs", "hidden layer", "output layer"])
def test_column_halves(N, K, form):
    """Row blocks in two column halves (up to 74 of them on 148 SMs) against whole
    ones (more): the same rows give the same bits, as every column's sum is formed alike."""
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from roundabout_b200 import _ffi

    g = torch.Generator(device="cuda").manual_seed(N + K)
    few = torch.cuda.get_device_properties(0).multi_processor_count // 2 * 128
    A = torch.randn(few + 133, K, generator=g, device="cuda").to(torch.bfloat16)
    B = torch.randn(N, K, generator=g, device="cuda").to(torch.bfloat16)
    bias = torch.randn(N, generator=g, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    P = lambda t: ctypes.c_void_p(t.data_ptr()) if t is not None else None  # noqa: E731
    f32, b16, b16t, act = {"three outputs": (1, 1, 1, 1), "hidden layer": (0, 1, 0, 1), "output layer": (1, 0, 0, 0)}[form]
    got = []
    for M in (few, few - 51, few + 133):
        o32 = torch.full((M, N), float("nan"), device="cuda") if f32 else None
        o16 = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda") if b16 else None
        o16t = torch.full((N, M), float("nan"), dtype=torch.bfloat16, device="cuda") if b16t else None
        _ffi.check(_ffi.get_lib().vphys_gemm_tn_bf16(P(A), K, P(B), K, M, N, K, 1.0, P(bias), None, N, act, P(o32), N, P(o16),
                                                     N, P(o16t), M, P(err), None), "vphys_gemm_tn_bf16")
        got.append([o[:few - 51] for o in (o32, o16, o16t.T if b16t else None) if o is not None])
    assert int(err.item()) == 0
    for other in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0], other))
    want = A[:few - 51].float() @ B.float().T + bias
    if f32:
        assert (got[0][0] - want).abs().max() <= 2e-3 * want.abs().max()   # FP32 sums in another order
