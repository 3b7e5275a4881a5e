"""The surrogate's GEMM over its operand layouts and ragged tiles, and its
depthwise kernels at channel counts with and without whole vectors."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# whole tiles, ragged multiples of 8 (the pipelined kernel), odd sizes (the other)
@pytest.mark.parametrize("M,N,K", [(64, 64, 32), (128, 192, 96), (72, 8, 40), (8, 200, 256),
                                   (136, 72, 24), (65, 66, 33), (63, 64, 40), (64, 62, 40)])
@pytest.mark.parametrize("ak", [True, False])
@pytest.mark.parametrize("bk", [True, False])
@pytest.mark.parametrize("splits", [1, 3])
def test_gemm_layouts(cuda, M, N, K, ak, bk, splits):
    import torch
    from pyphasefield_gb300 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(M + 7 * N + K)
    A = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    B = torch.randn(K, N, generator=g, device="cuda").bfloat16()
    a = A.contiguous() if ak else A.t().contiguous()
    b = B.t().contiguous() if bk else B.contiguous()
    y = torch.ones(M, N, device="cuda")
    bias = torch.randn(N, generator=g, device="cuda") if splits == 1 else None
    acc = 1 if splits > 1 else 0
    L.call("ppf_sg_gemm", C.c_void_p(a.data_ptr()), *((K, 1) if ak else (1, M)),
           C.c_void_p(b.data_ptr()), *((1, K) if bk else (N, 1)), C.c_void_p(y.data_ptr()), N,
           C.c_void_p(bias.data_ptr()) if bias is not None else None, acc, M, N, K, splits,
           C.c_void_p(torch.cuda.current_stream().cuda_stream))
    ref = A.double() @ B.double() + (bias.double() if bias is not None else 1.0)
    # float32 accumulation of K products of order one
    assert float((y.double() - ref).abs().max()) < 1e-6 * K


@pytest.mark.parametrize("Cn,E", [(6, 16), (16, 24), (18, 32), (64, 40), (72, 16)])
def test_block_channels(cuda, Cn, E):
    """Gradients of every parameter at channel counts of whole and of broken
    vectors, against the float64 oracle with the same bfloat16 roundings."""
    import torch
    from oracle import surrogate_ref as R
    from pyphasefield_gb300.surrogate import SurrogateNet
    P, B, H, W = 4, 2, 20, 28
    rng = np.random.default_rng(Cn)
    net = SurrogateNet(P=P, C=Cn, E=E, nblocks=2, delta_scale=(2.0, 3.0))
    net.load_params(R.random_params(P, Cn, E, 2, rng))
    f = rng.random((2, B, 2, H, W)).astype(np.float32)
    old, new = (torch.from_numpy(v).cuda() for v in f)
    s = torch.cuda.current_stream()
    net.forward(old, B, H, W, W, s)
    net.backward(old, new, B, H, W, W, s)
    _, ref, _ = R.loss_and_grads(net.params_numpy(), f[0].astype(np.float64),
                                 f[1].astype(np.float64), P, 2, net.in_norm, net.delta_scale)
    got = net.grads_numpy()
    for n, r in ref.items():
        assert np.linalg.norm(got[n] - r) < 1e-2 * np.linalg.norm(r), n


# gathers of whole 16-byte groups (tokens: ragged tiles, one and several splits), then
# an odd pitch, patches of 6 and channel counts without whole vectors (the other kernel)
@pytest.mark.parametrize("P,B,gh,gw,Cn,pad", [(4, 1, 3, 5, 8, 0), (8, 2, 5, 7, 24, 4),
                                              (16, 3, 6, 11, 72, 0), (4, 2, 21, 25, 64, 8),
                                              (12, 1, 9, 8, 136, 0), (8, 2, 5, 7, 24, 1),
                                              (6, 2, 5, 7, 24, 0), (8, 2, 5, 7, 18, 0)])
def test_patch_gather(cuda, P, B, gh, gw, Cn, pad):
    import torch
    from pyphasefield_gb300 import _lib as L
    H, W = gh * P, gw * P
    T, K, pitch = B * gh * gw, 2 * P * P, W + pad
    g = torch.Generator(device="cuda").manual_seed(P + 7 * Cn + T)
    f = torch.randn(B, 2, H, pitch, generator=g, device="cuda")
    w = torch.randn(Cn, K, generator=g, device="cuda").bfloat16()
    b = torch.randn(Cn, generator=g, device="cuda")
    dy = torch.randn(T, Cn, generator=g, device="cuda").bfloat16()
    y, yb = torch.empty(T, Cn, device="cuda"), torch.empty(T, Cn, device="cuda").bfloat16()
    dw, db = torch.ones(Cn, K, device="cuda"), torch.zeros(Cn, device="cuda")
    s = L.PpfSgShape()
    s.B, s.H, s.W, s.pitch, s.P, s.C, s.E = B, H, W, pitch, P, Cn, 8
    s.in_off0, s.in_sc0, s.in_off1, s.in_sc1 = 0.25, 2.0, -0.5, 0.75
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    L.call("ppf_sg_patch_fwd", C.byref(s), ptr(f), ptr(w), ptr(b), ptr(y), ptr(yb), st)
    L.call("ppf_sg_patch_bwd_weight", C.byref(s), ptr(f), ptr(dy), ptr(dw), ptr(db), st)
    off = torch.tensor([0.25, -0.5], device="cuda").view(1, 2, 1, 1)
    sc = torch.tensor([2.0, 0.75], device="cuda").view(1, 2, 1, 1)
    x = ((f[..., :W] - off) * sc).bfloat16().double()
    x = x.view(B, 2, gh, P, gw, P).permute(0, 2, 4, 1, 3, 5).reshape(T, K)
    # float32 accumulation of K (then T) products of order one
    assert float((y.double() - (x @ w.double().t() + b.double())).abs().max()) < 1e-6 * max(K, 64)
    assert torch.equal(yb, y.bfloat16())
    assert float((dw.double() - 1.0 - dy.double().t() @ x).abs().max()) < 1e-6 * max(T, 64)


# vectors of four and single elements, a ragged last CTA, more elements than one sweep
@pytest.mark.parametrize("P,B,gh,gw,pad", [(4, 1, 1, 1, 0), (4, 3, 5, 7, 4), (6, 2, 3, 5, 0),
                                           (8, 2, 3, 3, 1), (16, 2, 36, 40, 0), (5, 1, 90, 91, 0)])
def test_loss_and_its_gradient(cuda, P, B, gh, gw, pad):
    import torch
    from pyphasefield_gb300 import _lib as L
    H, W = gh * P, gw * P
    T, K, pitch = B * gh * gw, 2 * P * P, W + pad
    g = torch.Generator(device="cuda").manual_seed(T)
    out = torch.randn(T, K, generator=g, device="cuda")
    old, new = (torch.randn(B, 2, H, pitch, generator=g, device="cuda") for _ in range(2))
    grad = torch.empty(T, K, device="cuda").bfloat16()
    loss = torch.zeros(1, dtype=torch.float64, device="cuda")
    s = L.PpfSgShape()
    s.B, s.H, s.W, s.pitch, s.P, s.C, s.E = B, H, W, pitch, P, 8, 8
    s.s0, s.s1 = 2.0, 3.0
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    L.call("ppf_sg_mse", C.byref(s), ptr(out), ptr(old), ptr(new), ptr(grad), ptr(loss),
           C.c_void_p(torch.cuda.current_stream().cuda_stream))
    d = (new - old).double()[..., :W] * torch.tensor([2.0, 3.0], device="cuda").view(1, 2, 1, 1)
    d = out.double() - d.view(B, 2, gh, P, gw, P).permute(0, 2, 4, 1, 3, 5).reshape(T, K)
    # d^2 and sums of 32 in float32: 2^-24 times their few operations each
    assert abs(float(loss) / float((d * d).mean()) - 1.0) < 1e-6
    ref = 2.0 * d / (T * K)
    # bfloat16 rounding of a float32 difference of numbers of order ten
    assert float((grad.double() - ref).abs().max()) < 2.0**-8 * float(ref.abs().max())


# channels one by one (7, 1346), then in pairs
@pytest.mark.parametrize("Cn", [7, 1346, 6, 8])
def test_block_gradient_pair(cuda, Cn):
    """The bf16 copy of dy, written over dy_out's, and no copy: the same dy."""
    import torch
    from pyphasefield_gb300 import _lib as L
    B, gh, gw, E = 2, 3, 5, 16
    T = B * gh * gw
    g = torch.Generator(device="cuda").manual_seed(Cn)
    r = lambda *n: torch.randn(*n, generator=g, device="cuda")  # noqa: E731
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    s = L.PpfSgShape()
    s.B, s.H, s.W, s.pitch, s.P, s.C, s.E = B, 4 * gh, 4 * gw, 4 * gw, 4, Cn, E
    y, h, pre, act = r(T, Cn), r(T, Cn).bfloat16(), r(T, E), r(T, E).bfloat16()
    w1, w2, wd, dyo = r(E, Cn).bfloat16(), r(Cn, E).bfloat16(), r(Cn, 9), r(T, Cn)
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)

    def run(name, pair):
        dyb = dyo.bfloat16()
        dpre, dh, dhb = r(T, E).bfloat16(), r(T, Cn), r(T, Cn).bfloat16()
        dy = torch.empty(T, Cn, device="cuda")
        grads = [torch.zeros(n, device="cuda") for n in (E * Cn, E, Cn * E, Cn, Cn * 9, Cn)]
        L.call(name, C.byref(s), ptr(y), ptr(h), ptr(pre), ptr(act), ptr(w1), ptr(w2), ptr(wd),
               ptr(dyo), ptr(dyb), ptr(dpre), ptr(dh), ptr(dhb), ptr(dy),
               *([ptr(dyb)] if pair else []), *(ptr(q) for q in grads), st)
        # both bias gradients: a float32 sum of T numbers
        assert torch.allclose(grads[1].double(), dpre.double().sum(0), rtol=0, atol=1e-4)
        assert torch.allclose(grads[3].double(), dyo.double().sum(0), rtol=0, atol=1e-4)
        return dy, dyb

    dy, keep = run("ppf_sg_block_bwd", False)
    dy2, dyb = run("ppf_sg_block_bwd_pair", True)
    assert torch.equal(dy, dy2) and torch.equal(dyb, dy.bfloat16())
    assert torch.equal(keep, dyo.bfloat16())


# tcgen05 tiles of 64 columns (ragged N, and N = 520) and of 128 (512, 640); ragged M, K
@pytest.mark.parametrize("M", [4096, 4200])
@pytest.mark.parametrize("N,K", [(8, 64), (64, 192), (136, 40), (192, 384), (520, 72), (512, 192),
                                 (640, 8)])
def test_tensor_core_tiles(cuda, M, N, K):
    import torch
    from pyphasefield_gb300 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(M + 7 * N + K)
    A = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    B = torch.randn(N, K, generator=g, device="cuda").bfloat16()
    bias = torch.randn(N, generator=g, device="cuda")
    y = torch.empty(M, N, device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    L.call("ppf_sg_gemm", ptr(A), K, 1, ptr(B), 1, K, ptr(y), N, ptr(bias), 0, M, N, K, 1,
           C.c_void_p(torch.cuda.current_stream().cuda_stream))
    ref = A.double() @ B.double().t() + bias.double()
    # float32 accumulation of K products of order one
    assert float((y.double() - ref).abs().max()) < 1e-6 * max(K, 64)
