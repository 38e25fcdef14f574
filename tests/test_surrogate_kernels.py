"""The surrogate's GEMM of few tiles and its data-movement kernels at the sizes
where their tiles, vectors and ranges end.  Operands are small integers, so every
product and sum is exact in float32 and the results have to be equal."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def _p(t, off=0):
    return C.c_void_p(int(t.data_ptr()) + off)


def _ints(torch, g, *shape):
    return torch.randint(-2, 3, shape, device="cuda", generator=g).to(torch.bfloat16)


@pytest.mark.parametrize("M,N,K", [
    (128, 64, 64),               # 64 x 16 tiles, one K step of 20 stages
    (128, 64, 20 * 64),          # as many steps as stages
    (128, 64, 3001 * 64),
    (1024, 128, 41 * 64),        # 128 tiles of 64 x 16
    (1152, 128, 17 * 64),        # 144
    (1280, 128, 33 * 64),        # 160: 64 x 32
    (256, 1152, 16 * 64),
    (1024, 512, 13 * 64),        # 64 x 64
    (64 * 74, 128, 12 * 64),     # 148 tiles of 64 x 64
    (64 * 76, 128, 12 * 64),     # 152: 128-row tiles
])
@pytest.mark.parametrize("form", ["f32", "bias_relu", "bf16"])
def test_gemm_of_few_tiles_is_exact(M, N, K, form):
    import torch
    from solargpu_b200 import api
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    A, B = _ints(torch, g, M, K), _ints(torch, g, N, K)
    want = (A.double() @ B.double().T).float()           # |sum| <= 4 K < 2^24
    bias = torch.randint(-9, 10, (N,), device="cuda", generator=g).float()
    if form == "f32":
        assert torch.equal(api.gemm_bf16(A, B), want)
    elif form == "bias_relu":
        assert torch.equal(api.gemm_bf16(A, B, bias=bias, relu=True), torch.relu(want + bias))
    else:
        out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
        api.gemm_bf16(A, B, out_bf16=out, bias=bias)
        assert torch.equal(out, (want + bias).to(torch.bfloat16))


@pytest.mark.parametrize("M,N,K", [(128, 64, 8192), (1024, 128, 4096), (1280, 128, 1024), (1024, 512, 2112)])
def test_gemm_of_few_tiles_has_the_bits_of_wide_ones(M, N, K, monkeypatch):
    """The same K order, whatever the tile: equal bits for any operands."""
    import torch
    from solargpu_b200 import api
    g = torch.Generator(device="cuda").manual_seed(5)
    A = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    B = torch.randn(N, K, device="cuda", generator=g).to(torch.bfloat16)
    got = api.gemm_bf16(A, B)
    monkeypatch.setenv("SGB_GEMM_BN", "64")
    assert torch.equal(got, api.gemm_bf16(A, B))


@pytest.mark.parametrize("M,N,K", [
    (64, 128, 64), (64, 128, 64 * 20), (64, 128, 64 * 1003), (128, 1024, 64 * 21), (128, 64, 64 * 3),
    (128, 2048, 64 * 9), (512, 2112, 64 * 5), (384, 512, 64 * 16), (64, 2304, 64 * 6),
])
def test_weight_gradient(M, N, K, monkeypatch):
    """Exact on integers, at every tile width; and for any operands the bits of the
    product of transposed copies, whichever operand gives the rows."""
    import torch
    from solargpu_b200 import api, surrogate
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    L = surrogate._lib()

    def grad(X, Y):
        out = torch.full((M, N), 7.0, device="cuda")
        api._check(L.solar_gpu_sg_weight_grad(_p(X), _p(Y), K, M, N, _p(out), None))
        return out
    X, Y = _ints(torch, g, K, M), _ints(torch, g, K, N)
    assert torch.equal(grad(X, Y), (X.double().T @ Y.double()).float())
    X, Y = (torch.randn(K, n, device="cuda", generator=g).to(torch.bfloat16) for n in (M, N))
    monkeypatch.setenv("SGB_GEMM_BN", "64")
    got, xt, yt = grad(X, Y), X.T.contiguous(), Y.T.contiguous()
    if M % 128 == 0:
        assert torch.equal(got, api.gemm_bf16(xt, yt))
    if N % 128 == 0:
        assert torch.equal(got, api.gemm_bf16(yt, xt).T)


def test_weight_gradient_refuses_what_the_products_refuse():
    from solargpu_b200 import surrogate
    L, p = surrogate._lib(), C.c_void_p(256)
    for rows, n_out, n_in in [(100, 64, 128), (64, 60, 128), (64, 64, 120), (64, 192, 64), (0, 64, 128)]:
        assert L.solar_gpu_sg_weight_grad(p, p, rows, n_out, n_in, p, None) in (-1, -2)
    assert L.solar_gpu_sg_weight_grad(C.c_void_p(264), p, 64, 64, 128, p, None) == -1


@pytest.mark.parametrize("R,Cc", [(1, 1), (8, 8), (64, 64), (72, 200), (65, 64), (63, 129), (4104, 72), (7, 513)])
@pytest.mark.parametrize("off", [0, 2])                  # bytes past a 16-byte boundary
def test_transpose_and_column_sums(R, Cc, off):
    import torch
    from solargpu_b200 import api
    g = torch.Generator(device="cuda").manual_seed(R * 1000 + Cc)
    buf = _ints(torch, g, R * Cc + 8)
    x = buf[off // 2: off // 2 + R * Cc].view(R, Cc)
    out = torch.zeros(R * Cc + 8, dtype=torch.bfloat16, device="cuda")
    L = api.lib()
    api._check(L.solar_gpu_sg_transpose(_p(x), R, Cc, _p(out, off), None))
    sums = torch.empty(Cc, device="cuda")
    api._check(L.solar_gpu_sg_colsum(_p(x), R, Cc, _p(sums), None))
    torch.cuda.synchronize()
    assert torch.equal(out[off // 2: off // 2 + R * Cc].view(Cc, R), x.T)
    assert not out[off // 2 + R * Cc:].any()
    assert torch.equal(sums, x.float().sum(0))


@pytest.mark.parametrize("Cin,Kp", [(1, 64), (2, 64), (2, 128), (3, 64), (4, 64), (8, 128), (24, 448)])
@pytest.mark.parametrize("Hi,Wi", [(2, 2), (2, 6), (10, 4), (64, 64)])
def test_im2col_against_padded_windows(Cin, Kp, Hi, Wi):
    import torch
    from solargpu_b200 import api
    g = torch.Generator(device="cuda").manual_seed(Cin * 100 + Hi + Wi)
    n = 3 * Hi * Wi * Cin
    for off in ([0, 1] if Cin < 8 else [0]):             # elements: 2-byte aligned images too
        x = _ints(torch, g, n + 1)[off: off + n].view(3, Hi, Wi, Cin)
        cols = torch.full((3 * (Hi // 2) * (Wi // 2), Kp), 9.0, dtype=torch.bfloat16, device="cuda")
        api._check(api.lib().solar_gpu_sg_im2col(_p(x), 3, Hi, Wi, Cin, Kp, _p(cols), None))
        pad = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
        taps = [pad[:, ky: ky + Hi: 2, kx: kx + Wi: 2] for ky in range(4) for kx in range(4)]
        want = torch.stack(taps, 3).reshape(-1, 16 * Cin)
        assert torch.equal(cols[:, :16 * Cin], want)
        assert not cols[:, 16 * Cin:].any()
