"""Tensor-core contractions of few tiles (32 matrix rows each) against the same
rows and columns of a product large enough for the wide tiles: the sums run in
the same order, so the results are equal bit for bit.  Sizes sit at the edges of
tiles, of 16-column chunks, of 16-byte stores and of the rule's limit (38 wide
tiles)."""
import ctypes

import pytest

from hmclab_gb300 import _lib

torch = pytest.importorskip("torch")


def _pad(n):
    return (n + 15) // 16 * 16


def _operand(rows, K, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.zeros((rows, _pad(K)), dtype=torch.bfloat16, device="cuda")
    x[:, :K] = torch.randn((rows, K), generator=g, device="cuda").to(torch.bfloat16)
    return x


def _mlp(mode, M, N, K, x, w, bias, ld, scale, shift):
    pM, pN = _pad(M), _pad(N)
    f = lambda *s: torch.full(s, 7.0, dtype=torch.float32, device="cuda")  # noqa: E731
    h = lambda *s: torch.full(s, 7.0, dtype=torch.bfloat16, device="cuda")  # noqa: E731
    out = {"z": f(M, ld), "act": h(M, pN), "act_t": h(N, pM), "y": f(M, ld), "g_state": f(N, M), "g": f(N, M)}
    o = _lib.HmcMlpOut()
    for k, v in out.items():
        setattr(o, k, v.data_ptr())
    o.ldz = o.ldy = ld
    o.ld_act, o.ld_act_t = pN, pM
    o.out_scale, o.out_shift, o.accumulate = scale.data_ptr(), shift.data_ptr(), 1
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.call("hmc_tc_mlp", mode, M, N, K, x.data_ptr(), x.shape[1], w.data_ptr(), w.shape[1], bias.data_ptr(),
              ctypes.byref(o), status.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert int(status) == 0
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (64, 600, 512), (256, 512, 600), (128, 33, 31), (129, 47, 33), (130, 257, 640),
                                   (127, 250, 641), (200, 16, 1300), (128, 9728, 40), (19 * 128, 512, 24)])
def test_few_tiles(M, N, K):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    big_m, big_n = max(M, 20 * 128), max(N, 512)  # 40 wide tiles
    x, w = _operand(big_m, K, 1), _operand(big_n, K, 2)
    g = torch.Generator(device="cuda").manual_seed(3)
    bias, scale, shift = (torch.randn(big_n, generator=g, device="cuda") for _ in range(3))
    for mode in (_lib.HMC_MLP_HIDDEN, _lib.HMC_MLP_OUT, _lib.HMC_MLP_BACK, _lib.HMC_MLP_WGRAD):
        a = _mlp(mode, M, N, K, x[:M], w[:N], bias, N + (N & 1), scale, shift)  # pitches with and without 16-byte rows
        b = _mlp(mode, big_m, big_n, K, x, w, bias, big_n, scale, shift)
        if mode == _lib.HMC_MLP_HIDDEN:
            assert torch.equal(a["z"][:, :N], b["z"][:M, :N]) and not torch.any(a["z"][:, :N] == 7.0)
        if mode in (_lib.HMC_MLP_HIDDEN, _lib.HMC_MLP_BACK):
            assert torch.equal(a["act"][:, :N], b["act"][:M, :N])
            assert torch.equal(a["act_t"][:, :M], b["act_t"][:N, :M])
            assert torch.all(a["act_t"][:, M:] == 7.0)
        if mode == _lib.HMC_MLP_OUT:
            assert torch.equal(a["y"][:, :N], b["y"][:M, :N]) and torch.all(a["y"][:, N:] == 7.0)
            assert torch.equal(a["g_state"], b["g_state"][:N, :M])
            # BF16 products are exact in FP32; K terms of magnitude ~1 accumulate in FP32
            want = x[:M, :K].double() @ w[:N, :K].double().t() + bias[:N].double()
            assert float((a["y"][:, :N].double() - want).abs().max()) <= 2.0**-22 * K * 5.0 + 1e-5
        if mode == _lib.HMC_MLP_WGRAD:
            assert torch.equal(a["g"], b["g"][:N, :M])


@pytest.mark.gpu
@pytest.mark.parametrize("rows,C,K", [(50, 96, 50), (257, 129, 257), (1000, 64, 1000)])
def test_few_tiles_split_products(rows, C, K):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    big_r, big_c = max(rows, 512), 20 * 128

    def product(r, c, ops):
        out = torch.zeros((r, c), device="cuda")
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        _lib.call("hmc_tc_gradient", r, K, c, ops[0].data_ptr(), ops[1].data_ptr(), ops[0].shape[1], ops[2].data_ptr(),
                  ops[3].data_ptr(), ops[2].shape[1], bias.data_ptr(), out.data_ptr(), 0, status.data_ptr(),
                  torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert int(status) == 0
        return out

    ops = [_operand(big_r, K, 1), _operand(big_r, K, 2) / 256, _operand(big_c, K, 3), _operand(big_c, K, 4) / 256]
    bias = torch.randn(big_r, device="cuda")
    assert torch.equal(product(rows, C, ops), product(big_r, big_c, ops)[:rows, :C])
