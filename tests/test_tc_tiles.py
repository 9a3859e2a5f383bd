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


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(256, 512, 512), (1, 16, 30), (130, 48, 65), (100, 37, 40), (2560, 512, 24)])
def test_potential_steps_in_the_epilogue(M, N, K):
    """Product and element-wise step in one launch against the product and
    hmc_pot_elementwise, which evaluate the same expressions.  The product is
    equal bit for bit; the step may be contracted differently, so its FP32
    results agree to a few ulp and its BF16 ones to one (2^-7 relative)."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    g = torch.Generator(device="cuda").manual_seed(9)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    x, w = _operand(M, K, 1), _operand(N, K, 2)
    bias, vec, aux, z = rnd(N), rnd(N), rnd(M, N), rnd(M, N)
    pM, pN = _pad(M), _pad(N) + 16
    stream = torch.cuda.current_stream().cuda_stream
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    mm = (M, N, K, x.data_ptr(), x.shape[1], w.data_ptr(), w.shape[1])
    bf = lambda *s: torch.full(s, 7.0, dtype=torch.bfloat16, device="cuda")  # noqa: E731

    for mode in range(5):
        hidden = mode == _lib.HMC_POT_DELTA2
        y, zr = torch.zeros((M, N), device="cuda"), z.clone()
        a1, a1t, want, want_t, wf = bf(M, _pad(N)), bf(N, pM), bf(M, pN), bf(N, pM), torch.zeros((M, N), device="cuda")
        if hidden:
            o = _lib.HmcMlpOut(z=zr.data_ptr(), ldz=N, act=a1.data_ptr(), ld_act=_pad(N), act_t=a1t.data_ptr(), ld_act_t=pM)
            _lib.call("hmc_tc_mlp", _lib.HMC_MLP_HIDDEN, *mm, bias.data_ptr(), ctypes.byref(o), status.data_ptr(), stream)
        else:
            zero = torch.zeros(N, device="cuda")
            o = _lib.HmcMlpOut(y=y.data_ptr(), ldy=N)
            _lib.call("hmc_tc_mlp", _lib.HMC_MLP_OUT, *mm, zero.data_ptr(), ctypes.byref(o), status.data_ptr(), stream)
        _lib.call("hmc_pot_elementwise", mode, M, N, y.data_ptr(), N, zr.data_ptr(), N, aux.data_ptr(), N, vec.data_ptr(),
                  want.data_ptr(), pN, want_t.data_ptr(), pM, wf.data_ptr(), N, stream)

        for transposed in (True, False):
            y2, z2, f2 = torch.zeros((M, N), device="cuda"), z.clone(), torch.zeros((M, N), device="cuda")
            a2, a2t, got, got_t = bf(M, _pad(N)), bf(N, pM), bf(M, pN), bf(N, pM)
            o = _lib.HmcPotOut(z=z2.data_ptr(), ldz=N, act=a2.data_ptr(), ld_act=_pad(N), act_t=a2t.data_ptr(), ld_act_t=pM,
                               out=got.data_ptr(), ld_out=pN, aux=aux.data_ptr(), ld_aux=N, vec=vec.data_ptr(),
                               f=f2.data_ptr(), ld_f=N)
            if transposed:
                o.out_t, o.ld_out_t = got_t.data_ptr(), pM
            if not hidden:
                o.y, o.ldy = y2.data_ptr(), N
            _lib.call("hmc_tc_pot", mode, *mm, bias.data_ptr(), ctypes.byref(o), status.data_ptr(), stream)
            torch.cuda.synchronize()
            assert int(status) == 0
            assert torch.equal(y, y2) and torch.equal(zr, z2)
            if hidden:
                assert torch.equal(a1[:, :N], a2[:, :N]) and torch.equal(a1t[:, :M], a2t[:, :M])
            close = lambda p, q, ulp: bool(((p.float() - q.float()).abs() <= ulp * q.float().abs() + 1e-6).all())  # noqa: E731
            assert close(got[:, :N], want[:, :N], 2.0**-7) and torch.all(got[:, N:] == 7.0)
            assert torch.all(got_t == 7.0) if not transposed else torch.equal(got_t[:, :M], got[:, :N].t())
            assert close(f2, wf, 2.0**-21) if mode == _lib.HMC_POT_DBAR1 else not bool(f2.any())


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [(1,), (300, 7, 70000, 1, 513), (5,) * 8])
def test_adam_of_several_arrays(sizes):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    stream = torch.cuda.current_stream().cuda_stream
    one = [[torch.rand(n, device="cuda") for _ in range(4)] for n in sizes]
    many = [[t.clone() for t in a] for a in one]
    for step in (1, 2):
        for w, g, m, v in one:
            _lib.call("hmc_mlp_adam", w.numel(), w.data_ptr(), g.data_ptr(), m.data_ptr(), v.data_ptr(), 1e-3, 0.9, 0.999, 1e-8,
                      step, stream)
        arrays = (_lib.HmcAdamArray * len(sizes))(*((a[0].numel(), *(t.data_ptr() for t in a)) for a in many))
        _lib.call("hmc_mlp_adam_many", len(sizes), arrays, 1e-3, 0.9, 0.999, 1e-8, step, stream)
    assert all(torch.equal(p, q) for a, b in zip(one, many) for p, q in zip(a, b))
