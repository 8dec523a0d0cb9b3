"""GPU: each kernel through the C ABI against the CPU oracle on the same seeded inputs."""
import ctypes as C
import os

import numpy as np
import pytest
import torch

from helpers import GOLDEN, rel_err
from oracle import quant_oracle as qo
from oracle.rwkv7_oracle import Oracle

pytestmark = pytest.mark.gpu


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _gemv(pm, x):
    from albatross_b200 import _lib
    y = torch.empty(pm.n_out, dtype=torch.float16, device="cuda")
    mat = pm.as_mat()
    _lib.check(_lib.lib.ab_gemv(C.byref(mat), x.data_ptr(), y.data_ptr(), _stream()), "ab_gemv")
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    return y


@pytest.mark.parametrize("fmt", ["int8", "nvfp4"])
@pytest.mark.parametrize("shape", [(64, 256), (100, 768), (257, 4096)])
def test_dequantised_weights_bit_exact(fmt, shape):
    """The kernels' in-register de-quantisation equals the specification bit for bit."""
    from albatross_b200 import quant
    torch.manual_seed(3)
    w = torch.randn(*shape) * 0.02
    w[1] = 0
    pm = quant.quantize(w.cuda(), fmt)
    want = qo.fake_quantize(w.numpy(), fmt)
    got = pm.dequantize().cpu().numpy()
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


def test_int8_col_scale_dequant_bit_exact():
    from albatross_b200 import quant
    torch.manual_seed(4)
    w = torch.randn(64, 512) * 0.02
    c = qo.int8_col_scale(w.numpy())
    pm = quant.quantize_int8(w.cuda(), torch.from_numpy(c).cuda())
    q, s = qo.int8_quantize(w.numpy(), c)
    assert np.array_equal(pm.w.cpu().numpy(), q)
    assert np.array_equal(pm.dequantize().cpu().numpy(), qo.int8_dequantize(q, s, c))


def test_gemv_int8_config1_against_reference_fixture():
    """Baseline config 1: x fp16 [1,4096] ~N(0,1), W fp16 [4096,4096] ~N(0,0.02), seed 0."""
    from albatross_b200 import quant
    g = np.load(os.path.join(GOLDEN, "gemv_int8_4096.npz"))
    torch.manual_seed(0)
    x = torch.randn(1, 4096).half()
    w = (torch.randn(4096, 4096) * 0.02).half()
    pm = quant.quantize_int8(w.cuda())
    y = _gemv(pm, x.cuda().view(-1)).float().cpu().numpy()
    assert rel_err(y, g["y"][0]) < 2e-3          # fp16 output rounding; the integer sums are exact
    c = torch.from_numpy(qo.int8_col_scale(w.float().numpy())).cuda()
    pm2 = quant.quantize_int8(w.cuda(), c)
    y2 = _gemv(pm2, x.cuda().view(-1)).float().cpu().numpy()
    assert rel_err(y2, g["y_colscale"][0]) < 2e-3


@pytest.mark.parametrize("fmt", ["int8", "nvfp4", "none"])
@pytest.mark.parametrize("n,k", [(8, 256), (61, 768), (4096, 1024), (1000, 16384), (5, 3072)])
def test_gemv_against_oracle(fmt, n, k):
    """Ragged row counts (not a multiple of the rows per warp), K not a multiple of the 1024 tile."""
    from albatross_b200 import quant
    torch.manual_seed(n * 31 + k)
    w = torch.randn(n, k) * 0.02
    x = torch.randn(k).half()
    x[::97] *= 30                                    # activation outliers
    pm = quant.quantize(w.cuda(), None if fmt == "none" else fmt)
    wq = qo.fake_quantize(w.half().float().numpy() if fmt == "none" else w.numpy(), fmt)
    want = wq.astype(np.float64) @ x.double().numpy()
    got = _gemv(pm, x.cuda()).float().cpu().numpy()
    assert rel_err(got, want) < 3e-3


def test_gemv_zero_and_linearity():
    from albatross_b200 import quant
    torch.manual_seed(9)
    w = torch.randn(512, 1024) * 0.02
    pm = quant.quantize_int8(w.cuda())
    z = _gemv(pm, torch.zeros(1024, dtype=torch.float16, device="cuda"))
    assert torch.count_nonzero(z) == 0
    x = torch.randn(1024).half().cuda()
    y1 = _gemv(pm, x).float()
    y2 = _gemv(pm, (x * 2)).float()                  # scaling by 2 is exact in fp16 and in the fixed-point split
    assert torch.equal(y2, y1 * 2)


@pytest.mark.parametrize("B,T,H", [(1, 1, 2), (3, 1, 4), (2, 7, 2), (1, 33, 1)])
def test_wkv7_operator_against_oracle(B, T, H):
    """Same contract as the reference operator: state updated in place, y returned."""
    from albatross_b200 import RWKV7_BATCH_OP, RWKV7_OP
    torch.manual_seed(B * 100 + T)
    Cn = H * 64
    f = lambda s=1.0: (torch.randn(B, T, Cn) * s).half()
    r, k, v = f(), f(), f()
    w = (-torch.nn.functional.softplus(-torch.randn(B, T, Cn)) - 0.5).half()
    kk = torch.nn.functional.normalize(torch.randn(B, T, H, 64), dim=-1).view(B, T, Cn).half()
    a, b = -kk, (kk * torch.sigmoid(torch.randn(B, T, Cn)).half())
    S0 = torch.randn(B, H, 64, 64) * 0.1
    S_ref = S0.clone()
    y_ref = Oracle.wkv7_kernel(S_ref, r, w, k, v, a, b)
    S = S0.clone().cuda()
    dev = [t.cuda().contiguous() for t in (r, w, k, v, a, b)]
    y = RWKV7_BATCH_OP(S, *dev)
    torch.cuda.synchronize()
    assert rel_err(y.float().cpu(), y_ref.float()) < 2e-3
    assert rel_err(S.cpu(), S_ref) < 1e-4
    if B == 1:                                        # the unbatched wrapper takes [T,C] and [H,64,64]
        S1 = S0[0].clone().cuda()
        y1 = RWKV7_OP(S1, *[t[0].contiguous() for t in dev])
        assert torch.equal(y1, y[0]) and torch.equal(S1, S[0])


@pytest.mark.parametrize("T", [2, 7, 8, 9, 16, 31, 33, 41, 130])
@pytest.mark.parametrize("B,H,shift", [(1, 2, 0), (3, 1, 0), (1, 1, 1)])
def test_wkv7_sequences_around_the_chunk_size(B, H, T, shift):
    """The sequence kernel works in chunks of 8 steps through a ring of four: lengths around both, several sequences, and
    inputs on odd 2-byte boundaries (shift = 1), which take the plain kernel. Bound: y is rounded to fp16 once (2**-11 of
    the value); the state differs by the order of fp32 sums only."""
    from albatross_b200 import RWKV7_BATCH_OP
    torch.manual_seed(T * 10 + B)
    Cn = H * 64
    kk = torch.nn.functional.normalize(torch.randn(B, T, H, 64), dim=-1).view(B, T, Cn)
    vec = [torch.randn(B, T, Cn), -torch.nn.functional.softplus(-torch.randn(B, T, Cn)) - 0.5, torch.randn(B, T, Cn),
           torch.randn(B, T, Cn), -kk, kk * torch.sigmoid(torch.randn(B, T, Cn))]
    vec = [v.half() for v in vec]
    S0 = torch.randn(B, H, 64, 64) * 0.3
    S_ref = S0.clone()
    y_ref = Oracle.wkv7_kernel(S_ref, *vec)
    S, dev = S0.cuda(), []
    for v in vec:
        buf = torch.empty(v.numel() + shift, dtype=torch.float16, device="cuda")
        buf[shift:] = v.flatten().cuda()
        dev.append(buf[shift:].view(B, T, Cn))
    y = RWKV7_BATCH_OP(S, *dev)
    torch.cuda.synchronize()
    from albatross_b200 import _lib
    assert _lib.device_status() == 0
    assert rel_err(y.float().cpu(), y_ref.float()) < 2e-3
    assert rel_err(S.cpu(), S_ref) < 1e-5


@pytest.mark.parametrize("T", [2, 8, 9, 40, 67])
def test_wkv7_sequences_do_not_depend_on_the_batch(T):
    """A head's result does not depend on the other sequences of the call or on where its block runs, and a sequence cut into
    calls of any length gives the same bits: step by step (the plain kernel), and in two calls that end inside a chunk."""
    from albatross_b200 import RWKV7_BATCH_OP, _lib
    torch.manual_seed(T)
    B, H = 40, 2
    kk = torch.nn.functional.normalize(torch.randn(B, T, H, 64), dim=-1).view(B, T, H * 64)
    vec = [torch.randn(B, T, H * 64), -torch.rand(B, T, H * 64) * 2 - 0.5, torch.randn(B, T, H * 64), torch.randn(B, T, H * 64), -kk,
           kk * torch.rand(B, T, H * 64)]
    vec = [v.half().cuda() for v in vec]
    S0 = torch.randn(B, H, 64, 64, device="cuda") * 0.3
    S_all = S0.clone()
    y_all = RWKV7_BATCH_OP(S_all, *vec)
    for b in (0, 17, 39):
        S = S0[b:b + 1].clone()
        y = RWKV7_BATCH_OP(S, *[v[b:b + 1].contiguous() for v in vec])
        assert torch.equal(y, y_all[b:b + 1]) and torch.equal(S, S_all[b:b + 1])
        S = S0[b:b + 1].clone()
        for t in range(T):
            yt = RWKV7_BATCH_OP(S, *[v[b:b + 1, t:t + 1].contiguous() for v in vec])
            assert torch.equal(yt, y_all[b:b + 1, t:t + 1])
        assert torch.equal(S, S_all[b:b + 1])
        cut = 3 * T // 5                               # 67 = 40 + 27, 40 = 24 + 16, 9 = 5 + 4, 8 = 4 + 4, 2 = 1 + 1
        S = S0[b:b + 1].clone()
        ys = [RWKV7_BATCH_OP(S, *[v[b:b + 1, t0:t1].contiguous() for v in vec]) for t0, t1 in ((0, cut), (cut, T))]
        assert torch.equal(torch.cat(ys, 1), y_all[b:b + 1]) and torch.equal(S, S_all[b:b + 1])
    assert _lib.device_status() == 0


def test_wkv7_operator_rejects_bad_shapes():
    from albatross_b200 import _lib
    assert _lib.lib.ab_wkv7_fwd(1, 1, 96, 2, 16, 16, 16, 16, 16, 16, 16, 16, None) == -1
    assert b"C == H*64" in _lib.lib.ab_last_error()


def _gemm(pm, x, epi=0, resid=None):
    from albatross_b200 import _lib
    rows = x.shape[0]
    y = torch.empty(rows, pm.n_out, dtype=torch.float16, device="cuda")
    mat = pm.as_mat()
    scratch = torch.zeros(max(256, _lib.lib.ab_gemm_scratch_bytes(C.byref(mat), rows)), dtype=torch.uint8, device="cuda")
    _lib.check(_lib.lib.ab_gemm(C.byref(mat), rows, x.data_ptr(), y.data_ptr(), epi,
                                None if resid is None else resid.data_ptr(), scratch.data_ptr(), _stream()), "ab_gemm")
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    return y


@pytest.mark.parametrize("fmt", ["int8", "nvfp4", "none"])
@pytest.mark.parametrize("rows,n,k", [(1, 128, 64), (3, 200, 256), (17, 128, 768), (64, 1000, 1024), (320, 512, 4096),
                                      (300, 130, 3072), (400, 256, 512), (320, 256, 16384)])
def test_batched_product_against_oracle(fmt, rows, n, k):
    """Tensor-core path: ragged batch (not a multiple of 16), ragged output rows (not a multiple of 128),
    batch 320 (two MMAs of N = 160) and more than one batch tile (400 rows)."""
    from albatross_b200 import quant
    torch.manual_seed(rows * 7 + n + k)
    w = torch.randn(n, k) * 0.02
    x = torch.randn(rows, k).half()
    pm = quant.quantize(w.cuda(), None if fmt == "none" else fmt)
    wq = qo.fake_quantize(w.half().float().numpy() if fmt == "none" else w.numpy(), fmt)
    want = x.double().numpy() @ wq.astype(np.float64).T
    got = _gemm(pm, x.cuda()).float().cpu().numpy()
    assert rel_err(got, want) < 3e-3


@pytest.mark.parametrize("rows", [16, 32, 48, 80, 100, 130, 200, 256])
def test_batched_product_split_k_batch_sizes(rows):
    """Few output tiles and a long K loop: split K. The batch size sets how much shared memory a block has for the
    other blocks' partial sums (for some sizes the split is narrowed to make one chunk's slices fit), whether the
    last 32-row chunk is ragged, and how many chunks each block of a tile finishes. With and without the residual
    epilogue; a second call must reproduce the first bit for bit (fixed summation order)."""
    from albatross_b200 import _lib, quant
    torch.manual_seed(rows)
    n, k = 256, 4096
    w = torch.randn(n, k) * 0.02
    x = torch.randn(rows, k).half()
    resid = torch.randn(rows, n).half()
    pm = quant.quantize(w.cuda(), "nvfp4")
    base = x.double().numpy() @ qo.fake_quantize(w.numpy(), "nvfp4").astype(np.float64).T
    for epi, want in ((_lib.EPI_NONE, base), (_lib.EPI_RESID, base + resid.double().numpy())):
        r = resid.cuda() if epi == _lib.EPI_RESID else None
        got = _gemm(pm, x.cuda(), epi, r)
        assert rel_err(got.float().cpu().numpy(), want) < 3e-3
        assert torch.equal(_gemm(pm, x.cuda(), epi, r), got)


@pytest.mark.parametrize("rows", [321, 400, 511, 640, 768, 1025])
@pytest.mark.parametrize("fmt,n,k,epi", [("int8", 4096, 512, 0), ("nvfp4", 300, 1024, 4), ("none", 16384, 128, 3)])
def test_batched_product_tall_batches(fmt, n, k, epi, rows):
    """More rows than one tile: whatever tile height the launcher picks, with a ragged last tile, residual and relu^2."""
    from albatross_b200 import quant
    torch.manual_seed(rows)
    w = torch.randn(n, k, device="cuda") * 0.02
    x, resid = torch.randn(rows, k, device="cuda").half(), torch.randn(rows, n, device="cuda").half()
    pm = quant.quantize(w, None if fmt == "none" else fmt)
    want = x.double() @ pm.dequantize().double().t()
    want = torch.relu(want) ** 2 if epi == 3 else want + resid.double() if epi == 4 else want
    got = _gemm(pm, x, epi, resid if epi == 4 else None)
    assert rel_err(got.float().cpu().numpy(), want.cpu().numpy()) < 4e-3     # fp16 output rounding, as in the tests above


@pytest.mark.parametrize("fmt,rows,n,k", [("none", 320, 4096, 4096), ("int8", 320, 2048, 4096), ("nvfp4", 320, 2048, 8192),
                                          ("none", 256, 2048, 4160), ("none", 100, 256, 4160), ("int8", 128, 512, 4160), ("int8", 40, 300, 8256), ("nvfp4", 40, 300, 8512)])
def test_batched_product_recycles_its_weight_slots(fmt, rows, n, k):
    """The weight slots in shared memory are reused many times while copies complete in any order (tall batches leave the
    fewest slots; one, two or four k-steps of 64 inputs per slot, the last slot partly used): every launch gives the same
    bits, and the right ones."""
    from albatross_b200 import quant
    torch.manual_seed(rows + k)
    w = torch.randn(n, k, device="cuda") * 0.02
    x = torch.randn(rows, k, device="cuda").half()
    pm = quant.quantize(w, None if fmt == "none" else fmt)
    want = (x.double() @ pm.dequantize().double().t()).cpu().numpy()
    got = _gemm(pm, x)
    assert rel_err(got.float().cpu().numpy(), want) < 3e-3          # fp16 output rounding, as in the tests above
    for _ in range(20):
        assert torch.equal(_gemm(pm, x), got)


@pytest.mark.parametrize("fmt,rows,n,k", [("none", 768, 12288, 4096), ("none", 320, 8192, 4096), ("none", 100, 16384, 2048), ("int8", 768, 12288, 4096),
                                          ("nvfp4", 768, 12288, 4096)])
def test_batched_product_reads_its_weight_slots_before_it_gives_them_back(fmt, rows, n, k):
    """A slot of weights is refilled as soon as the warps that read it say so. With fp16 weights a piece of a row was now and
    then that of the refill (768 x 12288 x 4096: in one call of two); so call after call has to give the same bits, and those within
    one rounding of the product (fp16: 2**-11 of a value) plus fp32 sums (k / 16 additions, each off by 2**-23 of a sum below 8)."""
    from albatross_b200 import quant
    torch.manual_seed(n + rows)
    pm = quant.quantize((torch.randn(n, k, device="cuda") * 0.02), None if fmt == "none" else fmt)
    x = torch.randn(rows, k, device="cuda").half()
    first = _gemm(pm, x, 0, None)
    want = x.double() @ pm.dequantize().double().t()
    assert ((first.double() - want).abs() <= 2 ** -11 * 1.02 * want.abs() + k / 16 * 8 * 2 ** -23).all()
    assert all(torch.equal(_gemm(pm, x, 0, None), first) for _ in range(60))


def test_batched_product_small_k_and_epilogues():
    """Adapter-sized products (K = 16 ... 480, not multiples of the 64-input k-step) and the fused epilogues."""
    from albatross_b200 import _lib, quant
    torch.manual_seed(5)
    for k in (16, 48, 96, 480):
        w = torch.randn(256, k) * 0.1
        x = torch.randn(20, k).half()
        pm = quant.pack_fp16(w.cuda())
        want = x.double().numpy() @ w.half().double().numpy().T
        assert rel_err(_gemm(pm, x.cuda()).float().cpu().numpy(), want) < 3e-3
    w = torch.randn(192, 256) * 0.05
    x = torch.randn(33, 256).half()
    pm = quant.quantize_int8(w.cuda())
    base = x.double().numpy() @ qo.fake_quantize(w.numpy(), "int8").astype(np.float64).T
    resid = torch.randn(33, 192).half()
    for epi, fn in ((_lib.EPI_TANH, np.tanh), (_lib.EPI_SIGMOID, lambda v: 1 / (1 + np.exp(-v))),
                    (_lib.EPI_RELU2, lambda v: np.maximum(v, 0) ** 2), (_lib.EPI_RESID, lambda v: v + resid.double().numpy())):
        got = _gemm(pm, x.cuda(), epi, resid.cuda() if epi == _lib.EPI_RESID else None).float().cpu().numpy()
        assert rel_err(got, fn(base)) < 4e-3


def test_device_sampler_matches_argsort():
    """ab_sample_rows: noise 0 is the arg-max the reference takes from a descending argsort; with noise the chosen
    logit is within `noise` of the row maximum and the draw is reproducible per seed."""
    from albatross_b200 import sampler_simple_batch
    torch.manual_seed(2)
    for rows, V in ((1, 65536), (320, 65536), (7, 1000), (3, 37)):
        logits = (torch.randn(rows, V, device="cuda") * 3).half()
        logits[0, min(V - 1, 11)] = logits[0].max() + 1                       # a clear winner in row 0
        got = sampler_simple_batch(logits, noise=0.0)
        want = torch.argsort(logits.float(), dim=-1, descending=True, stable=True)[:, :1]
        assert got.shape == (rows, 1) and got.dtype == torch.int64
        assert torch.equal(got, want)
        a = sampler_simple_batch(logits, noise=1.0, seed=5)
        b = sampler_simple_batch(logits, noise=1.0, seed=5)
        c = sampler_simple_batch(logits, noise=1.0, seed=6)
        assert torch.equal(a, b)
        picked = logits.float().gather(1, a)
        assert (picked >= logits.float().max(dim=1, keepdim=True).values - 1.0).all()
        if rows * V > 100000:
            assert not torch.equal(a, c)
    ties = torch.zeros(2, 64, device="cuda").half()
    assert sampler_simple_batch(ties, noise=0.0).flatten().tolist() == [0, 0]  # ties go to the lowest index
    # ids written by the kernel straight into pinned host memory (no copy of their own)
    pinned = torch.full((3, 1), -1, dtype=torch.int64).pin_memory()
    logits = torch.randn(3, 1000, device="cuda").half()
    ret = sampler_simple_batch(logits, noise=0.0, out=pinned)
    torch.cuda.current_stream().synchronize()
    assert ret.data_ptr() == pinned.data_ptr() and pinned.flatten().tolist() == logits.float().argmax(-1).tolist()


def _noisy_argmax(logits, noise, seed):
    """The sampler's definition in numpy: first index of the largest logit + noise * hash(seed, row, column), in fp32."""
    x = logits.cpu().float().numpy()
    rows, V = x.shape
    u32 = np.uint32
    with np.errstate(over="ignore"):
        h = u32(seed) ^ (np.arange(rows, dtype=u32)[:, None] * u32(0x9E3779B9)) ^ (np.arange(V, dtype=u32)[None] * u32(0x85EBCA6B))
        h ^= h >> u32(16); h *= u32(0x7FEB352D); h ^= h >> u32(15); h *= u32(0x846CA68B); h ^= h >> u32(16)
    u = (h >> u32(8)).astype(np.float32) * np.float32(1.0 / 16777216.0)
    v = x + np.float32(noise) * u if noise > 0 else x
    v = np.where(np.isnan(v), -np.inf, v)
    best = v.max(axis=1, keepdims=True)
    ok = (v == best) & ~np.isnan(x)
    return ok.argmax(axis=1)


@pytest.mark.parametrize("rows", [1, 16, 17, 40])
@pytest.mark.parametrize("V", [1, 7, 8, 37, 1000, 4096, 8191, 32776, 50277])
@pytest.mark.parametrize("kind", ["normal", "ties", "infinite", "flat"])
def test_device_sampler_exact(rows, V, kind):
    """Rows on any 2-byte boundary, sizes around the 16-byte chunks and the batches, ties, infinities, NaNs: the same id
    as the definition, for every noise."""
    from albatross_b200 import sampler_simple_batch
    g = torch.Generator().manual_seed(rows * V)
    x = torch.randn(rows, V, generator=g) * 3
    if kind == "ties":
        x = x.round()
    if kind == "infinite" and V > 1:
        x[:, ::3] = -float("inf")
        x[:, V // 2] = float("nan")
        x[0] = -float("inf")
        if rows > 1:
            x[1, V - 1] = float("inf")
    if kind == "flat":
        x = torch.full((rows, V), -1.5)
    x = x.half()
    for noise in (0.0, 0.01, 1.0, 50.0):
        got = sampler_simple_batch(x.cuda(), noise=noise, seed=9)
        assert got.flatten().tolist() == _noisy_argmax(x, noise, 9).tolist(), (noise, kind)


@pytest.mark.parametrize("D,B,T", [(D, B, T) for D in (128, 256, 768, 4096, 5120) for B, T in ((1, 2), (3, 5), (2, 260), (5, 410))] +
                         [(256, 3, 171), (4096, 3, 171), (8192, 3, 5), (8192, 3, 171), (8192, 5, 410)])
def test_sequence_norm_and_lerps_through_a_model(B, T, D):
    """The one-pass norm + token-shift kernel (1 row per block, 2 from 512 rows, 4 from 2048; row lengths up to its limit of
    8192): the state it hands over after T tokens is the normalised last row; a prefix gives what its tokens give one by one
    (other kernels); and a prompt gives, at every position and in every state, what it gives in pieces of under 512 rows,
    which one-row blocks work on (171 = 3 mod 4 tokens and 410 = 2 mod 4: the last block of a sequence is not full)."""
    from albatross_b200 import RWKV_x070, synth
    import types
    cfg = (1, D, 64, (16, 16, 16, 16))
    args = types.SimpleNamespace(MODEL_NAME="", n_layer=1, n_embd=D, head_size=64, vocab_size=64)
    model = RWKV_x070(args, quant="int8", state_dict=dict(synth.iter_checkpoint(cfg, seed=D, device="cuda")))
    g = torch.Generator().manual_seed(T)
    ids = torch.randint(0, 64, (B, T), generator=g).tolist()
    _, st = model.forward_batch(ids, None)
    z = model.z
    last = z["emb.weight"][torch.tensor([r[-1] for r in ids])].float()
    want = torch.nn.functional.layer_norm(last, (D,), z["blocks.0.ln1.weight"].float(), z["blocks.0.ln1.bias"].float())
    assert rel_err(st[0].float().cpu(), want.cpu()) < 1e-3          # one fp16 rounding
    one = None
    for t in range(min(T, 12)):                                     # a prefix, token by token through the T = 1 kernels
        _, one = model.forward_batch([[r[t]] for r in ids], one)
    _, pre = model.forward_batch([r[:min(T, 12)] for r in ids], None)
    for a, b in zip(pre, one):
        assert rel_err(a.float().cpu(), b.float().cpu()) < 1e-2     # fp16 activations along two kernel families
    if B * T >= 512:
        whole, st = model.forward_batch(ids, None, True)            # logits of every position
        parts, pst, n = [], None, 500 // B
        for t in range(0, T, n):
            lg, pst = model.forward_batch([r[t:t + n] for r in ids], pst, True)
            parts.append(lg.view(B, -1, 64))
        parts = torch.cat(parts, 1).float()
        # The products of other row counts sum in another order, which moves fp16 roundings of the block's dozen stages (2**-11
        # each, of the largest value at most); a wrong token-shift row changes its position by as much as the logits themselves.
        assert rel_err(whole.view(B, T, 64).float().cpu(), parts.cpu()) < 2e-2
        for a, b in zip(st, pst):
            assert rel_err(a.float().cpu(), b.float().cpu()) < 2e-2


@pytest.mark.parametrize("fmt", ["int8", "nvfp4", "none"])
@pytest.mark.parametrize("rows,n,k", [(1, 64, 64), (7, 300, 192), (8, 4096, 320), (8, 129, 4096), (5, 4100, 448), (8, 1024, 16384), (9, 1000, 1024),
                                      (16, 96, 4096), (13, 2560, 2560), (17, 768, 768), (24, 1000, 2048), (24, 31, 12288)])
def test_products_of_few_rows(fmt, rows, n, k):
    """The kernel for up to 24 rows at its edges: ragged weight tiles (32 rows) and row pieces (128 bytes: 64, 128 or 256
    inputs), one to three groups of eight batch rows, K split over the blocks of a cluster, NVFP4 scales with and without a
    tensor map (k a multiple of 256 or not), every epilogue; a second call gives the same bits. Bound: one fp16 rounding of the
    product (2**-11), one more by the epilogue, and fp32 sums."""
    from albatross_b200 import quant
    torch.manual_seed(rows * 7 + n + k)
    pm = quant.quantize((torch.randn(n, k) * 0.02).cuda(), None if fmt == "none" else fmt)
    x, r = torch.randn(rows, k).half().cuda(), torch.randn(rows, n).half().cuda()
    want = x.double() @ pm.dequantize().double().t()
    fns = [lambda t: t, torch.tanh, torch.sigmoid, lambda t: torch.relu(t) ** 2, lambda t: t + r.double()]
    for epi, fn in enumerate(fns):
        got = _gemm(pm, x, epi, r if epi == 4 else None)
        ref = fn(want)
        assert rel_err(got.double().cpu(), ref.cpu()) < 2e-3, epi
        assert ((got.double() - ref).norm() / ref.norm()).item() < 2 ** -10.5, epi
        assert torch.equal(_gemm(pm, x, epi, r if epi == 4 else None), got)


def test_products_of_few_rows_leave_their_neighbours_alone():
    """Outputs beyond the last row and column stay as they were (ragged rows and columns are clipped, not written)."""
    from albatross_b200 import _lib, quant
    torch.manual_seed(3)
    for rows, n, k in ((3, 70, 512), (9, 33, 256), (8, 4099, 128)):
        pm = quant.quantize((torch.randn(n, k) * 0.02).cuda(), "int8")
        mat, x = pm.as_mat(), torch.randn(rows, k).half().cuda()
        buf = torch.full((rows * n + 64,), 7.0, dtype=torch.float16, device="cuda")
        scratch = torch.zeros(max(256, _lib.lib.ab_gemm_scratch_bytes(C.byref(mat), rows)), dtype=torch.uint8, device="cuda")
        _lib.check(_lib.lib.ab_gemm(C.byref(mat), rows, x.data_ptr(), buf.data_ptr(), 0, None, scratch.data_ptr(), _stream()), "ab_gemm")
        torch.cuda.synchronize()
        assert _lib.device_status() == 0
        assert torch.equal(buf[rows * n:], torch.full_like(buf[rows * n:], 7.0))
        assert rel_err(buf[:rows * n].view(rows, n).double().cpu(), (x.double() @ pm.dequantize().double().t()).cpu()) < 2e-3


@pytest.mark.parametrize("rows", [1, 16, 17, 148, 149])
@pytest.mark.parametrize("V", [1, 9, 8191, 8200, 16384, 16393, 32777])
def test_sampler_at_the_edges_of_its_batches(rows, V):
    """Row lengths around a batch of each kernel (16 K logits of 512 threads, 8 K of 256, 64 K of 1024), rows that start off a
    16-byte boundary, and the row counts where the kernel changes. Whole numbers: the same ids as torch."""
    from albatross_b200 import sampler_simple_batch
    g = torch.Generator().manual_seed(rows + V)
    logits = (torch.randn(rows, V, generator=g) * 3).half()
    logits[:, V // 3] = logits.max() + 1                     # a winner whose position is known ...
    logits[rows // 2, V - 1] = logits.max() + 1              # ... and one in the last place
    dev = logits.cuda()
    assert torch.equal(sampler_simple_batch(dev, noise=0.0).flatten().cpu(), logits.float().argmax(1))
    a = sampler_simple_batch(dev, noise=0.5, seed=3).flatten().cpu()     # noise below the winner's margin of 1
    assert torch.equal(a, logits.float().argmax(1))


@pytest.mark.parametrize("fmt,rows,n,k", [("int8", 8, 65536, 2048), ("none", 8, 4096, 4096), ("nvfp4", 8, 65536, 2048), ("none", 16, 2560, 2560), ("nvfp4", 5, 8192, 4288)])
def test_products_of_few_rows_read_a_piece_before_it_is_asked_for_again(fmt, rows, n, k):
    """A warp's stages of weights are refilled as soon as it has read them: call after call the same bits, and those within one
    rounding of the product (fp16: 2**-11 of a value) plus fp32 sums (k / 16 additions, each off by 2**-23 of a sum below 8)."""
    from albatross_b200 import quant
    torch.manual_seed(n + rows)
    pm = quant.quantize((torch.randn(n, k, device="cuda") * 0.02), None if fmt == "none" else fmt)
    x = torch.randn(rows, k, device="cuda").half()
    first = _gemm(pm, x, 0, None)
    want = x.double() @ pm.dequantize().double().t()
    assert ((first.double() - want).abs() <= 2 ** -11 * 1.02 * want.abs() + k / 16 * 8 * 2 ** -23).all()
    assert all(torch.equal(_gemm(pm, x, 0, None), first) for _ in range(100))


@pytest.mark.parametrize("which,first,end", [
    (0, 0x3f800000, 0x7e800000), (0, 0x7fc00000, 0x80000000),                              # 1 <= d < 2^126, NaN
    (1, 0x21800000, 0x5d800000), (1, 0, 1), (1, 0x7f800000, 0x7f800001), (1, 0x7fc00000, 0x80000000),   # 2^-60 <= x < 2^60, 0, infinity, NaN
    (2, 0, 0x7c01 << 16), (2, 0x7e00 << 16, 0x8000 << 16)])                                # norms from 0 (1e-12) to infinity, NaN; every numerator
def test_glue_arithmetic_equals_the_operators(which, first, end):
    """Reciprocal, root and quotient of the per-step glue have the bits of `1.f / d`, `sqrtf(x)` and `x / d` for every operand they
    may be given: all floats of the range, and all pairs of an fp16 numerator and an fp16 norm."""
    from albatross_b200 import _lib
    differ = torch.zeros(1, dtype=torch.int64, device="cuda")
    _lib.check(_lib.lib.ab_glue_selftest(which, first, end - first, differ.data_ptr(), _stream()), "ab_glue_selftest")
    assert differ.item() == 0


@pytest.mark.parametrize("B,T,H", [(74, 41, 2), (75, 41, 2), (37, 19, 4), (38, 19, 4), (160, 33, 1)])
def test_wkv7_sequences_are_the_same_in_both_block_forms(B, T, H):
    """Up to 148 heads (one per SM) a sequence runs in a wide block, beyond that in a narrow one; over several chunks of eight steps
    and a cut one, a sequence gives the same bits alone (wide) and in batches on either side of the line."""
    from albatross_b200 import _lib
    torch.manual_seed(B + T)
    C_ = 64 * H
    kk = torch.nn.functional.normalize(torch.randn(B, T, H, 64), dim=-1).view(B, T, C_)
    ins = [torch.randn(B, T, C_), -torch.rand(B, T, C_) * 2 - 0.5, torch.randn(B, T, C_), torch.randn(B, T, C_), -kk, kk * torch.rand(B, T, C_)]
    ins = [t.half().cuda() for t in ins]
    state = torch.randn(B, H, 64, 64, device="cuda") * 0.3

    def run(sl):
        st, y = state[sl].clone(), torch.empty_like(ins[0][sl])
        args = [t[sl].contiguous() for t in ins]
        _lib.check(_lib.lib.ab_wkv7_fwd(st.shape[0], T, C_, H, st.data_ptr(), *[t.data_ptr() for t in args], y.data_ptr(), _stream()), "ab_wkv7_fwd")
        return y, st
    whole = run(slice(0, B))
    for b in (0, B // 2, B - 1):
        alone = run(slice(b, b + 1))
        assert torch.equal(whole[0][b:b + 1], alone[0]) and torch.equal(whole[1][b:b + 1], alone[1])
    assert torch.isfinite(whole[0].float()).all() and _lib.device_status() == 0


@pytest.mark.parametrize("fmt,rows,n,k", [("int8", 8, 65536, 2048), ("nvfp4", 2, 65536, 2048), ("int8", 2, 65536, 4096), ("nvfp4", 8, 65536, 4096), ("int8", 8, 37901, 1024),
                                          ("nvfp4", 3, 37901, 1024), ("int8", 8, 16384, 4096), ("nvfp4", 8, 16384, 4096), ("int8", 8, 4096, 16384)])
def test_products_of_few_rows_over_several_rounds_of_tiles(fmt, rows, n, k):
    """A block's warps work through more tiles than they hold at a time (the vocabulary head, wide feed-forwards): the request cursor
    moves on to the next tile, stage and phase bit are carried across tiles, and partial sums are read before the next tile's
    are written. 37901 rows: one more than eight tiles of 32 rows for every warp of 148 SMs, and a ragged end. Every epilogue; bounds as above."""
    from albatross_b200 import quant
    torch.manual_seed(n + k + rows)
    pm = quant.quantize((torch.randn(n, k, device="cuda") * 0.02), fmt)
    x, r = torch.randn(rows, k).half().cuda(), torch.randn(rows, n).half().cuda()
    want = x.double() @ pm.dequantize().double().t()
    for epi, fn in ((0, lambda t: t), (3, lambda t: torch.relu(t) ** 2), (4, lambda t: t + r.double())):
        got = _gemm(pm, x, epi, r if epi == 4 else None)
        ref = fn(want)
        assert rel_err(got.double().cpu(), ref.cpu()) < 2e-3, epi
        assert ((got.double() - ref).norm() / ref.norm()).item() < 2 ** -10.5, epi
        assert torch.equal(_gemm(pm, x, epi, r if epi == 4 else None), got)
