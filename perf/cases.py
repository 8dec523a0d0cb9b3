"""Performance cases: the calls that programs using this package spend their time in, at the sizes they use.

    listed()          the fixed cases          draw(rng)   one more case of the same ranges
    prepare(case, s)  inputs, weights, state   run(state)  one pass through the public entry points
    work(case)        bytes / flops a pass cannot do without
    tolerance(case)   how far a correct implementation may be off
    exact(case, s)    the same outputs in 64 bits, in plain torch

Kinds of cases:
    decode   one token of one sequence, `RWKV_x070.forward(id, state)`: interactive generation
    step     one token of B sequences, `RWKV_x070.forward_batch([[id], ..], state)`: serving
    prefill  prompts of T tokens, `RWKV_x070.forward([..], state)` (B = 1) or `forward_batch` (B > 1)
    gemv     one quantised matrix times one vector, `ab_gemv`
    gemm     one quantised matrix times a batch of rows with its epilogue, `ab_gemm`
    wkv      the state-update operator alone, `RWKV7_BATCH_OP`
    sample   next-token ids of a batch of logits, `sampler_simple_batch`

The `step` and `prefill` models are two blocks of the network with a small vocabulary (block 0 has no value residual, block
1 has everything): rounding differences grow with depth in a network of random weights, so whole networks appear as
`decode` cases only. States start as in the middle of a text, not at zero.
"""
import ctypes
import types

import torch

from albatross_b200 import RWKV7_BATCH_OP, RWKV_x070, _lib, quant, sampler_simple_batch

EPI = {"none": 0, "tanh": 1, "sigmoid": 2, "relu2": 3, "resid": 4}
FORMATS = ("int8", "nvfp4", "none")


# ------------------------------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------------------------------
def listed():
    return [
        # the smallest model of the family, one token at a time: many short dependent steps
        {"name": "decode_0.1b_int8", "kind": "decode", "L": 12, "D": 768, "V": 65536, "fmt": "int8"},
        # the 7.2B block shapes with four blocks and the full vocabulary: single-stream generation
        {"name": "decode_7.2b_int8", "kind": "decode", "L": 4, "D": 4096, "V": 65536, "fmt": "int8"},
        # a lightly loaded server
        {"name": "step_b8_int8", "kind": "step", "B": 8, "L": 2, "D": 4096, "V": 1024, "fmt": "int8"},
        # an ordinary one
        {"name": "step_b64_nvfp4", "kind": "step", "B": 64, "L": 2, "D": 4096, "V": 1024, "fmt": "nvfp4"},
        # the throughput configuration
        {"name": "step_b320_nvfp4", "kind": "step", "B": 320, "L": 2, "D": 4096, "V": 1024, "fmt": "nvfp4"},
        # a long prompt
        {"name": "prefill_t768_int8", "kind": "prefill", "B": 1, "T": 768, "L": 2, "D": 4096, "V": 1024, "fmt": "int8"},
        # a few short prompts of one (odd) length together
        {"name": "prefill_b5_t37_nvfp4", "kind": "prefill", "B": 5, "T": 37, "L": 2, "D": 4096, "V": 1024, "fmt": "nvfp4"},
        # single products: the smallest one-vector product, the widest batched one, one with few rows and a residual
        {"name": "gemv_int8_4096", "kind": "gemv", "n": 4096, "k": 4096, "fmt": "int8"},
        {"name": "gemm_b320_nvfp4_16384x4096", "kind": "gemm", "rows": 320, "n": 16384, "k": 4096, "fmt": "nvfp4", "epi": "relu2"},
        {"name": "gemm_b24_int8_4096x4096", "kind": "gemm", "rows": 24, "n": 4096, "k": 4096, "fmt": "int8", "epi": "resid"},
        # the operator as prompt processing calls it
        {"name": "wkv_t1024_h64", "kind": "wkv", "B": 1, "T": 1024, "H": 64},
        # greedy decoding with noise for a full batch
        {"name": "sample_b320", "kind": "sample", "B": 320, "V": 65536, "noise": 1.0},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(("decode", "step", "step", "prefill", "prefill", "gemv", "gemm", "gemm", "wkv", "sample"))
    D, fmt = rng.choice((256, 768, 1024, 2048, 2560, 4096)), rng.choice(FORMATS)
    if kind == "decode":
        return {"kind": kind, "L": rng.randint(1, 4), "D": D, "V": rng.choice((1024, 32768, 65536)), "fmt": fmt}
    if kind == "step":
        return {"kind": kind, "B": _log(rng, 2, 320), "L": 2, "D": D, "V": 1024, "fmt": fmt}
    if kind == "prefill":
        B = rng.choice((1, 1, 1, 2, 3, 8))
        return {"kind": kind, "B": B, "T": _log(rng, 2, 768 // B), "L": 2, "D": D, "V": 1024, "fmt": fmt}
    if kind == "gemv":
        return {"kind": kind, "n": _log(rng, 64, 16384), "k": 64 * _log(rng, 4, 256), "fmt": fmt}
    if kind == "gemm":
        return {"kind": kind, "rows": _log(rng, 1, 768), "n": _log(rng, 64, 16384), "k": 64 * _log(rng, 1, 64), "fmt": fmt,
                "epi": rng.choice(tuple(EPI))}
    if kind == "wkv":
        B = _log(rng, 1, 64)
        return {"kind": kind, "B": B, "T": _log(rng, 1, max(1, 1024 // B)), "H": rng.choice((4, 12, 32, 40, 64))}
    return {"kind": kind, "B": _log(rng, 1, 320), "V": rng.choice((1000, 32003, 50277, 65536)), "noise": rng.choice((0.0, 1.0))}


# ------------------------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------------------------
class _Draws:
    """Tensors on the GPU from one seed, in the order they are asked for."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(1000003 * (int(seed) + 1))

    def normal(self, *shape, std=1.0, mean=0.0):
        return torch.empty(shape, device="cuda").normal_(mean, std, generator=self.g)

    def uniform(self, *shape, lo=0.0, hi=1.0):
        return torch.empty(shape, device="cuda").uniform_(lo, hi, generator=self.g)

    def ints(self, n, hi):
        return torch.randint(hi, (n,), device="cuda", generator=self.g).tolist()


def _ranks(D):
    """Adapter ranks (w, a, v, g) of the published sizes, and in between."""
    return {256: (32, 32, 16, 48), 768: (64, 64, 32, 128), 4096: (128, 128, 96, 480)}.get(D, (96, 96, 64, 256))


def _checkpoint(d, L, D, V):
    """A random checkpoint in the reference's key schema (fp32, in the order a loader meets the keys)."""
    rw, ra, rv, rg = _ranks(D)
    z = {"emb.weight": d.normal(V, D), "blocks.0.ln0.weight": d.uniform(D, lo=0.8, hi=1.2), "blocks.0.ln0.bias": d.normal(D, std=0.05)}
    for i in range(L):
        b = "blocks.%d." % i
        a, f = b + "att.", b + "ffn."
        for ln in (b + "ln1", b + "ln2", a + "ln_x"):
            z[ln + ".weight"], z[ln + ".bias"] = d.uniform(D, lo=0.8, hi=1.2), d.normal(D, std=0.05)
        for c in "rwkvag":
            z[a + "x_" + c] = d.uniform(1, 1, D)
        z[a + "w0"], z[a + "a0"] = d.uniform(1, 1, D, lo=-3.0, hi=1.0), d.normal(1, 1, D, std=0.5)
        for n, r in (("w", rw), ("a", ra), ("v", rv), ("g", rg)):
            if n == "v" and i == 0:
                continue
            z[a + n + "1"], z[a + n + "2"] = d.normal(D, r, std=0.02), d.normal(r, D, std=0.1)
        if i > 0:
            z[a + "v0"] = d.normal(1, 1, D, std=0.5)
        z[a + "k_k"], z[a + "k_a"] = d.uniform(1, 1, D, lo=0.7, hi=1.0), d.uniform(1, 1, D, lo=0.8, hi=1.2)
        z[a + "r_k"] = d.normal(D // 64, 64, std=0.1)
        for n in ("receptance", "key", "value", "output"):
            z[a + n + ".weight"] = d.normal(D, D, std=0.02)
        z[f + "x_k"] = d.uniform(1, 1, D)
        z[f + "key.weight"], z[f + "value.weight"] = d.normal(4 * D, D, std=0.02), d.normal(D, 4 * D, std=0.02)
    z["ln_out.weight"], z["ln_out.bias"] = d.uniform(D, lo=0.8, hi=1.2), d.normal(D, std=0.05)
    z["head.weight"] = d.normal(V, D, std=0.02)
    return z


def _state(d, L, D, B):
    """A state in the middle of a text: layer-normalised token-shift rows, a kv state of ordinary size."""
    lead = () if B is None else (B,)
    st = []
    for _ in range(L):
        st += [d.normal(*lead, D).half(), d.normal(*lead, D // 64, 64, 64, std=0.3), d.normal(*lead, D).half()]
    return st


def _model_inputs(case, seed):
    d, kind = _Draws(seed), case["kind"]
    B, T = case.get("B", 1), case.get("T", 1)
    raw = _checkpoint(d, case["L"], case["D"], case["V"])
    alone = kind == "decode" or (kind == "prefill" and B == 1)
    state = _state(d, case["L"], case["D"], None if alone else B)
    ids = d.ints(B * T, case["V"])
    return raw, state, ids, alone


def _product_inputs(case, seed):
    d = _Draws(seed)
    w = d.normal(case["n"], case["k"], std=0.02)
    x = d.normal(case.get("rows", 1), case["k"]).half()
    resid = d.normal(case.get("rows", 1), case["n"]).half()
    return w, x, resid


def _wkv_inputs(case, seed):
    d, B, T, H = _Draws(seed), case["B"], case["T"], case["H"]
    C = H * 64
    r, k, v = (d.normal(B, T, C, std=0.7).half() for _ in range(3))
    w = (-torch.nn.functional.softplus(-d.normal(B, T, C)) - 0.5).half()
    kk = torch.nn.functional.normalize(d.normal(B, T, H, 64), dim=-1).view(B, T, C)
    a, b = (-kk).half(), (kk * torch.sigmoid(d.normal(B, T, C))).half()
    return d.normal(B, H, 64, 64, std=0.3), (r, w, k, v, a, b)


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind in ("decode", "step", "prefill"):
        raw, state, ids, alone = _model_inputs(case, seed)
        args = types.SimpleNamespace(MODEL_NAME="", n_layer=case["L"], n_embd=case["D"], head_size=64, vocab_size=case["V"])
        s["model"] = RWKV_x070(args, quant=None if case["fmt"] == "none" else case["fmt"], state_dict=raw)
        T = case.get("T", 1)
        s["ids"] = ids[0] if kind == "decode" else ids if alone else [ids[i:i + T] for i in range(0, len(ids), T)]
        s["state"], s["alone"] = state, alone
    elif kind in ("gemv", "gemm"):
        w, x, resid = _product_inputs(case, seed)
        pm = s["weights"] = quant.quantize(w, case["fmt"])
        s["mat"] = pm.as_mat()
        s["x"], s["y"] = x, torch.empty(x.shape[0], pm.n_out, dtype=torch.float16, device="cuda")
        if kind == "gemm":
            s["epi"], s["resid"] = EPI[case["epi"]], resid if case["epi"] == "resid" else None
            need = _lib.lib.ab_gemm_scratch_bytes(ctypes.byref(s["mat"]), x.shape[0])
            s["scratch"] = torch.zeros(max(256, need), dtype=torch.uint8, device="cuda")
    elif kind == "wkv":
        s["state"], s["vectors"] = _wkv_inputs(case, seed)
    else:
        s["logits"] = _Draws(seed).normal(case["B"], case["V"], std=3.0).half()
        s["noise"], s["seed"] = case["noise"], int(seed)
    return s


def run(s):
    kind = s["kind"]
    if kind in ("decode", "step", "prefill"):
        forward = s["model"].forward if s["alone"] else s["model"].forward_batch
        logits, s["state"] = forward(s["ids"], s["state"])
        return [logits] + list(s["state"])
    if kind == "gemv":
        _lib.check(_lib.lib.ab_gemv(ctypes.byref(s["mat"]), s["x"].data_ptr(), s["y"].data_ptr(),
                                    torch.cuda.current_stream().cuda_stream), "ab_gemv")
        return s["y"]
    if kind == "gemm":
        resid = s["resid"]
        _lib.check(_lib.lib.ab_gemm(ctypes.byref(s["mat"]), s["x"].shape[0], s["x"].data_ptr(), s["y"].data_ptr(), s["epi"],
                                    None if resid is None else resid.data_ptr(), s["scratch"].data_ptr(),
                                    torch.cuda.current_stream().cuda_stream), "ab_gemm")
        return s["y"]
    if kind == "wkv":
        return RWKV7_BATCH_OP(s["state"], *s["vectors"]), s["state"]
    return sampler_simple_batch(s["logits"], noise=s["noise"], seed=s["seed"])


# ------------------------------------------------------------------------------------------------------------------
# what a pass needs
# ------------------------------------------------------------------------------------------------------------------
_BYTES = {"int8": 1.0, "nvfp4": 0.5625, "none": 2.0}


def work(case):
    kind = case["kind"]
    if kind in ("decode", "step", "prefill"):
        L, D, V, B, T = case["L"], case["D"], case["V"], case.get("B", 1), case.get("T", 1)
        big, ranks = 12 * D * D, _ranks(D)
        adapters = [2 * D * (sum(ranks) - (ranks[2] if i == 0 else 0)) for i in range(L)]
        weights = (L * big + V * D) * _BYTES[case["fmt"]] + 2 * sum(adapters) + L * 20 * 2 * D
        state = B * L * (2 * 4 * 64 * D + 8 * D)
        rows = B * T
        return {"bytes": weights + state + 2 * rows * D + 2 * B * V,
                "flops": 2.0 * rows * (L * big + sum(adapters)) + 2.0 * B * V * D + 7.0 * rows * L * 64 * D}
    if kind in ("gemv", "gemm"):
        n, k, rows = case["n"], case["k"], case.get("rows", 1)
        passes = 2 if case.get("epi") == "resid" else 1
        return {"bytes": n * k * _BYTES[case["fmt"]] + 2.0 * rows * (k + passes * n), "flops": 2.0 * rows * n * k}
    if kind == "wkv":
        rows, H = case["B"] * case["T"], case["H"]
        return {"bytes": case["B"] * H * 2.0 * 16384 + 7.0 * 2 * rows * H * 64, "flops": 7.0 * rows * H * 4096}
    return {"bytes": 2.0 * case["B"] * case["V"] + 8.0 * case["B"], "flops": 0}


def tolerance(case):
    """About four times the distance to `exact` that a correct fp16 implementation shows over these ranges: one rounding per
    product (2e-4 .. 5e-4), 1e-3 .. 2e-3 behind a chain of blocks. Sampled ids are whole numbers from exact comparisons."""
    if case["kind"] == "sample":
        return "exact"
    return {"rel": 8e-3} if case["kind"] in ("decode", "step", "prefill") else {"rel": 1e-3} if case["kind"] == "wkv" else {"rel": 2e-3}


# ------------------------------------------------------------------------------------------------------------------
# the same in 64 bits
# ------------------------------------------------------------------------------------------------------------------
def _stored(w, fmt):
    """The values the weight format stores for w [n_out, k], in 64 bits."""
    if fmt == "none":
        return w.half().double()
    if fmt == "int8":
        amax = w.abs().amax(dim=1)
        s = amax / torch.full_like(amax, 127.0)
        return torch.round(w / s[:, None]).clamp(-127, 127).double() * s.double()[:, None]
    amax = w.abs().amax()
    t = amax / torch.full_like(amax, 448.0 * 6.0)
    blk = w.view(w.shape[0], -1, 16)
    sb = (blk.abs().amax(dim=2) / (torch.full_like(t, 6.0) * t)).clamp(max=448.0).to(torch.float8_e4m3fn).float()
    x = blk / (t * sb).clamp_min(1e-30)[:, :, None]
    mag, q = x.abs(), torch.zeros_like(x)
    # nearest of 0 .5 1 1.5 2 3 4 6, ties to the code with an even last bit
    for mid, step, up in ((0.25, 0.5, False), (0.75, 0.5, True), (1.25, 0.5, False), (1.75, 0.5, True), (2.5, 1.0, False),
                          (3.5, 1.0, True), (5.0, 2.0, False)):
        q += step * ((mag >= mid) if up else (mag > mid))
    return (torch.copysign(q, x).double() * sb.double()[:, :, None] * t.double()).view_as(w)


def _norm(x, w, b, eps):
    m = x.mean(-1, keepdim=True)
    return (x - m) / torch.sqrt(((x - m) ** 2).mean(-1, keepdim=True) + eps) * w + b


def _exact_model(case, seed):
    raw, state, ids, alone = _model_inputs(case, seed)
    L, D, B, T, fmt = case["L"], case["D"], case.get("B", 1), case.get("T", 1), case["fmt"]
    H, sg = D // 64, torch.sigmoid

    def big(name):
        return _stored(raw[name], fmt).t()

    def small(name):
        return raw[name].squeeze().half().double()

    state = [t.double().reshape((B,) + tuple(t.shape[0 if alone else 1:])) for t in state]
    tok = torch.tensor(ids, device="cuda").view(B, T)
    x = _norm(small("emb.weight")[tok], small("blocks.0.ln0.weight"), small("blocks.0.ln0.bias"), 1e-5)
    v_first, out = None, []
    for i in range(L):
        b = "blocks.%d." % i
        a, f = b + "att.", b + "ffn."
        prev, S, prev2 = state[3 * i:3 * i + 3]
        xn = _norm(x, small(b + "ln1.weight"), small(b + "ln1.bias"), 1e-5)
        dx = torch.cat([prev[:, None], xn[:, :-1]], 1) - xn
        xr, xw, xk, xv, xa, xg = (xn + dx * small(a + "x_" + c) for c in "rwkvag")
        r, k, v = xr @ big(a + "receptance.weight"), xk @ big(a + "key.weight"), xv @ big(a + "value.weight")
        wd = torch.exp(-0.606531 * sg(small(a + "w0") + torch.tanh(xw @ small(a + "w1")) @ small(a + "w2")))
        aa = sg(small(a + "a0") + (xa @ small(a + "a1")) @ small(a + "a2"))
        g = sg(xg @ small(a + "g1")) @ small(a + "g2")
        kk = torch.nn.functional.normalize((k * small(a + "k_k")).view(B, T, H, 64), dim=-1)
        k = k * (1 + (aa - 1) * small(a + "k_a"))
        if i == 0:
            v_first = v
        else:
            v = v + (v_first - v) * sg(small(a + "v0") + (xv @ small(a + "v1")) @ small(a + "v2"))
        hd = lambda t: t.reshape(B, T, H, 64)  # noqa: E731
        y, S = _wkv(S, hd(r), hd(wd), hd(k), hd(v), -kk, kk * hd(aa))
        y = _norm(y, small(a + "ln_x.weight").view(H, 64), small(a + "ln_x.bias").view(H, 64), 64e-5)
        y = y + (hd(r) * hd(k) * small(a + "r_k").view(H, 64)).sum(-1, keepdim=True) * hd(v)
        x = x + (y.reshape(B, T, D) * g) @ big(a + "output.weight")
        xn2 = _norm(x, small(b + "ln2.weight"), small(b + "ln2.bias"), 1e-5)
        kx = xn2 + (torch.cat([prev2[:, None], xn2[:, :-1]], 1) - xn2) * small(f + "x_k")
        x = x + torch.relu(kx @ big(f + "key.weight")) ** 2 @ big(f + "value.weight")
        out += [xn[:, -1], S, xn2[:, -1]]
    logits = _norm(x[:, -1], small("ln_out.weight"), small("ln_out.bias"), 1e-5) @ big("head.weight")
    out = [logits] + out
    return [t[0] for t in out] if alone else out


def _wkv(S, r, w, k, v, a, b):
    """S [B,H,64,64] and vectors [B,T,H,64] in 64 bits -> y, new S."""
    S, ys = S.clone(), []
    for t in range(r.shape[1]):
        sa = S @ a[:, t, :, :, None]
        S = S * w[:, t, :, None] + sa * b[:, t, :, None] + v[:, t, :, :, None] * k[:, t, :, None]
        ys.append((S @ r[:, t, :, :, None])[..., 0])
    return torch.stack(ys, 1), S


def exact(case, seed):
    kind = case["kind"]
    if kind in ("decode", "step", "prefill"):
        return _exact_model(case, seed)
    if kind in ("gemv", "gemm"):
        w, x, resid = _product_inputs(case, seed)
        y = x.double() @ _stored(w, case["fmt"]).t()
        fn = {"tanh": torch.tanh, "sigmoid": torch.sigmoid, "relu2": lambda t: torch.relu(t) ** 2, "resid": lambda t: t + resid.double()}
        return fn.get(case.get("epi"), lambda t: t)(y)
    if kind == "wkv":
        S, vec = _wkv_inputs(case, seed)
        r, w, k, v, a, b = (t.double().view(case["B"], case["T"], case["H"], 64) for t in vec)
        y, S = _wkv(S.double(), r, torch.exp(-torch.exp(w)), k, v, a, b)
        return y.view(case["B"], case["T"], -1), S
    return None
