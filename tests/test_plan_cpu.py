"""CPU: the block partition of the matrix-vector kernels (host-side planner of the library, no GPU needed)."""
import ctypes as C

import numpy as np
import pytest
from hypothesis import given, settings, strategies as st

from albatross_b200 import _lib, synth

F16, I8, FP4 = 0, 1, 2


def _check(fmt, rows, k, n_blocks):
    n = len(fmt)
    arr = lambda v: (C.c_int32 * n)(*v)
    items, spread = C.c_int32(0), C.c_int32(0)
    rc = _lib.lib.ab_gemv_plan_selftest(arr(fmt), arr(rows), arr(k), n, n_blocks, C.byref(items), C.byref(spread))
    assert rc == 0, _lib.lib.ab_last_error().decode()
    return items.value, spread.value


@pytest.mark.parametrize("D", [64, 128, 256, 768, 1024, 2048, 2560, 4096])
@pytest.mark.parametrize("big", [F16, I8, FP4])
@pytest.mark.parametrize("n_blocks", [148, 132, 80])
def test_head_aligned_plan_covers_every_row_once(D, big, n_blocks):
    """r, k, v and the adapters over two or more blocks per head: the library's self-check goes over that plan as well when a
    launch has this form and the blocks suffice (with the fewest, the default and the most row groups on a head's first block)."""
    for ranks in ((64, 64, 32, 128), (4, 4, 4), (128, 128, 96, 480)):
        _check([big] * 3 + [F16] * len(ranks), [D] * 3 + list(ranks), [D] * (3 + len(ranks)), n_blocks)


@pytest.mark.parametrize("cfg", ["tiny", "0.1b", "7.2b"])
@pytest.mark.parametrize("big", [I8, FP4])
def test_every_phase_of_the_decode_program_is_covered(cfg, big):
    L, D, V, (rw, ra, rv, rg) = synth.CONFIGS[cfg]
    phases = {
        "rkv+downs": ([big] * 3 + [F16] * 4, [D] * 3 + [rw, ra, rv, rg], [D] * 7),
        "ups": ([F16] * 4, [D] * 4, [rw, ra, rv, rg]),
        "output": ([big], [D], [D]),
        "ffn key": ([big], [4 * D], [D]),
        "ffn value": ([big], [D], [4 * D]),
        "head": ([big], [V], [D]),
    }
    for name, (fmt, rows, k) in phases.items():
        items, spread = _check(fmt, rows, k, 148)
        assert items >= 1, name
        if cfg == "7.2b":
            assert spread <= 12, (name, spread)      # the most loaded block is at most 12 % above the mean cost


@settings(max_examples=60, deadline=None)
@given(st.lists(st.tuples(st.sampled_from([F16, I8, FP4]), st.integers(1, 3000), st.integers(1, 64)), min_size=1, max_size=7),
       st.integers(1, 200))
def test_random_segment_lists_are_covered_exactly_once(segs, n_blocks):
    fmt = [s[0] for s in segs]
    rows = [s[1] for s in segs]
    k = [s[2] * 32 for s in segs]          # NVFP4 rows need k % 32 == 0
    _check(fmt, rows, k, n_blocks)


def _al(v):
    return (v + 255) & ~255


def _model(D, V, fmt, head=True, L=2):
    """A model handle on made-up (never followed) addresses: sizes only."""
    layers = (_lib.Layer * L)()
    ptr = 1 << 20
    mat = lambda f, n, k: _lib.Mat(f, n, k, 0, ptr, None if f == F16 else ptr, None, 1.0, 0.0)
    for ly in layers:
        for name in _lib._LAYER_PTRS + _lib._LAYER_UPS:
            setattr(ly, name, ptr)
        for name in ("receptance", "key", "value", "output"):
            setattr(ly, name, mat(fmt, D, D))
        ly.ffn_key, ly.ffn_value = mat(fmt, 4 * D, D), mat(fmt, D, 4 * D)
        for n in "wavg":
            setattr(ly, n + "1t", mat(F16, 64, D))
            setattr(ly, n + "2t", mat(F16, D, 64))
    d = _lib.ModelDesc()
    d.n_layer, d.n_embd, d.vocab, d.emb, d.layers = L, D, V, ptr, C.cast(layers, C.POINTER(_lib.Layer))
    if head:
        d.lnout_w = d.lnout_b = ptr
        d.head = mat(fmt, V, D)
    h = C.c_void_p()
    _lib.check(_lib.lib.ab_model_create(C.byref(d), C.byref(h)))
    return h, d.head


@pytest.mark.parametrize("fmt", [I8, FP4, F16])
@pytest.mark.parametrize("D,V", [(1024, 1024), (2048, 1024), (2560, 2048), (4096, 512), (4096, 4096), (4096, 65536)])
def test_workspace_holds_the_partial_sums_of_a_prompts_last_product(fmt, D, V):
    """After a prompt of T tokens the vocabulary head sees only the B last rows, and few rows are split along K where B * T
    rows were not: the scratch part of the workspace has to hold either. What the head adds to a workspace is compared with
    the one of the same blocks without a head, whose scratch part is at least the arrival counters' 16 KB + 256."""
    h, head = _model(D, V, fmt)
    bare, _ = _model(D, V, fmt, head=False)
    ws = _lib.lib.ab_workspace_bytes
    counters = 4096 * 4 + 256
    for B in (1, 2, 3, 5, 8, 40):
        for T in (2, 7, 37, 128, 513, 700, 1025, 2305, 3000):
            need = _lib.lib.ab_gemm_scratch_bytes(C.byref(head), B)
            rest = ws(bare, B, T) - _al(counters)       # everything else, if the blocks' own products are not split
            if B * T >= 2305:                           # ... which holds for so many rows of these widths
                assert ws(h, B, T) >= rest + need, (B, T)
            assert ws(h, B, T) >= need and ws(h, B, T) >= ws(bare, B, T), (B, T)
    # one sequence of 513 tokens, 4096 wide: no product of 513 rows is split, the head's single row is, eight ways
    if (D, V, fmt) == (4096, 4096, I8):
        assert ws(h, 1, 513) - ws(bare, 1, 513) >= _lib.lib.ab_gemm_scratch_bytes(C.byref(head), 1) - counters - 256 > 1 << 19
    for x in (h, bare):
        _lib.lib.ab_model_destroy(x)


def _gemm_plan(ops, rows, n_sm=148):
    n = len(ops)
    arr = lambda v: (C.c_int32 * n)(*v)
    tile, blocks, ks = C.c_int32(0), C.c_int32(0), (C.c_int32 * n)()
    rc = _lib.lib.ab_gemm_plan_selftest(arr([o[0] for o in ops]), arr([o[1] for o in ops]), arr([o[2] for o in ops]), n, rows, n_sm,
                                        C.byref(tile), C.byref(blocks), ks)
    assert rc == 0, _lib.lib.ab_last_error().decode()
    return tile.value, blocks.value, list(ks)


@pytest.mark.parametrize("fmt", [I8, FP4, F16])
@pytest.mark.parametrize("n_out,k,rows,blocks,ksteps", [
    (2560, 10240, 400, 100, 54), (2560, 10240, 512, 100, 54), (4096, 16384, 400, 100, 128), (2048, 8192, 640, 100, 43),   # long K: split
    (2560, 2560, 400, 80, 40), (768, 768, 768, 36, 12),                                                                    # short: low tiles
    (16384, 4096, 400, 256, 64), (4096, 4096, 768, 128, 64)])
def test_tile_height_weighs_the_split_along_k(fmt, n_out, k, rows, blocks, ksteps):
    """The k-steps a block is left with and the SMs at work, for products on both sides of the choice between low tiles and
    tall ones that are split (bounds: the fastest of the seven heights, timed)."""
    _, b, (ks,) = _gemm_plan([(fmt, n_out, k)], rows)
    assert b >= blocks and -(-(k // 64) // ks) <= ksteps, (b, ks)


@settings(max_examples=200, deadline=None)
@given(st.lists(st.tuples(st.sampled_from([F16, I8, FP4]), st.integers(1, 20000), st.integers(1, 300)), min_size=1, max_size=7),
       st.integers(1, 4000), st.sampled_from([148, 132, 1]))
def test_every_plan_of_products_fits_its_scratch_and_the_gpu(segs, rows, n_sm):
    """Checked inside: partial sums within the scratch area, a split grid resident at once, tiles of whole chunks."""
    tile, _, _ = _gemm_plan([(f, n, 64 * k) for f, n, k in segs], rows, n_sm)
    assert 16 <= tile <= 320


def test_state_list_forgets_its_checks_when_changed():
    """The list forward() hands back carries the model's validation and program key; any in-place change of the list
    drops them, so a changed list is checked from scratch (it is still a plain list to its user)."""
    from albatross_b200.rwkv7 import _State
    owner = object()
    mark = (owner, None, (1, 2, 3))
    for change in (lambda s: s.__setitem__(0, "x"), lambda s: s.append("x"), lambda s: s.pop(), lambda s: s.extend(["y"]),
                   lambda s: s.insert(0, "z"), lambda s: s.clear(), lambda s: s.reverse(), lambda s: s.__delitem__(0),
                   lambda s: s.__iadd__(["w"])):
        st = _State(["a", "b", "c"], mark)
        assert st._ab is mark and isinstance(st, list) and list(st) == ["a", "b", "c"]
        change(st)
        assert st._ab is None
    st = _State(["a", "b"], mark)
    assert st[1] == "b" and len(st) == 2 and st._ab is mark          # reading keeps them
    assert not hasattr(list(st), "_ab") and _State(st)._ab is None   # a copy starts unchecked


def _program_check(D, L, ranks, fmt, n_blocks, options=()):
    """ab_decode_plan_selftest of a model whose pointers are stand-ins (the library only looks at shapes)."""
    p = 1 << 20
    mat = lambda n, k, f=F16: _lib.Mat(fmt=f, n_out=n, k=k, w=p, scale=p if f != F16 else None, tscale=1.0)
    rw, ra, rv, rg = ranks
    layers = (_lib.Layer * L)()
    for i, l in enumerate(layers):
        for name, _ in _lib.Layer._fields_[:19]: setattr(l, name, p)
        for name in ("receptance", "key", "value", "output"): setattr(l, name, mat(D, D, fmt))
        l.ffn_key, l.ffn_value = mat(4 * D, D, fmt), mat(D, 4 * D, fmt)
        l.w1t, l.a1t, l.g1t = mat(rw, D), mat(ra, D), mat(rg, D)
        l.w2t, l.a2t, l.g2t = mat(D, rw), mat(D, ra), mat(D, rg)
        l.w2 = l.a2 = l.g2 = p
        if i > 0: l.v1t, l.v2t, l.v2 = mat(rv, D), mat(D, rv), p
    desc = _lib.ModelDesc(n_layer=L, n_embd=D, vocab=512, emb=p, lnout_w=p, lnout_b=p, head=mat(512, D, fmt), layers=layers)
    model = C.c_void_p()
    assert _lib.lib.ab_model_create(C.byref(desc), C.byref(model)) == 0, _lib.lib.ab_last_error().decode()
    try:
        for name, value in options: assert _lib.lib.ab_model_set_option(model, name, value) == 0
        rc = _lib.lib.ab_decode_plan_selftest(model, n_blocks)
        assert rc == 0, _lib.lib.ab_last_error().decode()
    finally:
        _lib.lib.ab_model_destroy(model)


@pytest.mark.parametrize("D,ranks", [(64, (16, 16, 16, 16)), (256, (32, 32, 16, 48)), (768, (64, 64, 32, 128)), (2048, (96, 96, 64, 256)),
                                     (4096, (128, 128, 96, 480))])
@pytest.mark.parametrize("fmt", [F16, I8, FP4])
@pytest.mark.parametrize("options", [(), ((b"fuse_heads", 0),), ((b"merge_ups", 1),)])
def test_decode_program_orders_the_token_shift_states(D, ranks, fmt, options):
    """Without a barrier among all blocks a token-shift state may be overwritten only behind inputs that depend on every block that
    read the old one: not by a head's own phase (its inputs come from a few blocks), and not ahead of the wait for the inputs."""
    for n_blocks in (148, 132): _program_check(D, 3, ranks, fmt, n_blocks, options)


@pytest.mark.parametrize("D,ranks", [(256, (32, 32, 16, 48)), (768, (64, 64, 32, 128)), (768, (128, 64, 256, 128)), (2048, (96, 96, 64, 256)),
                                     (2560, (96, 96, 64, 320))])
@pytest.mark.parametrize("fmt", [F16, I8, FP4])
def test_decode_program_keeps_a_head_on_its_block(D, ranks, fmt):
    """The first layer has fewer adapter rows than the others, which would leave more blocks to its heads; but a head's part of
    that layer's value vector is read in all the others, without a tag: the same block has to run the head in every layer."""
    for n_blocks in (148, 144, 132): _program_check(D, 3, ranks, fmt, n_blocks)


@pytest.mark.parametrize("rows", [2, 8, 24, 100])
@pytest.mark.parametrize("scratch", [None, (1 << 20) + 8])
def test_products_that_split_k_are_refused_without_a_scratch_area(rows, scratch):
    """... whichever kernel would run them: the ones of few rows need no scratch, but what a caller may pass does not depend on that."""
    p = 1 << 20
    m = _lib.Mat(fmt=I8, n_out=1024, k=16384, w=p, scale=p, tscale=1.0)
    assert _lib.lib.ab_gemm(C.byref(m), rows, p, p, 0, None, scratch, None) == -1
    assert b"scratch" in _lib.lib.ab_last_error()
