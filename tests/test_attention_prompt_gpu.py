"""GPU parity of the many-query attention kernel (head dimension 128, enough row tiles to occupy the GPU) against the CPU oracle.

Tolerance: f32 throughout; sums of up to a few hundred rounded terms in chains of 32, so about 3e-7 relative: NMSE 1e-12 (ten times
that squared)."""
import ctypes as C

import numpy as np
import pytest

from oracle import sgref
from tests import util as U

pytestmark = pytest.mark.gpu
TOL = 1e-12
SCALE = float(1.0 / np.sqrt(128))


def _run(sm100, stream, q, k, v, causal, offset, mask=None, mask_heads=1, positions=None):
    hq, nq, d = q.shape
    hkv, nk, _ = k.shape
    qb, kb, vb = (U.to_device(sm100, stream, a) for a in (q, k, v))
    mb = U.to_device(sm100, stream, mask) if mask is not None else None
    pb = U.to_device(sm100, stream, np.array(positions, np.int32)) if positions is not None else None
    ob, optr = U.guarded_output(sm100, stream, hq * nq * d)
    before = sm100.lib().sm100_launch_count()
    sm100.check(sm100.lib().sm100_attention(stream.handle, qb.at(), kb.at(), vb.at(), mb.at() if mb else None, mask_heads, C.c_void_p(optr), d, d, nq, nk, hq, hkv,
                                            int(causal), offset, pb.at() if pb else None, SCALE), "attention")
    assert sm100.lib().sm100_launch_count() - before == 1
    stream.sync()
    return U.read_guarded(sm100, stream, ob, hq * nq * d).reshape(hq, nq, d).copy()


def _inputs(hq, hkv, nq, nk, seed=0):
    rng = np.random.default_rng(hq * 100 + nq + nk + seed)
    return tuple(rng.standard_normal(s).astype(np.float32) for s in ((hq, nq, 128), (hkv, nk, 128), (hkv, nk, 128)))


# whole and ragged row tiles, heads per group 1, 3, 4, 8; one key tile, a partial one, several; the first query sees one key or many
@pytest.mark.parametrize("hq,hkv,nq,nk", [(32, 8, 128, 128), (32, 8, 131, 200), (48, 16, 70, 97), (64, 64, 65, 65), (64, 8, 64, 33), (32, 8, 128, 31)], ids=lambda v: str(v))
def test_causal_full_and_masked(sm100, stream, hq, hkv, nq, nk):
    q, k, v = _inputs(hq, hkv, nq, nk)
    off = max(nk - nq, 0)
    want = sgref.attention(q, k, v, True, off, SCALE)
    assert sgref.nmse(_run(sm100, stream, q, k, v, True, off), want) <= TOL
    assert sgref.nmse(_run(sm100, stream, q, k, v, True, 0, positions=[off]), want) <= TOL
    assert sgref.nmse(_run(sm100, stream, q, k, v, False, 0), sgref.attention(q, k, v, False, 0, SCALE)) <= TOL
    for low in (-np.inf, np.finfo(np.float32).min):
        mask = np.zeros((1, nq, nk), np.float32)
        mask[0, :, nk // 3:] = low
        got = _run(sm100, stream, q, k, v, False, 0, mask=mask)
        assert sgref.nmse(got, sgref.attention(q, k[:, :nk // 3], v[:, :nk // 3], False, 0, SCALE)) <= TOL
    per_head = (0.5 * np.random.default_rng(3).standard_normal((hq, nq, nk))).astype(np.float32)
    got = _run(sm100, stream, q, k, v, True, off, mask=per_head, mask_heads=hq)
    g = hq // hkv
    s = np.einsum("hqd,hkd->hqk", q.astype(np.float64), np.repeat(k, g, 0).astype(np.float64)) * SCALE + per_head
    s[:, np.arange(nk)[None] > off + np.arange(nq)[:, None]] = -np.inf
    p = np.exp(s - s.max(-1, keepdims=True))
    want = np.einsum("hqk,hkd->hqd", p / p.sum(-1, keepdims=True), np.repeat(v, g, 0).astype(np.float64))
    assert sgref.nmse(got.astype(np.float64), want) <= TOL


def test_rows_without_keys_and_hidden_values(sm100, stream):
    """Queries before the first key give zeros; a value row holding NaN or infinity reaches the queries that see it and no other."""
    hq, hkv, nq, nk = 32, 8, 140, 120
    q, k, v = _inputs(hq, hkv, nq, nk)
    got = _run(sm100, stream, q, k, v, True, -20)
    want = sgref.attention(q[:, 20:], k, v, True, 0, SCALE)
    assert np.all(got[:, :20] == 0.0) and sgref.nmse(got[:, 20:], want) <= TOL
    bad = v.copy()
    bad[:, 100, 5] = np.nan
    bad[:, 110, 9] = np.inf
    got2 = _run(sm100, stream, q, k, bad, True, -20)
    assert np.array_equal(got2[:, :120], got[:, :120])
    assert np.isnan(got2[:, 120:, 5]).all() and not np.isfinite(got2[:, 130:, 9]).any()


# many-query kernel, decode kernel with the splits merged in the launch and by a second one (more than 128 splits), generic kernel
@pytest.mark.parametrize("hq,hkv,nq,nk,d", [(32, 8, 128, 200, 128), (32, 8, 128, 600, 128), (32, 8, 2, 600, 128), (8, 8, 3, 300, 256), (4, 4, 1, 5000, 128), (6, 2, 3, 200, 64)], ids=lambda v: str(v))
def test_nan_scores_stay_visible(sm100, stream, hq, hkv, nq, nk, d):
    """A NaN in a query or in any key that it sees makes the whole row NaN, wherever it stands: a row (or the part of one that a
    warp, a tile or a split sees) that holds nothing but NaN must not pass for one without a visible key."""
    rng = np.random.default_rng(hq + nq + nk)
    q, k, v = (rng.standard_normal(s).astype(np.float32) for s in ((hq, nq, d), (hkv, nk, d), (hkv, nk, d)))
    off, g = nk - nq, hq // hkv

    def run(q, k):
        qb, kb, vb = (U.to_device(sm100, stream, a) for a in (q, k, v))
        ob, optr = U.guarded_output(sm100, stream, hq * nq * d)
        sm100.check(sm100.lib().sm100_attention(stream.handle, qb.at(), kb.at(), vb.at(), None, 1, C.c_void_p(optr), d, d, nq, nk, hq, hkv, 1, off, None, SCALE), "attention")
        stream.sync()
        return U.read_guarded(sm100, stream, ob, hq * nq * d).reshape(hq, nq, d).copy()

    clean = run(q, k)
    bad = q.copy()
    bad[1, nq - 1, 3] = np.nan
    got = run(bad, k)
    assert np.isnan(got[1, nq - 1]).all()
    rest = np.ones((hq, nq), bool)
    rest[1, nq - 1] = False
    assert np.array_equal(got[rest], clean[rest])
    for first, last in ((0, 40), (off, off + 1), (0, off + 1)):   # every query sees them
        bad = k.copy()
        bad[hkv - 1, first:last, 7] = np.nan
        got = run(q, bad)
        assert np.isnan(got[(hkv - 1) * g:]).all(), (first, last)
        assert np.array_equal(got[:(hkv - 1) * g], clean[:(hkv - 1) * g])


def test_keys_hidden_beyond_the_first_span_of_tiles(sm100, stream):
    """The first 18 of 20 key tiles are masked: the sums set aside after eight of them belong to no visible key yet."""
    q, k, v = _inputs(32, 8, 128, 640)
    mask = np.zeros((1, 128, 640), np.float32)
    mask[0, :, :576] = -np.inf
    mask[0, 5] = -np.inf
    mask[0, 7, :] = 0
    got = _run(sm100, stream, q, k, v, False, 0, mask=mask)
    rows = [i for i in range(128) if i not in (5, 7)]
    assert sgref.nmse(got[:, rows], sgref.attention(np.ascontiguousarray(q[:, rows]), k[:, 576:], v[:, 576:], False, 0, SCALE)) <= TOL
    assert np.all(got[:, 5] == 0.0)
    assert sgref.nmse(got[:, 7:8], sgref.attention(np.ascontiguousarray(q[:, 7:8]), k, v, False, 0, SCALE)) <= TOL


@pytest.mark.parametrize("nk,bound", [(576, 2.0e-7), (8192, 2.4e-7)], ids=["576", "8192"])
def test_rounding_does_not_grow_with_the_context(sm100, stream, nk, bound):
    """Against float64.  The bounds are what the decode kernel leaves on these calls (1.9e-7 to 2.0e-7, 2.3e-7); one chain of additions
    over all key tiles left 2.3e-7 and 3.7e-7."""
    hq, hkv, nq = 64, 8, 64
    q, k, v = _inputs(hq, hkv, nq, nk)
    off, g = nk - nq, hq // hkv
    s = q[:g].astype(np.float64) @ k[0].astype(np.float64).T * SCALE
    s[:, np.arange(nk)[None] > off + np.arange(nq)[:, None]] = -np.inf
    p = np.exp(s - s.max(-1, keepdims=True))
    want = (p / p.sum(-1, keepdims=True)) @ v[0].astype(np.float64)
    err = np.linalg.norm(_run(sm100, stream, q, k, v, True, off)[:g] - want) / np.linalg.norm(want)
    assert err <= bound, err


# few tiles whose rows see very different numbers of keys; short rows, more tiles, a long prefix, heads in groups of 2, 8 and 1, no causal mask
@pytest.mark.parametrize("hq,hkv,nq,nk,causal,name", [(8, 2, 512, 512, True, "attn_splits"), (4, 1, 1024, 1300, True, "attn_splits"), (8, 2, 520, 560, True, "attn_splits"),
                                                      (12, 3, 345, 400, True, "attn_prompt"), (4, 2, 1024, 1024, True, "attn_prompt"), (8, 2, 768, 768, True, "attn_prompt"), (8, 2, 512, 1536, True, "attn_prompt"),
                                                      (8, 1, 512, 512, True, "attn_prompt"), (8, 8, 512, 512, True, "attn_prompt"), (8, 2, 512, 512, False, "attn_prompt"),
                                                      (32, 8, 128, 128, True, "attn_prompt")], ids=lambda v: str(v))
def test_uneven_prompts_take_the_faster_kernel(sm100, stream, hq, hkv, nq, nk, causal, name):
    """Same values whichever kernel serves a call; a captured one always has the kernel that needs no memory.  Calls on two streams
    share nothing."""
    q, k, v = _inputs(hq, hkv, nq, nk)
    off = nk - nq if causal else 0
    want = sgref.attention(q, k, v, causal, off, SCALE)
    assert sgref.nmse(_run(sm100, stream, q, k, v, causal, off), want) <= TOL
    assert (sm100.lib().sm100_matvec_last_kernel() or b"").decode() == name
    qb, kb, vb = (U.to_device(sm100, stream, a) for a in (q, k, v))
    ob, optr = U.guarded_output(sm100, stream, hq * nq * 128)
    stream.sync()
    graph = sm100.Graph(stream)
    with graph:
        sm100.check(sm100.lib().sm100_attention(stream.handle, qb.at(), kb.at(), vb.at(), None, 1, C.c_void_p(optr), 128, 128, nq, nk, hq, hkv, int(causal), off, None, SCALE), "attention")
    assert (sm100.lib().sm100_matvec_last_kernel() or b"").decode() == "attn_prompt"
    graph.launch()
    stream.sync()
    assert sgref.nmse(U.read_guarded(sm100, stream, ob, hq * nq * 128).reshape(hq, nq, 128), want) <= TOL
    graph.destroy()
    streams, outs = [stream, sm100.Stream(0)], [U.guarded_output(sm100, stream, hq * nq * 128) for _ in range(2)]
    stream.sync()
    for _ in range(3):
        for s, (_, p) in zip(streams, outs):
            sm100.check(sm100.lib().sm100_attention(s.handle, qb.at(), kb.at(), vb.at(), None, 1, C.c_void_p(p), 128, 128, nq, nk, hq, hkv, int(causal), off, None, SCALE), "attention")
    for s, (b, _) in zip(streams, outs):
        s.sync()
        assert sgref.nmse(U.read_guarded(sm100, s, b, hq * nq * 128).reshape(hq, nq, 128), want) <= TOL
    streams[1].close()
