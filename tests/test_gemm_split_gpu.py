"""GPU parity of the split-operand tensor-core MUL_MAT (batches of packed weights, Q6_K at any width) against the CPU oracle.

Tolerance: both operands are two bf16 numbers (16 bits: relative rounding at most 2^-17, about 2^-18.5 rms) and with more than 64 columns
the product of the two small parts is dropped (below 2^-17), so a product is off by 1e-5; the f32
accumulation in the tensor core truncates (up to 2e-5 over 768 steps, K = 12288).  NMSE bound: (3e-5)^2.
"""
import ctypes as C

import numpy as np
import pytest

from oracle import sgref
from tests import util as U

pytestmark = pytest.mark.gpu
TOL = 1e-9
COLUMNS_TOL = 2e-8   # the integer column kernels: 16-bit activations per 64 weights, their bound in test_matvec_gpu.py is 1e-6
# shapes of the lists below that the column kernel (test_quant_cols_gpu.py) serves instead
COLUMN_KERNEL = {(U.Q4_0, 1024, 1030, 4), (U.Q8_0, 512, 128 * 297, 5), (U.Q6_K, 5120, 13824, 8)}


def _name(dtype, k, n, m):
    return ("quant_cols" if (dtype, k, n, m) in COLUMN_KERNEL else "gemm_split") + ("" if n % 16 == 0 else "+rows")


def _check(sm100, stream, dtype, k, n, m):
    wq = U.quantize(dtype, U.seeded_weights(7000 + dtype + k, n, k))
    x = U.seeded_acts(3 * m + k, m, k)
    want = sgref.mul_mat(dtype, wq, k, x)
    got = U.device_mul_mat(sm100, stream, dtype, U.PACKED, wq, k, x)
    assert (sm100.lib().sm100_matvec_last_kernel() or b"").decode() == _name(dtype, k, n, m)
    assert np.isfinite(got).all()
    for t in range(m):   # per token, so that one wrong column cannot hide in the average
        assert sgref.nmse(got[t], want[t]) <= TOL, (t, sgref.nmse(got[t], want[t]))
    for r in {0, n // 2, n - 1}:
        assert sgref.nmse(got[:, r], want[:, r]) <= 4 * TOL, r


# rows below, at and past a tile; one block of K, a K range of one stage per CTA, long K; edges of the 16 / 32 column tiles
@pytest.mark.parametrize("dtype", U.QUANT, ids=lambda d: U.NAMES[d])
@pytest.mark.parametrize("shape", [(256, 24, 9), (512, 128, 16), (512, 257, 17), (4096, 130, 32), (12288, 48, 24)], ids=lambda s: f"k{s[0]}n{s[1]}m{s[2]}")
def test_batches(sm100, stream, dtype, shape):
    _check(sm100, stream, dtype, *shape)


# three to eight columns, from 1024 rows on: the matvec's own way here; rows at and past a tile of 128, a tail, K of one stage and more
@pytest.mark.parametrize("dtype,k,n,m", [(U.Q4_0, 1024, 1030, 4), (U.Q4_0, 128, 1024, 7), (U.Q8_0, 1024, 1030, 7), (U.Q8_0, 2176, 1152, 4),
                                         (U.Q6_K, 1024, 1030, 3), (U.Q6_K, 256, 1040, 5), (U.Q6_K, 4096, 1030, 8),
                                         (U.Q4_0, 1152, 1030, 4)], ids=lambda v: str(v))
def test_few_columns(sm100, stream, dtype, k, n, m):
    _check(sm100, stream, dtype, k, n, m)


# more tiles than SMs: whole waves of one CTA per tile, and the rest with K cut; row and token tiles ragged
@pytest.mark.parametrize("dtype,k,n,m", [(U.Q4_0, 512, 128 * 160 + 16, 24), (U.Q4_K, 1024, 128 * 150 + 5, 32), (U.Q8_0, 512, 128 * 297, 5), (U.Q6_K, 512, 4100, 700), (U.Q6_K, 1024, 6400, 200),
                                         (U.Q8_0, 640, 128 * 297, 5)],
                         ids=lambda v: str(v))
def test_whole_waves_and_cut_tiles(sm100, stream, dtype, k, n, m):
    """Rows repeat every 360 (no multiple of a tile), so that the oracle has few to multiply while every tile differs from its neighbours."""
    few = 360
    wq = U.quantize(dtype, U.seeded_weights(dtype + k, few, k))
    x = U.seeded_acts(k + m, m, k)
    want = sgref.mul_mat(dtype, wq, k, x)[:, np.arange(n) % few]
    got = U.device_mul_mat(sm100, stream, dtype, U.PACKED, np.ascontiguousarray(np.resize(wq, (n, wq.shape[1]))), k, x)
    assert (sm100.lib().sm100_matvec_last_kernel() or b"").decode() == _name(dtype, k, n, m)
    for r0 in range(0, n, 128):
        for t0 in range(0, m, 64):
            part = np.s_[t0:t0 + 64, r0:r0 + 128]
            assert sgref.nmse(got[part], want[part]) <= TOL, (r0, t0)


@pytest.mark.parametrize("dtype", [U.Q4_0, U.Q8_0], ids=lambda d: U.NAMES[d])
@pytest.mark.parametrize("shape", [(128, 16, 9), (384, 144, 31)], ids=lambda s: f"k{s[0]}n{s[1]}m{s[2]}")
def test_an_odd_number_of_chunk_pairs(sm100, stream, dtype, shape):
    """One stage of two chunks, and three."""
    _check(sm100, stream, dtype, *shape)


# rows that are not whole stages stay with the other kernels
@pytest.mark.parametrize("dtype", [U.Q4_0, U.Q8_0], ids=lambda d: U.NAMES[d])
@pytest.mark.parametrize("shape", [(32, 16, 9), (96, 130, 31)], ids=lambda s: f"k{s[0]}n{s[1]}m{s[2]}")
def test_short_rows(sm100, stream, dtype, shape):
    k, n, m = shape
    wq = U.quantize(dtype, U.seeded_weights(7000 + dtype + k, n, k))
    x = U.seeded_acts(3 * m + k, m, k)
    assert sgref.nmse(U.device_mul_mat(sm100, stream, dtype, U.PACKED, wq, k, x), sgref.mul_mat(dtype, wq, k, x)) <= TOL
    assert "gemm_split" not in (sm100.lib().sm100_matvec_last_kernel() or b"").decode()


@pytest.mark.parametrize("shape", [(256, 24, 33), (512, 130, 64), (512, 257, 65), (4096, 128, 129), (12288, 40, 48)], ids=lambda s: f"k{s[0]}n{s[1]}m{s[2]}")
def test_q6_k_prompts(sm100, stream, shape):
    _check(sm100, stream, U.Q6_K, *shape)


def test_q6_k_prompt_in_passes(sm100, stream):
    """More tokens than one pass of prepared activations holds (64 MiB: 1365 tokens at K = 12288)."""
    _check(sm100, stream, U.Q6_K, 12288, 16, 1400)


@pytest.mark.parametrize("dtype,m", [(U.Q4_0, 12), (U.Q8_0, 32), (U.Q4_K, 12), (U.Q6_K, 20), (U.Q6_K, 40)], ids=lambda v: str(v))
def test_token_magnitudes_and_poison(sm100, stream, dtype, m):
    """A column keeps its precision whatever its magnitude, and a NaN or an infinity poisons its own column only."""
    k, n = 1024, 144
    wq = U.quantize(dtype, U.seeded_weights(5, n, k))
    x = U.seeded_acts(6, m, k)
    x[0] *= 1e30
    x[1] *= 1e-25
    x[2] = 0.0
    x[3, 5] = 3e6
    x[4, 7] = np.nan
    x[5, 9] = np.inf
    want = sgref.mul_mat(dtype, wq, k, x)
    got = U.device_mul_mat(sm100, stream, dtype, U.PACKED, wq, k, x)
    assert np.all(got[2] == 0.0)
    assert not np.isfinite(got[4]).any() and not np.isfinite(got[5]).any()
    for t in [0, 1, 3] + list(range(6, m)):
        assert sgref.nmse(got[t].astype(np.float64), want[t].astype(np.float64)) <= TOL, t


def test_large_scales_stay_finite(sm100, stream):
    """Block scales near the top of f16: an f16 operand would overflow."""
    k, n, m = 512, 32, 10
    wq = U.quantize(U.Q8_0, U.seeded_weights(8, n, k) * np.float32(3e5))
    x = U.seeded_acts(9, m, k)
    got = U.device_mul_mat(sm100, stream, U.Q8_0, U.PACKED, wq, k, x)
    assert np.isfinite(got).all() and sgref.nmse(got, sgref.mul_mat(U.Q8_0, wq, k, x)) <= TOL


def test_captures_on_two_streams(sm100):
    """A Q6_K prompt needs memory for its prepared activations: each replay works on the inputs of the moment, and calls on two
    streams at a time do not share memory."""
    k, n, m = 768, 200, 200
    wq = U.quantize(U.Q6_K, U.seeded_weights(11, n, k))
    streams = [sm100.Stream(0) for _ in range(2)]
    img = sm100.pack(U.Q6_K, k, wq)
    wb = U.to_device(sm100, streams[0], img)
    xs = [U.seeded_acts(20 + i, m, k) for i in range(4)]
    want = [sgref.mul_mat(U.Q6_K, wq, k, x) for x in xs]
    xb = [U.to_device(sm100, streams[0], xs[i]) for i in range(2)]
    yb = [sm100.Buffer(4 * n * m) for _ in range(2)]
    streams[0].sync()
    graphs = []
    for s, x, y in zip(streams, xb, yb):
        g = sm100.Graph(s)
        with g:
            sm100.mul_mat(s, U.Q6_K, U.PACKED, wb, k, n, x, m, y)
        graphs.append(g)
    for turn in range(2):
        for i in range(2):
            xb[i].upload(streams[i], xs[2 * turn + i])
        for _ in range(3):
            for g in graphs:
                g.launch()
        for i, s in enumerate(streams):
            s.sync()
            got = yb[i].download(s, np.float32, n * m).reshape(m, n)
            assert sgref.nmse(got, want[2 * turn + i]) <= TOL, (turn, i)
    for _ in range(4):   # eager, both streams in flight
        for i, s in enumerate(streams):
            sm100.mul_mat(s, U.Q6_K, U.PACKED, wb, k, n, xb[i], m, yb[i])
    for i, s in enumerate(streams):
        s.sync()
        assert sgref.nmse(yb[i].download(s, np.float32, n * m).reshape(m, n), want[2 + i]) <= TOL
    for g in graphs:
        g.destroy()
    for s in streams:
        s.close()


# whole tiles only where nothing needs cutting, tiles of a prompt; and one shape below the limit
@pytest.mark.parametrize("dtype,k,n,m", [(U.Q4_0, 28672, 148 * 128, 4), (U.Q6_K, 28672, 1024, 130), (U.Q6_K, 14336, 512, 300), (U.Q6_K, 12288, 512, 300)], ids=lambda v: str(v))
def test_error_does_not_grow_with_k(sm100, stream, dtype, k, n, m):
    """The tensor core truncates when it adds: K is cut so that no chain is longer than 13312 weights, and the error against float64 stays
    below that of the integer column kernels (1.8e-5 to 2.1e-5 at any K; 3.1e-5 and more were seen at 28672 in one chain)."""
    wq = U.quantize(dtype, U.seeded_weights(7000 + dtype + k, min(n, 640), k))
    wq = np.ascontiguousarray(np.resize(wq, (n, wq.shape[1])))
    x = U.seeded_acts(3 * m + k, m, k)
    rows = np.r_[0:256, n - 256:n]
    want = x.astype(np.float64) @ sgref.dequantize(dtype, np.ascontiguousarray(wq[rows]), k).astype(np.float64).T
    got = U.device_mul_mat(sm100, stream, dtype, U.PACKED, wq, k, x)[:, rows]
    err = np.linalg.norm(got - want) / np.linalg.norm(want)
    assert err <= 1.8e-5, err


@pytest.mark.parametrize("dtype,k,n", [(U.Q4_0, 4096, 1040), (U.Q8_0, 2048, 3000), (U.Q4_K, 4096, 300), (U.Q6_K, 6144, 2064)], ids=lambda v: str(v))
def test_columns_do_not_depend_on_their_batch(sm100, stream, dtype, k, n):
    """Bit for bit, over the 16 and 32 column tiles (Q4_K: from 17 columns on, fewer belong to the column kernel)."""
    wq = U.quantize(dtype, U.seeded_weights(dtype + k, n, k))
    x = U.seeded_acts(k, 32, k)
    all_ = U.device_mul_mat(sm100, stream, dtype, U.PACKED, wq, k, x)
    for m in [24, 17] + ([] if dtype == U.Q4_K else [16, 9]) + ([7] if n >= 1024 and dtype != U.Q4_K else []):
        assert np.array_equal(U.device_mul_mat(sm100, stream, dtype, U.PACKED, wq, k, x[:m]), all_[:m]), m


# few rows, a filled wave of the split GEMM, a long row; many rows and up to 16 columns in two launches; rows that fit four at a
# time; a tail; more columns, and Q6_K, stay with the more accurate kernel
@pytest.mark.parametrize("dtype,k,n,m,name", [(U.Q4_K, 4096, 1024, 16, "gemm_split"), (U.Q4_K, 2048, 8192, 24, "gemm_split"), (U.Q4_K, 12288, 2048, 9, "gemm_split"),
                                              (U.Q4_K, 1024, 8192, 9, "matvec_q4k_imma_cols"), (U.Q4_K, 4096, 4096, 16, "matvec_q4k_imma_cols"),
                                              (U.Q4_K, 1024, 65536, 12, "matvec_q4k_imma_cols"), (U.Q4_K, 5120, 13824, 17, "gemm_split"),
                                              (U.Q4_K, 8192, 28672, 11, "matvec_q4k_imma_cols"), (U.Q4_K, 1024, 8203, 10, "matvec_q4k_imma_cols+rows"),
                                              (U.Q6_K, 5120, 13824, 8, "quant_cols"), (U.Q6_K, 5120, 13824, 9, "gemm_split")], ids=lambda v: str(v))
def test_batches_take_the_faster_kernel(sm100, stream, dtype, k, n, m, name):
    """Batches that the integer column kernels serve faster than one pass of the split GEMM stay with them.  Rows repeat every 480 (not a
    multiple of any tile), so that the oracle has few to multiply."""
    few = min(n, 480)
    wq = U.quantize(dtype, U.seeded_weights(dtype + k, few, k))
    x = U.seeded_acts(k + m, m, k)
    want = sgref.mul_mat(dtype, wq, k, x)
    got = U.device_mul_mat(sm100, stream, dtype, U.PACKED, np.ascontiguousarray(np.resize(wq, (n, wq.shape[1]))), k, x)
    assert (sm100.lib().sm100_matvec_last_kernel() or b"").decode() == name
    want = want[:, np.arange(n) % few]
    for t in range(m):
        assert sgref.nmse(got[t], want[t]) <= (COLUMNS_TOL if "imma_cols" in name else TOL), t
    for r0 in range(0, n, 1024):
        part = slice(r0, min(n, r0 + 1024))
        assert sgref.nmse(got[:, part], want[:, part]) <= 4 * (COLUMNS_TOL if "imma_cols" in name else TOL), r0


# the last N mod 16 rows behind whole tiles (one row, 15 rows; one panel of 8 columns, a ragged one, many), fewer rows than a tile, rows
# that are not whole units of the integer kernels, rows too long for them
@pytest.mark.parametrize("dtype,k,n,m,tail", [(U.Q4_0, 1024, 1025, 5, 1), (U.Q8_0, 4096, 47, 17, 15), (U.Q4_K, 512, 140, 9, 12), (U.Q4_K, 12288, 24, 32, 8),
                                              (U.Q6_K, 768, 1031, 3, 7), (U.Q6_K, 4096, 29, 12, 13), (U.Q6_K, 4096, 520, 300, 8), (U.Q6_K, 12288, 31, 40, 15),
                                              (U.Q4_K, 1024, 8, 9, 8), (U.Q6_K, 4096, 15, 64, 15), (U.Q4_0, 160, 48, 31, 48), (U.Q8_0, 4064, 64, 12, 64),
                                              (U.Q4_K, 14592, 32, 12, 32)], ids=lambda v: str(v))
def test_rows_that_stay_in_f32(sm100, stream, dtype, k, n, m, tail):
    """What the f32 kernels serve of a batch keeps their precision.  Against float64: 2e-7 to 1.2e-6 measured; the split GEMM, whose
    operands have 16 bits, leaves 5e-6 or more."""
    wq = U.quantize(dtype, U.seeded_weights(7000 + dtype + k, n, k))
    x = U.seeded_acts(3 * m + k, m, k)
    want = x.astype(np.float64) @ sgref.dequantize(dtype, wq, k).astype(np.float64).T
    got = U.device_mul_mat(sm100, stream, dtype, U.PACKED, wq, k, x)
    part = slice(n - tail, n)
    err = np.linalg.norm(got[:, part] - want[:, part]) / np.linalg.norm(want[:, part])
    assert err <= 2e-6, err
    assert sgref.nmse(got.astype(np.float64), want) <= 4 * TOL


# the second environment: as if there were no memory to be had
@pytest.mark.parametrize("env", [{}, {"SM100_CALL_SCRATCH": "0"}], ids=["", "no_memory"])
@pytest.mark.parametrize("dtype,m,k,n", [(U.Q6_K, 8, 768, 1061), (U.Q6_K, 200, 768, 1061), (U.Q4_0, 8, 768, 1061), (U.Q4_K, 24, 768, 1061), (U.Q4_K, 12, 2048, 8203)], ids=lambda v: str(v))
def test_first_product_of_a_process_is_captured(dtype, m, k, n, env):
    """Nothing has to come before the capture, and the graph holds kernel nodes only (kind 0): it can be copied, be part of another
    graph and have several instances."""
    import json
    import os
    import subprocess
    import sys
    worker = os.path.join(os.path.dirname(os.path.abspath(__file__)), "capture_worker.py")
    r = subprocess.run([sys.executable, worker, str(dtype), str(m), str(k), str(n)], capture_output=True, text=True, timeout=300, env=dict(os.environ, **env))
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    res = json.loads(r.stdout.strip().splitlines()[-1])
    assert res["kinds"] == [0], res
    assert res["worst"] <= (COLUMNS_TOL if n == 8203 and not env else TOL), res


@pytest.mark.parametrize("family,dtype,m", [(0, U.Q8_0, 40), (1, U.Q4_0, 12), (2, U.Q4_K, 1), (2, U.Q4_K, 4)], ids=lambda v: str(v))
def test_give_ups_of_replays_are_reported(sm100, stream, family, dtype, m):
    """A kernel that gives up on a wait leaves its mark in a host word (written here by the test): every synchronisation and blocking
    read of the device reports it once, also when the kernel came from a graph that was captured long before."""
    k, n = 512, 96
    wb = U.to_device(sm100, stream, sm100.pack(dtype, k, U.quantize(dtype, U.seeded_weights(3, n, k))))
    xb, yb = U.to_device(sm100, stream, U.seeded_acts(4, m, k)), sm100.Buffer(4 * n * m)
    sm100.mul_mat(stream, dtype, U.PACKED, wb, k, n, xb, m, yb)
    stream.sync()
    graph = sm100.Graph(stream)
    with graph:
        sm100.mul_mat(stream, dtype, U.PACKED, wb, k, n, xb, m, yb)
    word = C.POINTER(C.c_int)()
    sm100.check(sm100.lib().sm100_fault_word(0, family, C.byref(word)), "fault_word")
    graph.launch()
    stream.sync()
    other = sm100.Stream(0)
    for wait in (stream.sync, lambda: yb.download(stream, np.float32, 1), other.sync):
        graph.launch()
        assert word[0] == 0
        word[0] = 4
        with pytest.raises(sm100.Sm100Error, match="gave up.*site 3") as e:
            wait()
        assert e.value.status == 4 and word[0] == 0
        stream.sync()
    graph.destroy()
    other.close()
    for b in (wb, xb, yb):
        b.free()
