"""GPU parity of the column kernel (packed weights, up to 8 columns, integers times two f16 numbers on mma.sync) against float64.

Tolerance: activations have 22 bits (2^-23), block scales and block sums are f32; the tensor core truncates its sums (2^-23 of the
largest term, two to four MMAs a block), and the minima of Q4_K (and the offset of 32 in the form of Q6_K that keeps it) make the terms up to three times as large as
what is left of them: 3 (2^-23 + 4 2^-23) is 1.8e-6 at most per block, measured 8e-8 to 1.4e-6 over whole rows.  Bound: 4e-6, so NMSE 1.6e-11.
"""
import numpy as np
import pytest

from oracle import sgref
from tests import util as U

pytestmark = pytest.mark.gpu
TOL = 1.6e-11


def _want(dtype, wq, k, x):
    return x.astype(np.float64) @ sgref.dequantize(dtype, wq, k).astype(np.float64).T


def _served(sm100):
    return (sm100.lib().sm100_matvec_last_kernel() or b"").decode()


def _check(sm100, stream, dtype, k, n, m, seed=0):
    few = min(n, 416)   # rows repeat, not in step with any tile, so that the oracle has few to multiply
    wq = U.quantize(dtype, U.seeded_weights(900 + dtype + k, few, k))
    x = U.seeded_acts(3 * m + k + seed, m, k)
    want = _want(dtype, wq, k, x)[:, np.arange(n) % few]
    got = U.device_mul_mat(sm100, stream, dtype, U.PACKED, np.ascontiguousarray(np.resize(wq, (n, wq.shape[1]))), k, x)
    assert (sm100.lib().sm100_matvec_last_kernel() or b"").decode() == ("quant_cols" if n % 16 == 0 else "quant_cols+rows")
    for t in range(m):
        assert sgref.nmse(got[t].astype(np.float64), want[t]) <= TOL, (t, sgref.nmse(got[t].astype(np.float64), want[t]))
    for r0 in range(0, n, 16):   # every row tile on its own
        assert sgref.nmse(got[:, r0:r0 + 16].astype(np.float64), want[:, r0:r0 + 16]) <= 4 * TOL, r0


# one unit of K, an odd number of units, 17 and 48 (clusters of two and three CTAs, 17 unevenly); fewer and more row tiles than CTAs, rows behind the last
# whole tile; one window of row tiles and several
SHAPES = [(256, 16384 + 16), (1280, 4096 + 5), (4352, 4096), (12288, 4096 + 48), (4096, 12288 + 16), (2048, 148 * 16 * 16)]


@pytest.mark.parametrize("dtype", U.QUANT, ids=lambda d: U.NAMES[d])
@pytest.mark.parametrize("m", [3, 4, 5, 8])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: f"k{s[0]}n{s[1]}")
def test_shapes(sm100, stream, dtype, shape, m):
    k, n = shape
    if dtype == U.Q4_K and m < 5:
        k = {12288: 13312}.get(k, k)
        if k <= 12288:
            pytest.skip("served by the integer kernel")
    _check(sm100, stream, dtype, k, n, m)


# the longest rows, few tiles, one and two columns; one column of Q6_K where an f32 kernel served before (signed integers)
@pytest.mark.parametrize("dtype,k,n,m", [(U.Q6_K, 16384, 1024, 2), (U.Q4_0, 512, 1024, 3), (U.Q8_0, 8192, 1040, 2), (U.Q4_K, 13824, 1024, 8), (U.Q4_K, 13312, 1024, 2),
                                         (U.Q6_K, 4096, 8192, 1), (U.Q6_K, 12288, 1040, 1), (U.Q6_K, 4352, 5008, 1), (U.Q6_K, 1280, 52016, 1)], ids=lambda v: str(v))
def test_longest_rows_few_tiles_one_column(sm100, stream, dtype, k, n, m):
    _check(sm100, stream, dtype, k, n, m)


def test_one_column_keeps_the_precision_of_f32(sm100, stream):
    """Rows that the f32 kernels served (2.3e-7 against float64)."""
    k, n = 5120, 5120
    wq = U.quantize(U.Q6_K, U.seeded_weights(1, n, k))
    x = U.seeded_acts(2, 1, k)
    got, want = U.device_mul_mat(sm100, stream, U.Q6_K, U.PACKED, wq, k, x), _want(U.Q6_K, wq, k, x)
    assert np.linalg.norm(got - want) / np.linalg.norm(want) <= 2e-7


@pytest.mark.parametrize("dtype", U.QUANT, ids=lambda d: U.NAMES[d])
@pytest.mark.parametrize("m", [4, 8])
def test_magnitudes_and_poison(sm100, stream, dtype, m):
    """A column keeps its precision whatever its magnitude, a NaN or an infinity poisons its own column only, and large block scales stay finite."""
    k, n = 13312 if dtype == U.Q4_K and m == 4 else 1024, 4096
    wq = np.ascontiguousarray(np.resize(U.quantize(dtype, U.seeded_weights(5, 416, k) * np.float32(1e4 if dtype in (U.Q4_0, U.Q8_0) else 1.0)), (n, U.quantize(dtype, U.seeded_weights(5, 1, k)).shape[1])))
    for poison in (np.nan, np.inf, -np.inf):
        x = U.seeded_acts(6, m, k)
        x[0] *= 1e30
        x[1] *= 1e-25
        x[1, 300:400] = 0.0
        x[2, 5] = 3e6
        x[3, 777] = poison
        got = U.device_mul_mat(sm100, stream, dtype, U.PACKED, wq, k, x).astype(np.float64)
        want = _want(dtype, wq[:416], k, np.where(np.isfinite(x), x, 0))[:, np.arange(n) % 416]
        assert not np.isfinite(got[3]).any()
        for t in [0, 1, 2] + list(range(4, m)):
            assert sgref.nmse(got[t], want[t]) <= TOL, t


@pytest.mark.parametrize("k,n", [(8192, 5120), (4352, 5008), (7168, 4096)])
def test_one_column_of_every_row_that_f32_kernels_served(sm100, stream, k, n):
    """K = 8192 among them, which the streaming kernel would serve: the bound of the rows above."""
    wq = np.ascontiguousarray(np.resize(U.quantize(U.Q6_K, U.seeded_weights(k, 416, k)), (n, k // 256 * 210)))
    x = U.seeded_acts(n, 1, k)
    got, want = U.device_mul_mat(sm100, stream, U.Q6_K, U.PACKED, wq, k, x), _want(U.Q6_K, wq[:416], k, x)[:, np.arange(n) % 416]
    assert _served(sm100).startswith("quant_cols")
    assert np.linalg.norm(got - want) / np.linalg.norm(want) <= 2e-7


def _zero_columns(dtype, k, n, large):
    """Packed rows (416, repeated) whose weights `large` are zero: the integer 0 in the three formats without minima."""
    w = U.seeded_weights(77 + dtype + k, 416, k)
    w[:, large] = 0.0
    wq = U.quantize(dtype, w)
    assert not sgref.dequantize(dtype, wq, k)[:, large].any()
    return wq, np.ascontiguousarray(np.resize(wq, (n, wq.shape[1])))


@pytest.mark.parametrize("ratio", [1e3, 1e5, 1e7], ids=lambda v: f"{v:.0e}")
@pytest.mark.parametrize("dtype,k,n,m", [(U.Q4_0, 1024, 4096, 4), (U.Q4_0, 1024, 4096, 8), (U.Q8_0, 1024, 4096, 4), (U.Q8_0, 1024, 4096, 8),
                                         (U.Q6_K, 1024, 4096, 3), (U.Q6_K, 1024, 4096, 8), (U.Q4_0, 5120, 6144, 1)], ids=lambda v: str(v))
def test_large_activations_at_zero_weights(sm100, stream, dtype, k, n, m, ratio):
    """A weight of zero leaves nothing of its activation, however large that is beside the 255 others of its unit.  The others then have 22 bits and
    no cancelled offsets: the bound of ordinary inputs."""
    large = np.arange(7, k, 256)
    wq, full = _zero_columns(dtype, k, n, large)
    x = U.seeded_acts(m + k, m, k)
    x[:, large] = np.float32(ratio) * np.where(np.arange(large.size) % 2, -1.0, 1.0).astype(np.float32)
    want = _want(dtype, wq, k, x)[:, np.arange(n) % 416]
    got = U.device_mul_mat(sm100, stream, dtype, U.PACKED, full, k, x)
    assert _served(sm100).startswith("quant_cols")
    for t in range(m):
        assert sgref.nmse(got[t].astype(np.float64), want[t]) <= TOL, (t, sgref.nmse(got[t].astype(np.float64), want[t]))


@pytest.mark.parametrize("ratio", [1e4, 1e6, 1e7, 1e9], ids=lambda v: f"{v:.0e}")
@pytest.mark.parametrize("k,n", [(5120, 5120), (8192, 5120)])
def test_one_column_keeps_24_bits_beside_large_activations(sm100, stream, k, n, ratio):
    """f32 kernels served these rows: 24 bits of each activation whatever stands beside it, the bound of ordinary inputs."""
    large = np.arange(7, k, 256)
    wq, full = _zero_columns(U.Q6_K, k, n, large)
    x = U.seeded_acts(3, 1, k)
    x[:, large] = np.float32(ratio)
    want = _want(U.Q6_K, wq, k, x)[:, np.arange(n) % 416]
    got = U.device_mul_mat(sm100, stream, U.Q6_K, U.PACKED, full, k, x)
    assert _served(sm100).startswith("quant_cols")
    assert np.linalg.norm(got - want) / np.linalg.norm(want) <= 2e-7


@pytest.mark.parametrize("k,n", [(5120, 5120), (8192, 5120)])
@pytest.mark.parametrize("where", [[5], [5, 300], [4095, 4900]], ids=str)
def test_one_column_infinities(sm100, stream, k, n, where):
    """What f32 kernels make of an infinite activation: an infinity of the product's sign, NaN where the weight is zero or infinities cancel; finite
    activations of any size beside it in the same unit do not show."""
    large = np.array([64, 400])
    wq, full = _zero_columns(U.Q6_K, k, n, large)
    x = U.seeded_acts(4, 1, k)
    x[0, 9], x[0, 310], x[0, 4097] = 1e30, -1e30, 1e-30
    for i, j in enumerate(where):
        x[0, j] = np.inf if i == 0 else -np.inf
    with np.errstate(invalid="ignore"):
        w = sgref.dequantize(U.Q6_K, wq, k).astype(np.float64)
        want = np.zeros(len(w)) + sum(w[:, j] * float(x[0, j]) for j in where)   # finite terms do not change an infinity or a NaN
    got = U.device_mul_mat(sm100, stream, U.Q6_K, U.PACKED, full, k, x)[0]
    assert _served(sm100).startswith("quant_cols")
    assert np.array_equal(got[:416], want.astype(np.float32), equal_nan=True)
    assert np.array_equal(got, got[np.arange(n) % 416], equal_nan=True)
    if len(where) == 1:
        assert np.isinf(got).any()


@pytest.mark.parametrize("exponent", [-120, -127, -135])
@pytest.mark.parametrize("dtype,k,n,m", [(U.Q6_K, 5120, 5120, 1), (U.Q6_K, 1024, 4096, 3), (U.Q4_0, 1024, 4096, 8), (U.Q8_0, 1024, 4096, 2)], ids=lambda v: str(v))
def test_columns_of_subnormal_numbers(sm100, stream, dtype, k, n, m, exponent):
    """Activations that are subnormal numbers count like others; block scales of 2^10 keep the results normal, so the bound is that of their own bits: one
    rounding of each input to 2^-149 is in the inputs already."""
    wq = U.quantize(dtype, U.seeded_weights(8, 416, k) * np.float32(2.0 ** 14))
    full = np.ascontiguousarray(np.resize(wq, (n, wq.shape[1])))
    x = (U.seeded_acts(9, m, k).astype(np.float64) * 2.0 ** exponent).astype(np.float32)
    want = _want(dtype, wq, k, x)[:, np.arange(n) % 416] * 2.0 ** -exponent
    got = U.device_mul_mat(sm100, stream, dtype, U.PACKED, full, k, x).astype(np.float64) * 2.0 ** -exponent
    assert _served(sm100).startswith("quant_cols")
    for t in range(m):
        assert sgref.nmse(got[t], want[t]) <= TOL, (t, sgref.nmse(got[t], want[t]))


def _child(args, env):
    import os
    import subprocess
    import sys
    r = subprocess.run([sys.executable] + args, capture_output=True, text=True, timeout=900, env=dict(os.environ, **env))
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    return r.stdout.strip().splitlines()[-1]


@pytest.mark.parametrize("env,left", [({}, ["q4_0", "q4_k", "q6_k", "q8_0"]), ({"SM100_QUANT_COLS": "0"}, []), ({"SM100_Q6K_IMMA": "0"}, ["q4_0", "q4_k", "q8_0"]),
                                      ({"SM100_B32_IMMA": "0"}, ["q4_k", "q6_k"]), ({"SM100_Q4K_IMMA": "0"}, ["q4_0", "q6_k", "q8_0"]),
                                      ({"SM100_Q4K_IMMA": "0", "SM100_Q4K_MMA": "0", "SM100_Q6K_IMMA": "0", "SM100_B32_IMMA": "0", "SM100_MV_WIDE": "0"}, [])],
                         ids=["default", "none", "no_q6k", "no_b32", "no_q4k", "cuda_core_only"])
def test_switches(env, left):
    """The family has a switch, and goes with those of the families whose calls it takes.  Every result against the oracle in the worker, bar of the matvec tests."""
    import json
    import os
    out = json.loads(_child([os.path.join(os.path.dirname(os.path.abspath(__file__)), "matvec_branch_worker.py")], env))
    assert out["worst"] <= 1e-6, out
    assert sorted({name.split(":")[0] for name in out["kernels"] if "quant_cols" in name}) == left


BATCHES = """
import numpy as np
from scrapgpulibrary_b200 import capi
from tests import util as U
s = capi.Stream(0)
bad = []
for dtype, k, n in [(U.Q4_0, 1024, 4112), (U.Q8_0, 2048, 6000), (U.Q6_K, 4096, 4096)]:
    wq = U.quantize(dtype, np.resize(U.seeded_weights(dtype + k, 250, k), (n, k)))
    x = U.seeded_acts(k, 32, k)
    both = U.device_mul_mat(capi, s, dtype, U.PACKED, wq, k, x)
    bad += [(dtype, m) for m in (24, 9, 8, 7, 5) if not np.array_equal(U.device_mul_mat(capi, s, dtype, U.PACKED, wq, k, x[:m]), both[:m])]
print(bad)
"""


def test_without_it_columns_do_not_depend_on_their_batch():
    """Bit for bit over 5 to 32 columns, from 4096 rows on too: for callers that want that rather than the faster and more accurate kernel."""
    import os
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = {"SM100_QUANT_COLS": "0", "PYTHONPATH": root + os.pathsep + os.environ.get("PYTHONPATH", "")}
    assert _child(["-c", BATCHES], env) == "[]"


# what plan_cols deals to clusters of five (35, 43 and 50 units; two row tiles a CTA and one) and six (53 and 54 units) CTAs, mostly unevenly; with rows behind the last whole tile
@pytest.mark.parametrize("dtype,k,n,m", [(U.Q6_K, 11008, 1184, 4), (U.Q4_0, 12800, 1093, 4), (U.Q8_0, 8960, 1552, 2), (U.Q4_K, 11008, 1184, 8), (U.Q4_K, 13824, 1632, 2),
                                         (U.Q6_K, 13568, 1648, 4), (U.Q4_K, 13568, 1616, 5), (U.Q8_0, 13824, 1653, 3)], ids=lambda v: str(v))
def test_clusters_of_five_and_six(sm100, stream, dtype, k, n, m):
    _check(sm100, stream, dtype, k, n, m)


# one column where the kernel that served it before is the faster one, and its neighbours: rows of one to three units below 24576 rows; K = 8192 with few rows or rows left over
@pytest.mark.parametrize("dtype,k,n,name", [(U.Q4_0, 512, 12288, "matvec_b32_imma"), (U.Q8_0, 1024, 16384, "matvec_b32_imma"), (U.Q4_0, 1280, 12288, "quant_cols"), (U.Q8_0, 512, 24576, "quant_cols"),
                                            (U.Q6_K, 512, 12288, "matvec_q6k_imma"), (U.Q6_K, 768, 12288, "quant_cols"), (U.Q6_K, 8192, 4592, "matvec_wide"), (U.Q6_K, 8192, 4608, "quant_cols"),
                                            (U.Q6_K, 8192, 5003, "matvec_wide")], ids=lambda v: str(v))
def test_one_column_takes_the_faster_kernel(sm100, stream, dtype, k, n, name):
    """Bound: 16-bit activations with a scale per 16 or 32 of them (1e-4), as in the matvec tests."""
    wq = np.ascontiguousarray(np.resize(U.quantize(dtype, U.seeded_weights(k, 416, k)), (n, U.quantize(dtype, U.seeded_weights(1, 1, k)).shape[1])))
    x = U.seeded_acts(n, 1, k)
    got, want = U.device_mul_mat(sm100, stream, dtype, U.PACKED, wq, k, x), _want(dtype, wq[:416], k, x)[:, np.arange(n) % 416]
    assert _served(sm100) == name
    assert np.linalg.norm(got - want) / np.linalg.norm(want) <= 1e-4
