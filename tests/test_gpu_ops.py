"""GPU: every kernel of the per-operator path through the C ABI against the CPU oracle.
Integer and byte results must be identical; f32 results differ only by summation order."""
import ctypes as C
import os
import threading

import numpy as np
import pytest

from spy_b200 import backend as B
from spy_b200 import quants

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(__file__), "golden")


@pytest.fixture(scope="module")
def be():
    b = B.B200Backend(0)
    yield b
    b.close()


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)


def close(got, want, rel=0.0):
    """f32 results are required to be bit-identical: every kernel follows the CPU's summation order."""
    return np.array_equal(bits(got), bits(want))


def run(be, op, inputs, out_ne, out_type=B.FP32, host_out=False, **params):
    """inputs: list of (np array, number_type, ne, nb or None, node_type). Returns the f32/u16 output array."""
    d = B.OpDesc()
    d.op_type, d.num_input = B.OP[op], len(inputs)
    dev = []
    for i, (a, nt, ne, nb, node) in enumerate(inputs):
        if node == B.NODE_IO:
            a = np.ascontiguousarray(a)
            ptr = a.ctypes.data
            dev.append((None, a))
        else:
            ptr = be.upload(a)
            dev.append((ptr, a))
        d.input[i] = B.make_tensor(ptr, nt, ne, nb, node)
    esz = 4 if out_type in (B.FP32, B.INT32) else 2
    n_out = int(np.prod(out_ne))
    host_buf = np.zeros(n_out, dtype=np.float32 if esz == 4 else np.uint16)
    if op == "Copy":
        d.output = B.make_tensor(None, out_type, out_ne)
    elif host_out:
        d.output = B.make_tensor(host_buf.ctypes.data, out_type, out_ne, None, B.NODE_IO)
    else:
        po = be.alloc_memory(max(1, n_out * esz))
        d.output = B.make_tensor(po, out_type, out_ne)
    d.softmax_scale = params.get("scale", 0.0)
    d.norm_eps = params.get("eps", 0.0)
    d.view_offset = params.get("offset", 0)
    if op == "Rope":
        r = d.rope
        r.mode, r.num_dim, r.num_context, r.num_origin_context = 0, params["n_dim"], params.get("n_context", 512), 4096
        r.freq_base, r.freq_scale, r.extend_factor, r.attention_factor, r.beta_fast, r.beta_slow = params.get("base", 10000.0), 1.0, 0.0, 1.0, 32.0, 1.0
    be.submit(d)
    be.sync()
    if op == "Copy":
        return d
    if host_out:
        res = host_buf
    else:
        res = be.download(d.output.data, (n_out,), np.float32 if esz == 4 else np.uint16)
        be.dealloc_memory(d.output.data, max(1, n_out * esz))
    for ptr, a in dev:
        if ptr:
            be.dealloc_memory(ptr, max(1, a.nbytes))
    return res


# ----------------------------------------------------------------------------- exact arithmetic
def test_q8_quantizer_bytes_golden(be):
    g = np.load(os.path.join(GOLD, "ops_reference.npz"))
    assert np.array_equal(be.quantize_q8_0(g["q8_x"]), g["q8_blocks"])


@pytest.mark.parametrize("seed", [0, 1])
def test_q8_quantizer_bytes_random(be, oracle, seed):
    rng = np.random.default_rng(seed)
    x = (rng.standard_normal(32 * 4096) * rng.choice([1e-6, 1e-2, 1.0, 1e3], size=32 * 4096)).astype(np.float32)
    x[:64] = 0.0
    x[64:96] = np.arange(32) * 0.5
    assert np.array_equal(be.quantize_q8_0(x), oracle.quantize_q8_0(x))


def test_q8_quantizer_empty(be):
    assert be.quantize_q8_0(np.zeros(0, dtype=np.float32)).size == 0


@pytest.mark.parametrize("qt", [quants.Q4_0, quants.Q8_0])
@pytest.mark.parametrize("k", [32, 4096, 11008])
def test_integer_block_dots_identical(be, oracle, qt, k):
    rng = np.random.default_rng(k + qt)
    w = quants.quantize((rng.standard_normal((1, k)) * 0.02).astype(np.float32), qt)[0]
    xq = oracle.quantize_q8_0(rng.standard_normal(k).astype(np.float32))
    assert np.array_equal(be.block_dots(qt, w, xq, k), oracle.blockdots(qt, w, xq))


def test_block_dots_extreme_values(be, oracle):
    k = 64
    w = np.zeros(k // 32 * 18, dtype=np.uint8)
    w[0:2] = np.frombuffer(np.float16(1.0).tobytes(), dtype=np.uint8)
    w[2:18] = 0xFF; w[18:20] = w[0:2]; w[20:36] = 0x00          # all nibbles 15, then all 0 (i.e. -8)
    xq = np.zeros(k // 32 * 34, dtype=np.uint8)
    xq[0:2] = w[0:2]; xq[2:34] = 127; xq[34:36] = w[0:2]; xq[36:68] = 128   # int8 127 and -128
    assert np.array_equal(be.block_dots(quants.Q4_0, w, xq, k), oracle.blockdots(quants.Q4_0, w, xq))


# ----------------------------------------------------------------------------- MatMul
SHAPES = [(4096, 4096), (11008, 4096), (4096, 11008), (32000, 4096)]   # (rows N, inner K)


@pytest.mark.parametrize("qt", [quants.Q4_0, quants.Q8_0])
@pytest.mark.parametrize("n,k", [(64, 256), (132, 1024), (4, 32)])
@pytest.mark.parametrize("t", [1, 3, 8, 11])
def test_matmul_small_shapes(be, oracle, qt, n, k, t):
    rng = np.random.default_rng(n * k + t)
    w = quants.quantize((rng.standard_normal((n, k)) * 0.02).astype(np.float32), qt)
    x = rng.standard_normal((t, k)).astype(np.float32)
    got = run(be, "MatMul", [(w, qt, (k, n), None, B.NODE_CONSTANT), (x, B.FP32, (k, t), None, B.NODE_DYNAMIC)], (n, t)).reshape(t, n)
    want = oracle.matmul(qt, w, k, n, x)
    assert close(got, want)


# MatMul of a prompt on the tensor cores (tcgen05): the same operator, the same bits
@pytest.mark.parametrize("qt", [quants.Q4_0, quants.Q8_0])
@pytest.mark.parametrize("n,k,t,norm", [(128, 32, 1, False), (128, 256, 16, False), (256, 1024, 37, True), (384, 96, 5, False), (128, 4096, 64, True),
                                        (1024, 11008, 19, False), (200, 512, 21, False), (4, 64, 3, False)])
def test_prefill_matmul_matches_oracle(be, oracle, qt, n, k, t, norm):
    """Block counts below, at and above the pipeline depths (1, 3, 8, 32, 128, 344 blocks), ragged token tiles, row counts that
    leave the last 128-row tile partly padding, with and without the RMSNorm in front; activations with a few outliers so that block scales differ widely."""
    rng = np.random.default_rng(n + k + t + qt)
    w = quants.quantize((rng.standard_normal((n, k)) * 0.02).astype(np.float32), qt)
    x = rng.standard_normal((t, k)).astype(np.float32)
    x[rng.integers(0, t, 8), rng.integers(0, k, 8)] *= 40.0
    nw = (1.0 + 0.1 * rng.standard_normal(k)).astype(np.float32) if norm else None
    got = be.prefill_matmul(qt, w, n, k, x, nw, 1e-5)
    xin = oracle.mul_rows(oracle.rmsnorm(x, 1e-5), nw) if norm else x
    want = oracle.matmul(qt, w, k, n, xin)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("qt", [quants.Q4_0, quants.Q8_0])
@pytest.mark.parametrize("n,k,t", [(2560, 32, 160), (2560, 96, 160), (2564, 160, 153), (9600, 160, 24), (9476, 224, 23), (640, 4096, 16)])
def test_prefill_matmul_walks_tiles_of_both_widths(be, oracle, qt, n, k, t):
    """More tiles than the chip has SMs (a CTA goes on from one tile to the next) in the wide and in the narrow token tiles, with
    block counts that end inside a step and odd numbers of steps, so that tiles begin on either accumulator buffer."""
    rng = np.random.default_rng(n + k + t + qt)
    w = quants.quantize((rng.standard_normal((n, k)) * 0.02).astype(np.float32), qt)
    x = rng.standard_normal((t, k)).astype(np.float32)
    got = be.prefill_matmul(qt, w, n, k, x)
    want = oracle.matmul(qt, w, k, n, x)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("qt", [quants.Q4_0, quants.Q8_0])
@pytest.mark.parametrize("n,k,t", [(19204, 1600, 7), (19204, 2880, 15), (132, 3104, 9), (516, 2976, 32)])
def test_prefill_matmul_shared_by_two_ctas(be, oracle, qt, n, k, t):
    """The form whose tiles are shared by a cluster of two CTAs beside that of one CTA a tile, in narrow and in wide token tiles: three rounds of tiles
    (the hand-over's buffer is used again), odd numbers of steps that end inside a step, a last row tile of four rows, ragged and full token tiles."""
    rng = np.random.default_rng(n + k + t + qt)
    w = quants.quantize((rng.standard_normal((n, k)) * 0.02).astype(np.float32), qt)
    x = rng.standard_normal((t, k)).astype(np.float32)
    x[rng.integers(0, t, 8), rng.integers(0, k, 8)] *= 40.0
    want = oracle.matmul(qt, w, k, n, x)
    for form in [(0, 0), (8, 1), (16, 1), (8, 2), (16, 2)]:
        got = be.prefill_matmul(qt, w, n, k, x, form=form)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), form


@pytest.mark.parametrize("qt", [quants.Q4_0, quants.Q8_0])
@pytest.mark.parametrize("n,k,t", [(9604, 4128, 32), (2564, 4128, 118), (6148, 2080, 130), (19204, 1568, 36)])
def test_prefill_matmul_shares_its_last_tiles(be, oracle, qt, n, k, t):
    """One to four rounds and a fraction of tiles in every form: the last tiles are cut between neighbours at odd and even steps, rows end inside a step, and
    calls follow one another (what one leaves in the buffer of the handing over, the next one does not find)."""
    rng = np.random.default_rng(n + k + t + qt)
    w = quants.quantize((rng.standard_normal((n, k)) * 0.02).astype(np.float32), qt)
    x = rng.standard_normal((t, k)).astype(np.float32)
    rows = np.unique(np.r_[np.arange(0, n, 128), n - 1, rng.integers(0, n, 60)])
    want = oracle.matmul(qt, np.ascontiguousarray(w[rows]), k, len(rows), x)
    for form in [(16, 1), (8, 1), (16, 2), (8, 2), (0, 0), (16, 1)]:
        got = be.prefill_matmul(qt, w, n, k, x, form=form)
        assert np.array_equal(got[:, rows].view(np.uint32), want.view(np.uint32)), form


@pytest.mark.parametrize("qt", [quants.Q4_0, quants.Q8_0])
@pytest.mark.parametrize("n,k,t", [(9604, 4128, 32), (2564, 4128, 118), (6148, 2080, 130), (19204, 1568, 36), (18944, 672, 32), (19204, 96, 24)])
def test_prefill_matmul_with_last_tiles_shared_and_whole(be, oracle, qt, n, k, t):
    """More tiles than walkers in every form, up to eleven rounds, and each form with its last tiles shared beside whole, whatever the sizes' own choice:
    they are cut between neighbours at odd and even steps (in whole rounds also at a tile's end), rows end inside a step or have two steps, and calls follow
    one another (what one leaves in the buffer of the handing over, the next one does not find)."""
    rng = np.random.default_rng(n + k + t + qt)
    w = quants.quantize((rng.standard_normal((n, k)) * 0.02).astype(np.float32), qt)
    x = rng.standard_normal((t, k)).astype(np.float32)
    rows = np.unique(np.r_[np.arange(0, n, 128), n - 1, rng.integers(0, n, 60)])
    want = oracle.matmul(qt, np.ascontiguousarray(w[rows]), k, len(rows), x)
    for form in [(16, 1, 2), (8, 1, 2), (16, 2, 2), (8, 2, 2), (0, 0, 0), (16, 1, 1), (8, 1, 1), (16, 2, 1), (8, 2, 1), (16, 1, 2)]:
        assert form[2] == 0 or B.prefill_plan(qt, n, k, t, form) == form
        got = be.prefill_matmul(qt, w, n, k, x, form=form)
        assert np.array_equal(got[:, rows].view(np.uint32), want.view(np.uint32)), form


@pytest.mark.parametrize("qt,k", [(quants.Q4_0, 2272), (quants.Q4_0, 4128), (quants.Q8_0, 8192), (quants.Q4_0, 8224), (quants.Q4_K, 4352), (quants.Q4_K, 9216),
                                  (quants.Q8_0, 13824), (quants.Q4_0, 14336), (quants.Q4_K, 13824), (quants.Q6_K, 14336)])
def test_prefill_quantizer_of_normed_rows(be, oracle, qt, k):
    """RMSNorm in front of the quantizer at the edges of its forms: one, two and four groups a thread, rows below and above what the four
    warps' running sum takes; a row of zeros among the others (the sum then falls back to the plain chain)."""
    rng = np.random.default_rng(k)
    n, t = 8, 3
    w = quants.quantize((rng.standard_normal((n, k)) * 0.02).astype(np.float32), qt)
    x = rng.standard_normal((t, k)).astype(np.float32)
    x[1] = 0.0
    nw = (1.0 + 0.1 * rng.standard_normal(k)).astype(np.float32)
    got = be.prefill_matmul(qt, w, n, k, x, nw, 1e-5)
    xin = oracle.mul_rows(oracle.rmsnorm(x, 1e-5), nw)
    want = oracle.matmul(qt, w, k, n, xin)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("qt", [quants.Q4_K, quants.Q6_K])
@pytest.mark.parametrize("n,k,t", [(19000, 256, 16), (2564, 768, 250), (1284, 512, 1000), (516, 2304, 31), (132, 256, 48), (640, 4096, 9)])
def test_prefill_matmul_k_quants_walk_tiles_of_all_widths(be, oracle, qt, n, k, t):
    """Token tiles of 16, 32 and 64, more tiles than SMs, ragged last tiles in both directions, one super-block and sixteen."""
    rng = np.random.default_rng(n + k + t + qt)
    w = quants.quantize((rng.standard_normal((n, k)) * 0.02).astype(np.float32), qt)
    x = rng.standard_normal((t, k)).astype(np.float32)
    got = be.prefill_matmul(qt, w, n, k, x)
    rows, cols = np.unique(np.r_[0, n - 1, rng.integers(0, n, 60)]), np.unique(np.r_[0, t - 1, rng.integers(0, t, 40)])
    want = oracle.matmul(qt, np.ascontiguousarray(w[rows]), k, len(rows), x[cols])
    assert np.array_equal(got[np.ix_(cols, rows)].view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("qt", [quants.Q4_K, quants.Q6_K])
@pytest.mark.parametrize("n,k,t", [(2564, 2304, 490), (9604, 4352, 63), (19204, 2560, 9), (1028, 5632, 600)])
def test_prefill_matmul_k_quants_share_their_last_tiles(be, oracle, qt, n, k, t):
    """One to four rounds and a fraction of tiles in every width, cut between neighbours at super-blocks; calls follow one another."""
    rng = np.random.default_rng(n + k + t + qt)
    w = quants.quantize((rng.standard_normal((n, k)) * 0.02).astype(np.float32), qt)
    x = rng.standard_normal((t, k)).astype(np.float32)
    rows, cols = np.unique(np.r_[np.arange(0, n, 128), n - 1, rng.integers(0, n, 20)]), np.unique(np.r_[np.arange(0, t, 16), t - 1])
    want = oracle.matmul(qt, np.ascontiguousarray(w[rows]), k, len(rows), x[cols])
    for form in [(64, 1), (32, 1), (16, 1), (0, 0), (64, 1)]:
        got = be.prefill_matmul(qt, w, n, k, x, form=form)
        assert np.array_equal(got[np.ix_(cols, rows)].view(np.uint32), want.view(np.uint32)), form


@pytest.mark.parametrize("qt", [quants.Q4_K, quants.Q6_K])
@pytest.mark.parametrize("n,k,t", [(2564, 2304, 490), (9604, 4352, 129), (19204, 2560, 9), (1028, 5632, 1100), (18944, 512, 128)])
def test_prefill_matmul_k_quants_with_last_tiles_shared_and_whole(be, oracle, qt, n, k, t):
    """Tiles of every width (where there are more of them than CTAs) with the last ones shared, cut between neighbours at super-blocks, beside whole,
    whatever the sizes' own choice; calls follow one another."""
    rng = np.random.default_rng(n + k + t + qt)
    w = quants.quantize((rng.standard_normal((n, k)) * 0.02).astype(np.float32), qt)
    x = rng.standard_normal((t, k)).astype(np.float32)
    rows, cols = np.unique(np.r_[np.arange(0, n, 128), n - 1, rng.integers(0, n, 20)]), np.unique(np.r_[np.arange(0, t, 16), t - 1])
    want = oracle.matmul(qt, np.ascontiguousarray(w[rows]), k, len(rows), x[cols])
    for form in [(64, 1, 2), (32, 1, 2), (16, 1, 2), (0, 0, 0), (64, 1, 1), (32, 1, 1), (16, 1, 1), (64, 1, 2)]:
        assert form[2] == 0 or B.prefill_plan(qt, n, k, t, form) == form
        got = be.prefill_matmul(qt, w, n, k, x, form=form)
        assert np.array_equal(got[np.ix_(cols, rows)].view(np.uint32), want.view(np.uint32)), form


@pytest.mark.parametrize("qt", [quants.Q4_K, quants.Q6_K])
@pytest.mark.parametrize("n,k,t,norm", [(128, 256, 1, False), (256, 1024, 70, True), (128, 2048, 64, False), (384, 4096, 129, True), (256, 11008 - 11008 % 256, 33, False)])
def test_prefill_matmul_k_quants_match_the_restatement(be, oracle, qt, n, k, t, norm):
    """K-quant weights through the tensor-core prompt kernel: 1 to 43 super-blocks, ragged tiles of 64 tokens, with and without
    the RMSNorm in front; bit-identical to the CPU restatement (the reference has no arithmetic for these types)."""
    rng = np.random.default_rng(n + k + t + qt)
    w = quants.quantize((rng.standard_normal((n, k)) * 0.02).astype(np.float32), qt)
    x = rng.standard_normal((t, k)).astype(np.float32)
    x[rng.integers(0, t, 8), rng.integers(0, k, 8)] *= 40.0
    nw = (1.0 + 0.1 * rng.standard_normal(k)).astype(np.float32) if norm else None
    got = be.prefill_matmul(qt, w, n, k, x, nw, 1e-5)
    xin = oracle.mul_rows(oracle.rmsnorm(x, 1e-5), nw) if norm else x
    want = oracle.matmul(qt, w, k, n, xin)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("qt", [quants.Q4_0, quants.Q8_0])
def test_prefill_matmul_extreme_bytes(be, oracle, qt):
    """Weight blocks written byte by byte over the whole range (Q8_0: -128 and 127 included, Q4_0: nibbles 0 and 15) against
    activations whose blocks quantize to +-127 and to zeros: every 8-bit value must be exact as an f16 operand of the tensor
    cores, and every sum in their f32 accumulators."""
    rng = np.random.default_rng(77 + qt)
    n, k, t = 136, 512, 21
    nb = k // 32
    bb = 18 if qt == quants.Q4_0 else 34
    raw = rng.integers(0, 256, size=(n, nb, bb), dtype=np.uint8)
    raw[:, :, 0:2] = rng.uniform(0.001, 0.05, size=(n, nb)).astype(np.float16).view(np.uint8).reshape(n, nb, 2)   # fp16 scales
    raw[0, :, 2:] = 0x80 if qt == quants.Q8_0 else 0x00          # a row of -128 / of nibble 0 (value -8)
    raw[1, :, 2:] = 0x7F if qt == quants.Q8_0 else 0xFF          # a row of 127 / of nibble 15 (value 7)
    w = np.ascontiguousarray(raw.reshape(n, nb * bb))
    x = rng.standard_normal((t, k)).astype(np.float32)
    x[0] = np.where(rng.random(k) < 0.5, 1.0, -1.0)              # every byte +-127
    x[1] = 0.0                                                   # every byte 0, scales 0
    x[2, ::2] = 0.0
    got = be.prefill_matmul(qt, w, n, k, x)
    want = oracle.matmul(qt, w, k, n, x)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


def test_prefill_matmul_full_size_rows_sample(be, oracle):
    """The 7B FFN-down shape with a 512-token prompt: a row and token sample against the oracle, bit for bit."""
    n, k, t = 4096, 11008, 512
    rng = np.random.default_rng(5)
    w = quants.quantize((rng.standard_normal((n, k), dtype=np.float32) * np.float32(0.02)), quants.Q4_0)
    x = rng.standard_normal((t, k)).astype(np.float32)
    got = be.prefill_matmul(quants.Q4_0, w, n, k, x)
    rows = np.unique(np.concatenate([[0, 127, 128, n - 1], rng.integers(0, n, size=28)]))
    cols = np.unique(np.concatenate([[0, 15, 16, t - 1], rng.integers(0, t, size=12)]))
    want = oracle.matmul(quants.Q4_0, np.ascontiguousarray(w[rows]), k, len(rows), x[cols])
    assert np.array_equal(got[np.ix_(cols, rows)].view(np.uint32), want.view(np.uint32))
    assert np.isfinite(got).all()


def test_prefill_kernel_wait_runs_out_and_is_reported():
    """A batch of blocks that is never copied: every role of the prompt kernel that waits for it gives up after the 2 ms
    bound, the kernel returns by itself, the status names the wait, and the backend computes correctly afterwards."""
    b = B.B200Backend(0)
    assert b.prefill_selftest_wait_timeout(2_000_000) in (4, 5, 6)
    w = quants.quantize((np.random.default_rng(1).standard_normal((128, 64)) * 0.02).astype(np.float32), quants.Q8_0)
    x = np.random.default_rng(2).standard_normal((3, 64)).astype(np.float32)
    got = b.prefill_matmul(quants.Q8_0, w, 128, 64, x)
    assert np.isfinite(got).all() and np.abs(got).max() > 0
    b.close()


def test_prefill_kernel_handover_too_late_is_reported_and_leaves_nothing(oracle):
    """Accumulators that come after their walker gave up: the kernels return by themselves, the status says so, and the words that were set
    too late are cleared, so that shared launches afterwards give the oracle's bits."""
    b = B.B200Backend(0)
    assert b.prefill_selftest_handoff_timeout(2_000_000) in (4, 5, 6)
    n, k, t = 9604, 4128, 32
    rng = np.random.default_rng(3)
    w = quants.quantize((rng.standard_normal((n, k)) * 0.02).astype(np.float32), quants.Q8_0)
    x = rng.standard_normal((t, k)).astype(np.float32)
    rows = np.arange(0, n, 97)
    want = oracle.matmul(quants.Q8_0, np.ascontiguousarray(w[rows]), k, len(rows), x)
    for form in [(16, 1), (16, 2)]:
        assert np.array_equal(b.prefill_matmul(quants.Q8_0, w, n, k, x, form=form)[:, rows].view(np.uint32), want.view(np.uint32)), form
    b.close()


def test_prefill_matmul_rejects_what_does_not_fit(be):
    w = np.zeros(100 * 18, dtype=np.uint8)
    x = np.zeros((2, 48), dtype=np.float32)
    with pytest.raises(B.SpybError) as e:
        be.prefill_matmul(quants.Q4_0, w, 100, 48, x)          # k not a multiple of 32
    assert e.value.status == B.UNSUPPORTED
    for qt, form in [(quants.Q4_0, (32, 1)), (quants.Q8_0, (0, 3)), (quants.Q4_K, (8, 0)), (quants.Q6_K, (16, 2)), (quants.Q4_0, (-8, 0))]:
        with pytest.raises(B.SpybError) as e:
            be.prefill_matmul(qt, w, 4, 256, np.zeros((2, 256), dtype=np.float32), form=form)          # no such form of the kernel
        assert e.value.status == B.UNSUPPORTED
    with pytest.raises(B.SpybError) as e:
        be.prefill_matmul(quants.Q4_K, w, 128, 128, np.zeros((2, 128), dtype=np.float32))   # K-quant rows: k a multiple of 256
    assert e.value.status == B.UNSUPPORTED


@pytest.mark.parametrize("qt", [quants.Q4_0, quants.Q8_0])
@pytest.mark.parametrize("n,k", SHAPES)
@pytest.mark.parametrize("t", [1, 4, 16])
def test_matmul_operator_sweep(be, oracle, qt, n, k, t):
    """The operator sweep of the benchmark configurations: weights N(0, 0.02), activations N(0, 1); the oracle checks a row sample."""
    rng = np.random.default_rng(99)
    w = quants.quantize((rng.standard_normal((n, k), dtype=np.float32) * np.float32(0.02)), qt)
    x = rng.standard_normal((t, k)).astype(np.float32)
    pw = be.upload_constant(f"sweep_{qt}_{n}_{k}", w, qt, (k, n))
    d = B.OpDesc(); d.op_type, d.num_input = B.OP["MatMul"], 2
    px = be.upload(x); po = be.alloc_memory(n * t * 4)
    d.input[0] = B.make_tensor(pw, qt, (k, n), None, B.NODE_CONSTANT)
    d.input[1] = B.make_tensor(px, B.FP32, (k, t))
    d.output = B.make_tensor(po, B.FP32, (n, t))
    be.submit(d); be.sync()
    got = be.download(po, (t, n), np.float32)
    be.dealloc_memory(px, x.nbytes); be.dealloc_memory(po, n * t * 4)
    rows = np.unique(np.concatenate([[0, 1, n - 2, n - 1], rng.integers(0, n, size=60)]))
    want = oracle.matmul(qt, np.ascontiguousarray(w[rows]), k, len(rows), x)
    assert close(got[:, rows], want)
    assert np.isfinite(got).all()


@pytest.mark.parametrize("qt", [quants.Q4_0, quants.Q8_0, quants.Q4_K, quants.Q6_K])
@pytest.mark.parametrize("n,k,t", [(132, 512, 1), (132, 512, 5), (200, 1024, 16), (260, 2816, 41), (1100, 512, 150), (132, 8192, 5), (64, 11008, 7), (2052, 6144, 8), (64, 8192, 9)])
def test_matmul_on_uploaded_constants_takes_the_model_kernels(be, oracle, qt, n, k, t):
    """MatMul through spyb_submit against a constant from spyb_upload_constant: K-quant constants run the K-quant mat-vec
    kernel, five columns and more run the tcgen05 GEMM against a tile copy made at first use. Either way the oracle's bits (for K-quants:
    the restatement's)."""
    rng = np.random.default_rng(n + k + t + qt)
    w = quants.quantize((rng.standard_normal((n, k)) * 0.02).astype(np.float32), qt)
    x = rng.standard_normal((t, k)).astype(np.float32)
    pw = be.upload_constant(f"const_{qt}_{n}_{k}_{t}", w, qt, (k, n))
    want = oracle.matmul(qt, w, k, n, x)
    for _ in range(2):   # the second call finds the copies the first one made
        d = B.OpDesc(); d.op_type, d.num_input = B.OP["MatMul"], 2
        px = be.upload(x); po = be.alloc_memory(n * t * 4)
        d.input[0] = B.make_tensor(pw, qt, (k, n), None, B.NODE_CONSTANT)
        d.input[1] = B.make_tensor(px, B.FP32, (k, t))
        d.output = B.make_tensor(po, B.FP32, (n, t))
        be.submit(d); be.sync()
        got = be.download(po, (t, n), np.float32)
        be.dealloc_memory(px, x.nbytes); be.dealloc_memory(po, n * t * 4)
        assert np.array_equal(bits(got), bits(want))


@pytest.mark.parametrize("qt", [quants.Q4_0, quants.Q8_0, quants.Q4_K, quants.Q6_K])
def test_first_gemm_submit_of_a_constant_reads_finished_tiles(be, oracle, qt):
    """The submit that makes a constant's tile copy and the ones right behind it, from two threads, against the oracle on a row sample: the
    GEMM reads its first weights ahead of the kernels in front of it, so the copy has to be complete before any GEMM is enqueued."""
    n, k, t = 19072, 1024, 16
    rng = np.random.default_rng(qt)
    x = rng.standard_normal((t, k)).astype(np.float32)
    rows = np.unique(np.r_[0, n - 1, rng.integers(0, n, 60)])
    w = quants.quantize((rng.standard_normal((n, k)) * 0.02).astype(np.float32), qt)
    want = oracle.matmul(qt, np.ascontiguousarray(w[rows]), k, len(rows), x)
    px = be.upload(x)
    for i in range(4):
        pw, po = be.upload_constant(f"first_{qt}_{i}", w.copy(), qt, (k, n)), [be.alloc_memory(4 * n * t) for _ in range(2)]

        def one(p):
            d = B.OpDesc(); d.op_type, d.num_input = B.OP["MatMul"], 2
            d.input[0] = B.make_tensor(pw, qt, (k, n), None, B.NODE_CONSTANT)
            d.input[1] = B.make_tensor(px, B.FP32, (k, t))
            d.output = B.make_tensor(p, B.FP32, (n, t))
            be.submit(d)

        threads = [threading.Thread(target=one, args=(p,)) for p in po]
        for th in threads:
            th.start()
        for th in threads:
            th.join()
        be.sync()
        for p in po:
            assert np.array_equal(bits(be.download(p, (t, n), np.float32)[:, rows]), bits(want))
            be.dealloc_memory(p, 4 * n * t)
    be.dealloc_memory(px, x.nbytes)


@pytest.mark.parametrize("n,t,taken", [(6, 1, False), (6, 5, False), (126, 15, False), (6, 40, False), (9470, 16, True), (9470, 15, False)])
def test_rows_that_are_no_multiple_of_four(be, oracle, n, t, taken):
    """Q4_0 constants with such row counts: refused, with a reason, whatever the number of columns, but for products large enough that they always ran
    on the GEMM."""
    rng = np.random.default_rng(n + t)
    w = quants.quantize((rng.standard_normal((n, 64)) * 0.02).astype(np.float32), quants.Q4_0)
    x = rng.standard_normal((t, 64)).astype(np.float32)
    pw, px, po = be.upload_constant(f"odd_rows_{n}_{t}", w, quants.Q4_0, (64, n)), be.upload(x), be.alloc_memory(4 * n * t)
    d = B.OpDesc(); d.op_type, d.num_input = B.OP["MatMul"], 2
    d.input[0] = B.make_tensor(pw, quants.Q4_0, (64, n), None, B.NODE_CONSTANT)
    d.input[1] = B.make_tensor(px, B.FP32, (64, t))
    d.output = B.make_tensor(po, B.FP32, (n, t))
    if taken:
        be.submit(d); be.sync()
        assert np.array_equal(bits(be.download(po, (t, n), np.float32)), bits(oracle.matmul(quants.Q4_0, w, 64, n, x)))
    else:
        with pytest.raises(B.SpybError, match="multiple of 4") as e:
            be.submit(d)
        assert e.value.status == B.UNSUPPORTED
    be.dealloc_memory(px, x.nbytes); be.dealloc_memory(po, 4 * n * t)


@pytest.mark.parametrize("qt", [quants.Q8_0, quants.Q4_K])
def test_matmul_without_room_for_the_tile_copy(oracle, qt):
    """Several columns against a constant when the device has no memory left for the copy the GEMM reads: the mat-vec kernels take the call, and the GEMM
    later calls once there is room. The same bits each time."""
    b = B.B200Backend(0, arena_bytes=1 << 24)
    n, k, t = 8192, 8192, 12
    rng = np.random.default_rng(qt)
    rows = rng.integers(0, n, 40)
    w = np.tile(quants.quantize((rng.standard_normal((64, k)) * 0.02).astype(np.float32), qt).reshape(64, -1), (n // 64, 1))
    x = rng.standard_normal((t, k)).astype(np.float32)
    want = oracle.matmul(qt, np.ascontiguousarray(w[rows]), k, len(rows), x)
    pw, px, po = b.upload_constant("tight", w.reshape(-1), qt, (k, n)), b.upload(x), b.alloc_memory(4 * n * t)
    d = B.OpDesc(); d.op_type, d.num_input = B.OP["MatMul"], 2
    d.input[0] = B.make_tensor(pw, qt, (k, n), None, B.NODE_CONSTANT)
    d.input[1] = B.make_tensor(px, B.FP32, (k, t))
    d.output = B.make_tensor(po, B.FP32, (n, t))
    hog_bytes = b.get_avail_memory_capacity() - (100 << 20)
    hog = b.alloc_memory(hog_bytes)
    with pytest.raises(B.SpybError):
        b.alloc_memory(2 * n * k)      # (the copy takes more than two bytes a weight)
    for full in (True, True, False):
        if not full and hog:
            b.dealloc_memory(hog, hog_bytes)
        b.submit(d); b.sync()
        assert np.array_equal(bits(b.download(po, (t, n), np.float32)[:, rows]), bits(want))
    b.close()


@pytest.mark.parametrize("qt", [quants.Q4_K, quants.Q6_K])
@pytest.mark.parametrize("n,k,t", [(4800, 256, 1), (4796, 1280, 3), (2, 256, 4), (300, 8448, 2), (292, 11008, 4), (9000, 768, 1)])
def test_k_quant_mat_vec_units_and_rounds(be, oracle, qt, n, k, t):
    """The K-quant mat-vec kernel on units of one, two and four row pairs, rows of 1 to 43 super-blocks (rounds of 32 that end inside a row
    and inside a unit), more units than warps and fewer, 1 to 4 columns; bit-identical to the restatement."""
    rng = np.random.default_rng(n + k + t + qt)
    w = quants.quantize((rng.standard_normal((n, k)) * 0.02).astype(np.float32), qt)
    x = rng.standard_normal((t, k)).astype(np.float32)
    pw, px, po = be.upload_constant(f"kq_units_{qt}_{n}_{k}_{t}", w, qt, (k, n)), be.upload(x), be.alloc_memory(4 * n * t)
    d = B.OpDesc()
    d.op_type, d.num_input = B.OP["MatMul"], 2
    d.input[0] = B.make_tensor(pw, qt, (k, n), None, B.NODE_CONSTANT)
    d.input[1] = B.make_tensor(px, B.FP32, (k, t))
    d.output = B.make_tensor(po, B.FP32, (n, t))
    be.submit(d); be.sync()
    got = be.download(po, (t, n), np.float32)
    assert np.array_equal(bits(got), bits(oracle.matmul(qt, w, k, n, x)))


@pytest.mark.parametrize("qt", [quants.Q4_K, quants.Q6_K])
@pytest.mark.parametrize("k", [1792, 2304, 3840])
def test_k_quant_mat_vec_of_two_columns_sums_the_end_of_a_row(be, oracle, qt, k):
    """Two columns of rows of seven, nine and fifteen super-blocks: what is left of a row behind its groups of eight, up to seven values."""
    test_k_quant_mat_vec_units_and_rounds(be, oracle, qt, 604, k, 2)


@pytest.mark.parametrize("qt", [quants.Q4_K, quants.Q6_K])
@pytest.mark.parametrize("t", [1, 2, 4, 16])
def test_k_quant_scales_beyond_the_half_range(be, oracle, qt, t):
    """Super-blocks whose f16 scale (or minimum) is infinite, as files written from very large weights hold: infinities where the restatement has
    them, NaN where it has NaN, on the mat-vec kernel and on the GEMM."""
    n, k = 64, 768
    rng = np.random.default_rng(t + qt)
    w = quants.quantize((rng.standard_normal((n, k)) * 0.02).astype(np.float32), qt)
    blocks = w.view(np.uint8).reshape(n, k // 256, -1)
    at = {quants.Q4_K: (0, 2), quants.Q6_K: (208,)}[qt]
    for row, (off, half) in enumerate([(o, h) for o in at for h in (0x7c00, 0xfc00)]):
        blocks[8 * row, 1, off:off + 2] = np.frombuffer(np.uint16(half).tobytes(), dtype=np.uint8)
    x = rng.standard_normal((t, k)).astype(np.float32)
    pw, px, po = be.upload_constant(f"inf_{qt}_{t}", w, qt, (k, n)), be.upload(x), be.alloc_memory(4 * n * t)
    d = B.OpDesc()
    d.op_type, d.num_input = B.OP["MatMul"], 2
    d.input[0] = B.make_tensor(pw, qt, (k, n), None, B.NODE_CONSTANT)
    d.input[1] = B.make_tensor(px, B.FP32, (k, t))
    d.output = B.make_tensor(po, B.FP32, (n, t))
    be.submit(d); be.sync()
    got, want = be.download(po, (t, n), np.float32), oracle.matmul(qt, w, k, n, x)
    nan = np.isnan(want)
    assert (~np.isfinite(want)).any() and np.array_equal(np.isnan(got), nan)
    assert np.array_equal(bits(got[~nan]), bits(want[~nan]))


def test_matmul_linearity_full_size(be):
    """Size-independent property at the 7B head shape: W(2x) == 2 W(x) exactly (power-of-two scaling commutes with Q8_0)."""
    rng = np.random.default_rng(5)
    n, k = 32000, 4096
    w = quants.quantize((rng.standard_normal((n, k), dtype=np.float32) * np.float32(0.02)), quants.Q4_0)
    pw = be.upload_constant("lin_head", w, quants.Q4_0, (k, n))
    x = rng.standard_normal((1, k)).astype(np.float32)
    outs = [_mm(be, pw, quants.Q4_0, n, k, xx) for xx in (x, 2 * x)]
    assert np.array_equal(bits(outs[1]), bits(2 * outs[0]))


def _mm(be, pw, qt, n, k, x):
    t = x.shape[0]
    d = B.OpDesc(); d.op_type, d.num_input = B.OP["MatMul"], 2
    px = be.upload(x); po = be.alloc_memory(n * t * 4)
    d.input[0] = B.make_tensor(pw, qt, (k, n), None, B.NODE_CONSTANT)
    d.input[1] = B.make_tensor(px, B.FP32, (k, t))
    d.output = B.make_tensor(po, B.FP32, (n, t))
    be.submit(d); be.sync()
    got = be.download(po, (t, n), np.float32)
    be.dealloc_memory(px, x.nbytes); be.dealloc_memory(po, n * t * 4)
    return got


@pytest.mark.parametrize("qt", [quants.Q4_K, quants.Q6_K])
@pytest.mark.parametrize("n,k,t", [(64, 256, 1), (132, 1024, 3), (4096, 4096, 1), (11008, 4096, 4), (4096, 11008 // 256 * 256, 16)])
def test_matmul_k_quants_within_tolerance(be, qt, n, k, t):
    """Q4_K / Q6_K: the reference only defines the block layouts (no compute), so parity is unpinned: the kernel is
    compared with decoded weights (numpy) times the f32 activations in float64, gate max-abs 2e-2 / rel 1e-2."""
    rng = np.random.default_rng(n + k + t)
    w = quants.quantize((rng.standard_normal((n, k), dtype=np.float32) * np.float32(0.02)), qt)
    x = rng.standard_normal((t, k)).astype(np.float32)
    got = _mm(be, be.upload(w), qt, n, k, x)
    want = x.astype(np.float64) @ quants.dequantize(w, qt).astype(np.float64).T
    err = float(np.abs(got - want).max())
    print(f"type {qt} {n}x{k} t={t}: max |d| = {err:.3e}, max |y| = {np.abs(want).max():.3e}")
    assert err <= 2e-2 and err <= 1e-2 * float(np.abs(want).max())


def test_matmul_unsupported_weight_type_is_reported(be):
    d = B.OpDesc(); d.op_type, d.num_input = B.OP["MatMul"], 2
    p = be.alloc_memory(144 * 4)
    d.input[0] = B.make_tensor(p, 3, (256, 4), (20, 160, 640, 640)); d.input[1] = B.make_tensor(p, B.FP32, (256, 1)); d.output = B.make_tensor(p, B.FP32, (4, 1))   # type 3 = Q4_1: no kernel
    with pytest.raises(B.SpybError) as e:
        be.submit(d)
    assert e.value.status == B.UNSUPPORTED


# ----------------------------------------------------------------------------- the small operators
def test_rmsnorm_mul_add_silu(be, oracle):
    rng = np.random.default_rng(3)
    x = rng.standard_normal((3, 4096)).astype(np.float32)
    w = rng.standard_normal(4096).astype(np.float32)
    got = run(be, "NormRMS", [(x, B.FP32, (4096, 3), None, B.NODE_DYNAMIC)], (4096, 3), eps=1e-5).reshape(3, 4096)
    assert close(got, oracle.rmsnorm(x, 1e-5), rel=5e-6)
    got = run(be, "Mul", [(x, B.FP32, (4096, 3), None, B.NODE_DYNAMIC), (w, B.FP32, (4096,), None, B.NODE_CONSTANT)], (4096, 3)).reshape(3, 4096)
    assert np.array_equal(bits(got), bits(oracle.mul_rows(x, w)))
    y = rng.standard_normal((3, 4096)).astype(np.float32)
    got = run(be, "Add", [(x, B.FP32, (4096, 3), None, B.NODE_DYNAMIC), (y, B.FP32, (4096, 3), None, B.NODE_DYNAMIC)], (4096, 3)).reshape(3, 4096)
    assert np.array_equal(bits(got), bits(x + y))
    g = (rng.standard_normal(11008) * 4).astype(np.float32)
    got = run(be, "Silu", [(g, B.FP32, (11008,), None, B.NODE_DYNAMIC)], (11008,))
    assert np.array_equal(bits(got), bits(oracle.silu(g)))   # table built with the same libm: identical bits


@pytest.mark.parametrize("n", [2300, 2304, 2308, 4096, 4100, 5120, 6144, 6148, 8192, 8196])
def test_rmsnorm_sum_keeps_its_order(be, oracle, n):
    """The running sum at the edges of its chunk sizes, bit for bit: plain rows, a few outliers, ties at most additions (small integers times a power
    of two), powers of two, zeros in front, one huge value, values of many magnitudes."""
    rng = np.random.default_rng(n)
    z = rng.standard_normal((9, n)).astype(np.float32)
    x = [z[0], z[1] * np.where(rng.random(n) < 0.02, 30, 0.3), rng.integers(0, 16, n) * 0.125, 2.0 ** rng.integers(-20, 20, n),
         np.where(np.arange(n) < n // 2, 0, z[2]), np.where(np.arange(n) == n // 3, 1e4, z[3] * 0.01), z[4] * np.exp(3 * z[5]),
         np.sqrt(1 + 2.0 ** -rng.integers(1, 24, n)), np.zeros(n), z[6] * 1e-18, z[7] * 1e17]
    x = np.array(x, dtype=np.float32)
    got = run(be, "NormRMS", [(x, B.FP32, x.shape[::-1], None, B.NODE_DYNAMIC)], x.shape[::-1], eps=1e-5).reshape(x.shape)
    assert np.array_equal(bits(got), bits(oracle.rmsnorm(x, 1e-5)))


def test_silu_golden(be):
    g = np.load(os.path.join(GOLD, "ops_reference.npz"))
    got = run(be, "Silu", [(g["silu_x"], B.FP32, (2048,), None, B.NODE_DYNAMIC)], (2048,))
    assert np.array_equal(bits(got), bits(g["silu_out"]))


def test_softmax_masked_with_host_mask(be, oracle):
    rng = np.random.default_rng(4)
    n_ctx, n_kv, heads = 64, 37, 3
    sc = (rng.standard_normal((heads, 1, n_kv)) * 3).astype(np.float32)
    mask = np.full((1, n_ctx), -np.inf, dtype=np.float32); mask[0, : n_kv - 2] = 0
    scale = float(np.float32(1.0) / np.sqrt(np.float32(128.0)))
    got = run(be, "Softmax", [(sc, B.FP32, (n_kv, 1, heads), None, B.NODE_DYNAMIC), (mask, B.INT32, (n_ctx, 1), None, B.NODE_IO)],
              (n_kv, 1, heads), scale=scale).reshape(heads, n_kv)
    for h in range(heads):
        want = oracle.softmax_masked(sc[h, 0], mask[0, :n_kv], scale)
        assert close(got[h], want, rel=2e-6)
        assert np.all(got[h][n_kv - 2:] == 0)


def test_rope_with_host_positions(be, oracle):
    rng = np.random.default_rng(6)
    x = rng.standard_normal((3, 4, 128)).astype(np.float32)
    pos = np.array([0, 17, 511], dtype=np.int32)
    got = run(be, "Rope", [(x, B.FP32, (128, 4, 3), None, B.NODE_DYNAMIC), (pos, B.INT32, (3,), None, B.NODE_IO)], (128, 4, 3), n_dim=128).reshape(3, 4, 128)
    assert np.array_equal(bits(got), bits(oracle.rope(x, pos, 10000.0)))   # cos/sin come from the host libm


def test_rope_tables_grow_and_make_room(oracle):
    """A backend whose first Rope calls have short contexts and many bases, and whose later ones need longer tables and further bases: the oracle's bits
    throughout, every call served from a kept table (the arena shrinks at a growth) and no more than eight of them kept."""
    b = B.B200Backend(0)
    rng = np.random.default_rng(8)

    def rope(base, positions, n_context=512):
        x = rng.standard_normal((len(positions), 2, 128)).astype(np.float32)
        pos = np.array(positions, dtype=np.int32)
        got = run(b, "Rope", [(x, B.FP32, (128, 2, len(pos)), None, B.NODE_DYNAMIC), (pos, B.INT32, (len(pos),), None, B.NODE_IO)], (128, 2, len(pos)),
                  n_dim=128, base=base, n_context=n_context)
        assert np.array_equal(bits(got.reshape(x.shape)), bits(oracle.rope(x, pos, base)))
        return b.get_avail_memory_capacity()

    short = rope(10000.0, [0, 511])
    assert rope(10000.0, [512, 3, 4095], 4096) <= short - (4096 - 512) * 64 * 8
    rope(10000.0, [4096, 511, 16383])
    rope(10000.0, [16384, 1])                       # beyond the longest table: a table for the call alone
    rope(10000.0, [40000])
    kept = [rope(5000.0 + 1000 * i, [i, 300]) for i in range(12)]
    assert kept[8] == kept[11]                      # eight tables of one size: each new one replaces the oldest
    rope(10000.0, [7, 2000])
    b.close()


def test_getrow_f32_and_q8_0(be, oracle):
    rng = np.random.default_rng(7)
    table = rng.standard_normal((50, 256)).astype(np.float32)
    ids = np.array([3, 49, 0, 3], dtype=np.int32)
    got = run(be, "GetRow", [(table, B.FP32, (256, 50), None, B.NODE_CONSTANT), (ids, B.INT32, (4,), None, B.NODE_IO)], (256, 4)).reshape(4, 256)
    assert np.array_equal(bits(got), bits(table[ids]))
    tq = quants.quantize(table, quants.Q8_0)
    got = run(be, "GetRow", [(tq, B.Q8_0, (256, 50), None, B.NODE_CONSTANT), (ids, B.INT32, (4,), None, B.NODE_IO)], (256, 4)).reshape(4, 256)
    assert np.array_equal(bits(got), bits(quants.dequantize(tq, quants.Q8_0)[ids]))


def test_getrow_q4_0_and_f16_tables(be):
    """Embedding tables the CPU backend cannot gather (it aborts on Q4_0 rows, backend/host/operator/view.cpp:65-77):
    rows decode to value = (nibble - 8) * d in the element order of the dot product (low nibbles = elements 0..15), F16
    rows widen exactly. A model with such a table runs end to end as well."""
    rng = np.random.default_rng(17)
    table = (rng.standard_normal((40, 256)) * 0.1).astype(np.float32)
    ids = np.array([39, 0, 7, 7, 12], dtype=np.int32)
    tq = quants.quantize(table, quants.Q4_0)
    got = run(be, "GetRow", [(tq, B.Q4_0, (256, 40), None, B.NODE_CONSTANT), (ids, B.INT32, (5,), None, B.NODE_IO)], (256, 5)).reshape(5, 256)
    assert np.array_equal(bits(got), bits(quants.dequantize(tq, quants.Q4_0).reshape(40, 256)[ids]))
    th = table.astype(np.float16)
    got = run(be, "GetRow", [(th.view(np.uint16), B.FP16, (256, 40), None, B.NODE_CONSTANT), (ids, B.INT32, (5,), None, B.NODE_IO)], (256, 5)).reshape(5, 256)
    assert np.array_equal(bits(got), bits(th.astype(np.float32)[ids]))


@pytest.mark.parametrize("qt", [quants.Q4_K, quants.Q6_K])
def test_getrow_k_quant_tables(be, qt):
    """Embedding tables in K-quant formats (stock Q4_K_M files keep token_embd that way): rows decode as (d * sc) * q - dmin * m
    (Q4_K) and q * (d * sc) (Q6_K), one f32 operation at a time - the numpy decoder's order."""
    rng = np.random.default_rng(19)
    table = (rng.standard_normal((24, 512)) * 0.1).astype(np.float32)
    ids = np.array([23, 0, 5, 5, 11], dtype=np.int32)
    tq = quants.quantize(table, qt)
    got = run(be, "GetRow", [(tq, qt, (512, 24), None, B.NODE_CONSTANT), (ids, B.INT32, (5,), None, B.NODE_IO)], (512, 5)).reshape(5, 512)
    assert np.array_equal(bits(got), bits(quants.dequantize(tq, qt).reshape(24, 512)[ids]))


def test_copy_into_strided_f16_cache_and_view(be, oracle):
    """KV append as the graph does it: View at a byte offset, Copy f32 -> f16 into a transposed destination."""
    rng = np.random.default_rng(8)
    n_ctx, d, t, past = 16, 64, 3, 5
    v = rng.standard_normal((t, d)).astype(np.float32)
    cache = np.zeros(d * n_ctx, dtype=np.uint16)
    pc = be.upload(cache)
    vd = B.OpDesc(); vd.op_type, vd.num_input = B.OP["View"], 1
    vd.input[0] = B.make_tensor(pc, B.FP16, (d * n_ctx,)); vd.output = B.make_tensor(None, B.FP16, (t, d), (2, 2 * n_ctx)); vd.view_offset = 2 * past
    be.submit(vd)
    assert vd.output.data == pc + 2 * past
    # source = V transposed view of [d, t] f32: elements (t, d), strides (d*4, 4)
    pv = be.upload(v)
    cd = B.OpDesc(); cd.op_type, cd.num_input = B.OP["Copy"], 2
    cd.input[0] = B.make_tensor(pv, B.FP32, (t, d), (4 * d, 4)); cd.input[1] = vd.output; cd.output = B.make_tensor(None, B.FP16, (t, d))
    be.submit(cd); be.sync()
    assert cd.output.data == vd.output.data
    got = be.download(pc, (d, n_ctx), np.uint16)
    want = np.zeros((d, n_ctx), dtype=np.uint16)
    want[:, past:past + t] = oracle.quantize_f16(v).reshape(t, d).T
    assert np.array_equal(got, want)


def test_matmul_f16_strided_scores(be, oracle):
    """attn_score as the graph issues it: K view [hd, n_kv, H] with strides (2, d*2, hd*2) times Q [hd, 1, H] f32."""
    rng = np.random.default_rng(9)
    hd, heads, n_kv = 128, 2, 9
    d = hd * heads
    kc = oracle.quantize_f16(rng.standard_normal(n_kv * d).astype(np.float32))
    q = rng.standard_normal((heads, 1, hd)).astype(np.float32)
    got = run(be, "MatMul", [(kc, B.FP16, (hd, n_kv, heads), (2, d * 2, hd * 2), B.NODE_CACHE), (q, B.FP32, (hd, 1, heads), None, B.NODE_DYNAMIC)],
              (n_kv, 1, heads)).reshape(heads, n_kv)
    k2 = kc.reshape(n_kv, heads, hd)
    for h in range(heads):
        qh = oracle.quantize_f16(q[h, 0])
        want = np.array([oracle.dot("f16_f16", np.ascontiguousarray(k2[j, h]), qh, hd) for j in range(n_kv)], dtype=np.float32)
        assert close(got[h], want, rel=2e-6)


def test_alloc_free_reuse_and_callback(be):
    a = be.alloc_memory(1000); b = be.alloc_memory(5000)
    assert a % 256 == 0 and b % 256 == 0 and a != b
    be.dealloc_memory(a, 1000)
    assert be.alloc_memory(900) == a
    fired = []
    x = np.ones(64, dtype=np.float32)
    d = B.OpDesc(); d.op_type, d.num_input = B.OP["Silu"], 1
    px = be.upload(x); po = be.alloc_memory(256)
    d.input[0] = B.make_tensor(px, B.FP32, (64,)); d.output = B.make_tensor(po, B.FP32, (64,))
    be.submit(d, callback=lambda: fired.append(1))
    import time
    for _ in range(200):
        if fired:
            break
        time.sleep(0.01)
    assert fired == [1]
    be.sync()
    assert be.get_max_memory_capacity() > 100 << 30 and be.get_avail_memory_capacity() > 0


def _attention_oracle(oracle, q16, k16, vt16, pos0, n_head, hd, n_ctx, n_total=0):
    """The reference attention sub-graph composed from oracle primitives, one (token, head) at a time. Every row
    spans all n_total positions of the step; the causal mask (-inf) zeroes the ones after the token itself."""
    t, d = q16.shape
    scale = float(np.float32(1.0) / np.sqrt(np.float32(hd)))
    out = np.zeros((t, d), dtype=np.float32)
    n_kv = n_total if n_total else pos0 + t
    for i in range(t):
        mask = np.where(np.arange(n_kv) <= pos0 + i, np.float32(0), np.float32(-np.inf)).astype(np.float32)
        for h in range(n_head):
            qh = np.ascontiguousarray(q16[i, h * hd:(h + 1) * hd])
            sc = np.array([oracle.dot("f16_f16", np.ascontiguousarray(k16[j, h * hd:(h + 1) * hd]), qh, hd) for j in range(n_kv)], dtype=np.float32)
            pr = oracle.quantize_f16(oracle.softmax_masked(sc, mask, scale))
            for e in range(hd):
                out[i, h * hd + e] = oracle.dot("f16_f16", np.ascontiguousarray(vt16[h * hd + e, :n_kv]), pr, n_kv)
    return out


@pytest.mark.parametrize("pos0,t,n_total", [(0, 1, 0), (0, 4, 0), (4, 4, 0), (6, 1, 0), (30, 3, 0), (31, 2, 0), (63, 2, 0), (100, 1, 0),
                                            (0, 4, 8), (4, 3, 9), (28, 4, 37), (60, 4, 70), (0, 8, 8)])
@pytest.mark.parametrize("spread", [0.5, 4.0, 30.0])
def test_fused_attention_bits(be, oracle, pos0, t, n_total, spread):
    """Fused scores / softmax / PV against the oracle on wide-range values, across the 32-element boundaries of
    both dot products (n_kv = 1 .. 101)."""
    rng = np.random.default_rng(pos0 * 7 + t + int(spread * 10))
    n_head, hd, n_ctx = 2, 128, 128
    d = n_head * hd
    wide = lambda n: (rng.standard_normal(n) * rng.choice([0.05, 1.0, spread], size=n)).astype(np.float32)
    q16 = oracle.quantize_f16(wide(t * d)).reshape(t, d)
    k16 = oracle.quantize_f16(wide(n_ctx * d)).reshape(n_ctx, d)
    vt16 = oracle.quantize_f16(wide(n_ctx * d)).reshape(d, n_ctx)
    got = be.attention(q16, k16, vt16, pos0, n_head, hd, n_ctx, n_total)
    want = _attention_oracle(oracle, q16, k16, vt16, pos0, n_head, hd, n_ctx, n_total)
    assert np.array_equal(bits(got), bits(want))


@pytest.mark.parametrize("pos0,t,n_total,n_ctx", [(255, 1, 0, 512), (256, 2, 0, 512), (300, 1, 0, 512), (511, 1, 0, 512), (700, 2, 703, 1024), (1023, 1, 0, 1024),
                                                  (0, 1, 0, 2048), (5, 3, 0, 2048), (1500, 2, 0, 2048), (3000, 3, 3010, 4096), (4094, 2, 0, 4096), (4095, 1, 0, 4096)])
def test_fused_attention_long_rows(be, oracle, pos0, t, n_total, n_ctx):
    """Rows longer than the CTA (more than 256 positions: several positions per thread, many 32-position PV steps) up to
    a full context, against the oracle. Contexts above 1024 positions take the cluster kernel, at short and at full rows."""
    rng = np.random.default_rng(pos0 + n_ctx)
    n_head, hd = 1, 128
    d = n_head * hd
    wide = lambda n: (rng.standard_normal(n) * rng.choice([0.05, 1.0, 4.0], size=n)).astype(np.float32)
    q16 = oracle.quantize_f16(wide(t * d)).reshape(t, d)
    k16 = oracle.quantize_f16(wide(n_ctx * d)).reshape(n_ctx, d)
    vt16 = oracle.quantize_f16(wide(n_ctx * d)).reshape(d, n_ctx)
    got = be.attention(q16, k16, vt16, pos0, n_head, hd, n_ctx, n_total)
    want = _attention_oracle(oracle, q16, k16, vt16, pos0, n_head, hd, n_ctx, n_total)
    assert np.array_equal(bits(got), bits(want))


@pytest.mark.parametrize("pos0,t,n_total,n_ctx", [(0, 5, 0, 64), (20, 7, 0, 132), (31, 6, 40, 60), (60, 5, 70, 128), (255, 6, 300, 516), (700, 5, 0, 1024), (1015, 5, 0, 1020)])
def test_fused_attention_of_more_ctas_than_sms(be, oracle, pos0, t, n_total, n_ctx):
    """More (head, token) pairs than the chip has SMs: the kernel of which an SM holds two CTAs, across the same boundaries."""
    rng = np.random.default_rng(pos0 + n_ctx + t)
    n_head, hd = 32, 128
    d = n_head * hd
    wide = lambda n: (rng.standard_normal(n) * rng.choice([0.05, 1.0, 4.0], size=n)).astype(np.float32)
    q16 = oracle.quantize_f16(wide(t * d)).reshape(t, d)
    k16 = oracle.quantize_f16(wide(n_ctx * d)).reshape(n_ctx, d)
    vt16 = oracle.quantize_f16(wide(n_ctx * d)).reshape(d, n_ctx)
    got = be.attention(q16, k16, vt16, pos0, n_head, hd, n_ctx, n_total)
    want = _attention_oracle(oracle, q16, k16, vt16, pos0, n_head, hd, n_ctx, n_total)
    assert np.array_equal(bits(got), bits(want))


@pytest.mark.parametrize("pos0,t,n_total", [(0, 11, 0), (250, 16, 0), (1200, 9, 1215), (31, 8, 40), (2030, 18, 2048)])
def test_attention_of_a_prompt_shares_k_and_v_rows(be, oracle, pos0, t, n_total):
    """Eight and more tokens above 1024 positions of context: tiles of eight tokens share the K rows (scores) and the V^T rows
    (PV); every token's result must still be the oracle's bits - ragged last tiles, tiles that straddle 32- and 256-position
    boundaries, rows that end at the context's end."""
    rng = np.random.default_rng(pos0 + t)
    n_head, hd, n_ctx = 2, 128, 2048
    d = n_head * hd
    wide = lambda n: (rng.standard_normal(n) * rng.choice([0.05, 1.0, 4.0], size=n)).astype(np.float32)
    q16 = oracle.quantize_f16(wide(t * d)).reshape(t, d)
    k16 = oracle.quantize_f16(wide(n_ctx * d)).reshape(n_ctx, d)
    vt16 = oracle.quantize_f16(wide(n_ctx * d)).reshape(d, n_ctx)
    got = be.attention(q16, k16, vt16, pos0, n_head, hd, n_ctx, n_total)
    want = _attention_oracle(oracle, q16, k16, vt16, pos0, n_head, hd, n_ctx, n_total)
    assert np.array_equal(bits(got), bits(want))


@pytest.mark.parametrize("pos0,t,n_total,n_ctx", [(0, 33, 0, 1028), (95, 34, 0, 1060), (896, 130, 1026, 1032), (1000, 41, 1100, 1100)])
def test_attention_of_a_prompt_across_its_tiles(be, oracle, pos0, t, n_total, n_ctx):
    """More than 32 tokens (a second group of the scores kernel), more than one chunk of 128 positions, contexts whose last K rows and
    last chunk are ragged, and masked positions behind the last token."""
    rng = np.random.default_rng(pos0 + t)
    n_head, hd = 2, 128
    d = n_head * hd
    q16 = oracle.quantize_f16(rng.standard_normal(t * d).astype(np.float32)).reshape(t, d)
    k16 = oracle.quantize_f16(rng.standard_normal(n_ctx * d).astype(np.float32)).reshape(n_ctx, d)
    vt16 = oracle.quantize_f16(rng.standard_normal(n_ctx * d).astype(np.float32)).reshape(d, n_ctx)
    got = be.attention(q16, k16, vt16, pos0, n_head, hd, n_ctx, n_total)
    want = _attention_oracle(oracle, q16, k16, vt16, pos0, n_head, hd, n_ctx, n_total)
    assert np.array_equal(bits(got), bits(want))


@pytest.mark.parametrize("t", [9, 3])
@pytest.mark.parametrize("q_off,v_off", [(2, 0), (0, 2), (0, 4), (8, 8), (16, 8)])
def test_attention_takes_q_and_v_of_any_alignment(be, oracle, t, q_off, v_off):
    """Q and V^T at addresses that only halves are aligned to: views into larger buffers, as before the tiled kernels read them in wider pieces."""
    rng = np.random.default_rng(q_off + v_off)
    n_head, n_ctx, pos0 = 1, 1032, 70
    q16 = oracle.quantize_f16(rng.standard_normal(t * 128).astype(np.float32)).reshape(t, 128)
    k16 = oracle.quantize_f16(rng.standard_normal(n_ctx * 128).astype(np.float32)).reshape(n_ctx, 128)
    vt16 = oracle.quantize_f16(rng.standard_normal(n_ctx * 128).astype(np.float32)).reshape(128, n_ctx)
    shift = lambda a, off: np.concatenate([np.zeros(off // 2, dtype=np.uint16), a.ravel()])
    pq, pk, pv, po = be.upload(shift(q16, q_off)), be.upload(k16), be.upload(shift(vt16, v_off)), be.alloc_memory(t * 128 * 4)
    be._check(be._l.spyb_attention(be.h, pq + q_off, pk, pv + v_off, po, pos0, t, pos0 + t, n_head, 128, n_ctx))
    got = be.download(po, (t, 128), np.float32)
    for p, n in ((pq, q16.nbytes + q_off), (pk, k16.nbytes), (pv, vt16.nbytes + v_off), (po, t * 128 * 4)):
        be.dealloc_memory(p, n)
    assert np.array_equal(bits(got), bits(_attention_oracle(oracle, q16, k16, vt16, pos0, n_head, 128, n_ctx, pos0 + t)))


@pytest.mark.parametrize("pos0,t,n_total,n_ctx,n_head", [(0, 1, 1, 1032, 2), (31, 1, 32, 1032, 1), (32, 1, 33, 1032, 1), (127, 1, 128, 1032, 2), (511, 1, 512, 1032, 1),
                                                         (512, 1, 513, 2048, 2), (1400, 3, 1403, 1408, 2), (4090, 1, 4091, 4096, 2), (2990, 7, 2997, 3000, 6), (700, 2, 740, 4104, 1),
                                                         (5000, 1, 5001, 16384, 1), (2500, 3, 2503, 8192, 12), (4100, 1, 4101, 28000, 1), (600, 1, 601, 31840, 1), (600, 1, 601, 31848, 1)])
def test_attention_of_a_step_over_a_long_context(be, oracle, pos0, t, n_total, n_ctx, n_head):
    """One to seven tokens in a context above 1024 positions: fewer positions than the CTAs of a head, ends on and beside the 32-position tiles and the
    512-position stages, rings of sixteen, eight and four stages that wrap, the smaller ring of many CTAs, the longest context whose ring fits and the one
    behind it, masked positions behind the last token."""
    rng = np.random.default_rng(pos0 + t)
    d = n_head * 128
    q16 = oracle.quantize_f16(rng.standard_normal(t * d).astype(np.float32)).reshape(t, d)
    k16 = oracle.quantize_f16(rng.standard_normal(n_ctx * d).astype(np.float32)).reshape(n_ctx, d)
    vt16 = oracle.quantize_f16(rng.standard_normal(n_ctx * d).astype(np.float32)).reshape(d, n_ctx)
    got = be.attention(q16, k16, vt16, pos0, n_head, 128, n_ctx, n_total)
    want = _attention_oracle(oracle, q16, k16, vt16, pos0, n_head, 128, n_ctx, n_total)
    assert np.array_equal(bits(got), bits(want))


def test_lookup_tables_identical_for_every_key(be, oracle):
    silu, ex = be.read_tables()
    want_silu, want_exp = oracle.tables()
    assert np.array_equal(bits(silu), bits(want_silu))
    assert np.array_equal(bits(ex), bits(want_exp))


# --------------------------------------------------------------------------- the mat-vec and GEMM quantizers on values that are hard to round
HARD_K = [32, 96, 1024, 4096, 4128, 6144, 8224, 11008, 13824, 14336]
HARD_KQ = [256, 4096, 4352, 6144, 8448, 12288, 13824, 14336]


def hard_values(k: int, seed: int) -> np.ndarray:
    """Blocks of ties (odd multiples of half a step), of zeros, of values so small that their f16 scale is zero (whatever the bytes are), of huge
    values, of one outlier, and of ordinary ones."""
    rng = np.random.default_rng(seed)
    x = rng.standard_normal(k).astype(np.float32).reshape(-1, 32)
    kind = np.arange(len(x)) % 7
    x[kind == 1] = 0.0
    ties = (rng.integers(-126, 126, size=(int((kind == 2).sum()), 32)) + 0.5).astype(np.float32)
    ties[:, 0] = 127.0
    x[kind == 2] = ties
    x[kind == 3] *= np.float32(1e-38)
    x[kind == 4] *= np.float32(1e5)
    x[kind == 5, 7] = 3000.0
    return x.reshape(-1)


def pick_rows(qt: int, n: int, k: int) -> np.ndarray:
    """Rows that pick one value each (a single nonzero weight)."""
    w = np.zeros((n, k), dtype=np.float32)
    w[np.arange(n), np.random.default_rng(5).integers(0, k, n) if n != k else np.arange(n)] = 1.0
    return quants.quantize(w, qt)


def constant_matmul(be, name: str, qt: int, raw: np.ndarray, n: int, x: np.ndarray, offset: int = 0) -> np.ndarray:
    """x [columns, k] times an uploaded constant; the activations lie `offset` floats behind an allocation's start."""
    cols, k = x.shape
    px = be.upload(np.concatenate([np.zeros(offset, dtype=np.float32), x.reshape(-1)]))
    pw, po = be.upload_constant(name, raw, qt, (k, n)), be.alloc_memory(4 * n * cols)
    d = B.OpDesc()
    d.op_type, d.num_input = B.OP["MatMul"], 2
    d.input[0] = B.make_tensor(pw, qt, (k, n), None, B.NODE_CONSTANT)
    d.input[1] = B.make_tensor(px + 4 * offset, B.FP32, (k, cols))
    d.output = B.make_tensor(po, B.FP32, (n, cols))
    be.submit(d)
    got = be.download(po, (cols, n), np.float32)
    be.dealloc_memory(px, 4 * (x.size + offset)); be.dealloc_memory(po, 4 * n * cols)
    return got


@pytest.mark.parametrize("qt,k", [(qt, k) for qt in (quants.Q4_0, quants.Q8_0) for k in HARD_K] + [(qt, k) for qt in (quants.Q4_K, quants.Q6_K) for k in HARD_KQ])
@pytest.mark.parametrize("cols", [1, 3, 9])
@pytest.mark.parametrize("offset", [0, 4])
def test_quantizer_on_hard_values(be, oracle, qt, cols, k, offset):
    """Each row of W picks one value of the quantized activations, so that the bytes show: the oracle's bits (K-quants: the restatement's) from the
    mat-vec kernels and the GEMM, over the remainders and numbers of values per thread of their quantizers, and for activations that lie on
    16 bytes only (offset: floats)."""
    x = np.stack([hard_values(k, 91 + c) for c in range(cols)])
    raw = pick_rows(qt, 64, k)
    got = constant_matmul(be, f"hard {qt} {k} {cols} {offset}", qt, raw, 64, x, offset)
    assert close(got, oracle.matmul(qt, raw, k, 64, x))


@pytest.mark.parametrize("qt", [quants.Q4_0, quants.Q8_0, quants.Q4_K, quants.Q6_K])
@pytest.mark.parametrize("cols", [1, 3, 9])
@pytest.mark.parametrize("k", [256, 8192])
def test_quantizer_takes_what_is_not_a_number_as_zero(be, oracle, qt, cols, k):
    """A NaN among ordinary values does not count for its block's scale and becomes the byte 0, as in the conversion to integers: the bits of the
    same activations with zeros there."""
    rng = np.random.default_rng(k + cols)
    x = rng.standard_normal((cols, k)).astype(np.float32)
    at = rng.random((cols, k)) < 0.05
    raw = quants.quantize((rng.standard_normal((64, k)) * 0.02).astype(np.float32), qt)
    want = oracle.matmul(qt, raw, k, 64, np.where(at, np.float32(0), x))
    for nan in (np.float32(np.nan), -np.float32(np.nan)):
        got = constant_matmul(be, f"nan {qt} {k} {cols}", qt, raw, 64, np.where(at, nan, x))
        assert np.array_equal(bits(got), bits(want))


@pytest.mark.parametrize("qt", [quants.Q4_0, quants.Q8_0])
@pytest.mark.parametrize("cols", [1, 3, 9])
def test_quantizer_on_infinities(be, qt, cols):
    """A block that holds an infinity has an infinite scale and bytes of 0 throughout (0 * infinity is not a number): every product is NaN, while any
    other byte would give an infinity. Each row picks one of the block's values."""
    for inf in (np.inf, -np.inf):
        x = np.random.default_rng(cols).standard_normal((cols, 32)).astype(np.float32)
        x[:, 11] = inf
        got = constant_matmul(be, f"inf {qt} {cols} {inf}", qt, pick_rows(qt, 32, 32), 32, x)
        assert np.isnan(got).all()


# --------------------------------------------------------------------------- operators beside their predecessors
@pytest.mark.parametrize("wtype,tokens", [("q4_0", 1), ("q8_0", 3), ("q4_0", 7)])
def test_operator_chain_with_and_without_programmatic_launch(wtype, tokens, monkeypatch):
    """The operators of a decoder layer, passes submitted one behind the other without a wait between them: kernels that start beside their
    predecessors (use_pdl) leave the same bits in the output and the caches as kernels that wait for them."""
    import functools

    import torch

    from perf import cases

    case = dict(kind="layer", wtype=wtype, n_head=6, n_ff=2112, tokens=tokens, past=37, n_ctx=64)
    make = B.B200Backend
    out = []
    for use_pdl in (True, False):
        monkeypatch.setattr(cases.B, "B200Backend", functools.partial(make, use_pdl=use_pdl))
        state = cases.prepare(case, 11)
        torch.cuda.synchronize()
        for _ in range(5):
            res = cases.run(state)
        state.backend.sync()
        out.append({name: t.cpu().numpy() for name, t in res.items()})
        state.backend.close()
    assert np.isfinite(out[0]["x"]).all()
    assert all(np.array_equal(out[0][name], out[1][name]) for name in out[0])
