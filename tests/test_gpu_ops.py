"""Parity of every single operator, called through the C ABI, against the CPU
oracle on the same seeded inputs.  Integer, index and KV-cache results are
compared bit for bit; f32-accumulated results within a relative L2 error of
1e-3 (the stated tolerance; observed values are around 1e-6)."""
import os
import shutil
import subprocess
import sys
import textwrap
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

TOL = 1e-3      # stated tolerance for Q8 GEMV / GEMM outputs
TIGHT = 2e-5    # what f32 accumulation in another order should reach


def _dev(llm, arr):
    return llm.DeviceBuffer.from_host(arr)


def test_generator_matches_oracle_bit_for_bit(llm, oracle):
    O = oracle
    n = 100_003
    for dtype, kind, npdt, a, b in ((llm.I8, 0, np.int8, 0.0, 0.0), (llm.F32, 1, np.float32, 1e-3, 1e-2),
                                    (llm.F32, 2, np.float32, 0.0, 1.0), (llm.F16, 2, np.uint16, 0.0, 1.0),
                                    (llm.BF16, 2, np.uint16, 0.5, 0.02), (llm.I32, 3, np.int32, 0.0, 151936.0),
                                    (llm.F32, 4, np.float32, 0.0, 0.0)):     # 4: Gumbel (temperature sampling)
        buf = llm.DeviceBuffer(n * np.dtype(npdt).itemsize)
        llm.synthFill(buf, dtype, kind, 42, 5, 7, n, a, b)
        got = buf.download(npdt, (n,))
        want = O.synth_fill(dtype, kind, 42, 5, 7, n, a, b)
        assert np.array_equal(got.view(np.uint8), want.view(np.uint8)), (dtype, kind)
        buf.free()


def test_quantize_and_synth_weights_bit_exact(llm, oracle):
    O = oracle
    n, k = 37, 224
    w = O.synth_fill(O.F32, 2, 1, 2, 0, n * k, 0.0, 0.02).reshape(n, k)
    w[3, 64:96] = 0.0
    dw, dq, ds = _dev(llm, w), llm.DeviceBuffer(n * k), llm.DeviceBuffer(n * (k // 32) * 4)
    llm.q8Quantize(dw, dq, ds, n, k)
    q0, s0 = O.q8_quantize(w)
    assert np.array_equal(dq.download(np.int8, (n, k)), q0)
    assert np.array_equal(ds.download(np.uint32, (n, k // 32)), s0.view(np.uint32))
    llm.q8SynthWeights(dq, ds, n, k, 5, 9, 77, 0.02)
    q1, s1 = O.q8_synth_weights(n, k, 9, 77, 0.02, row0=5)
    assert np.array_equal(dq.download(np.int8, (n, k)), q1)
    assert np.array_equal(ds.download(np.uint32, (n, k // 32)), s1.view(np.uint32))


@pytest.mark.parametrize("n,k", [(4096, 4096), (1, 32), (7, 96), (130, 1024), (33, 9728), (1000, 5120), (300, 512),
                                 (257, 8192), (65, 16384)])
def test_q8_gemv(llm, oracle, n, k):
    O = oracle
    q = O.synth_fill(O.I8, 0, 0, 1, 0, n * k).reshape(n, k)
    s = O.synth_fill(O.F32, 1, 0, 2, 0, n * (k // 32), 1e-3, 1e-2).reshape(n, k // 32)
    x = O.synth_fill(O.F32, 2, 0, 3, 0, k, 0.0, 1.0)
    y = llm.q8GemvHost(q, s, x)
    ref = O.q8_gemv(q, s, x)
    err = rel_l2(y, ref)
    assert err < TOL and err < TIGHT, err


def test_q8_gemv_golden(llm, golden):
    y = llm.q8GemvHost(golden["gemv_q"], golden["gemv_s"], golden["gemv_x"])
    assert rel_l2(y, golden["gemv_y"]) < TIGHT


def test_q8_gemv_empty(llm):
    llm.q8Gemv(llm.DeviceBuffer(0), llm.DeviceBuffer(0), llm.DeviceBuffer(128), llm.DeviceBuffer(0), 0, 32)


def _gemm_inputs(O, m, n, k, seed=0):
    a = O.f32_to_bf16(O.synth_fill(O.F32, 2, seed, 10, 0, m * k, 0.0, 1.0).reshape(m, k))
    q = O.synth_fill(O.I8, 0, seed, 11, 0, n * k).reshape(n, k)
    s = O.synth_fill(O.F32, 1, seed, 12, 0, n * (k // 32), 1e-3, 1e-2).reshape(n, k // 32)
    return a, q, s


@pytest.mark.parametrize("m,n,k", [(64, 256, 3584), (16, 1152, 896), (1, 128, 128), (5, 70, 96), (64, 512, 1024),
                                   (33, 384, 512)])
@pytest.mark.parametrize("simt", [False, True])
def test_q8_gemm_plain(llm, oracle, m, n, k, simt):
    O = oracle
    a, q, s = _gemm_inputs(O, m, n, k)
    c = O.bf16_to_f32(llm.q8GemmHost(a, q, s, simt=simt))
    ref32 = O.q8_gemm_f32(a, O.BF16, q, s)
    ref = O.bf16_to_f32(O.q8_gemm(a, q, s))
    assert rel_l2(c, ref) < TOL
    # compared before the bf16 rounding hides it: at most a few last-place flips
    assert np.mean(c != ref) < 5e-3
    assert rel_l2(c, ref32) < 3e-3  # bf16 output rounding alone is ~1.7e-3


@pytest.mark.parametrize("m,n,k", [(64, 256, 3584), (16, 1152, 896), (3, 200, 256), (64, 5120, 1024), (40, 128, 27648),
                                   (7, 96, 64)])
def test_q8_gemm_f32_activations(llm, oracle, m, n, k):
    """f32 activations through the two-plane tensor-core path: f32-class accuracy."""
    O = oracle
    a = O.synth_fill(O.F32, 2, 3, 10, 0, m * k, 0.0, 1.0).reshape(m, k)
    a[0, :8] = [0.0, 1e-7, -3e-5, 1000.0, -65000.0, 1.0, 0.333, -2.5]   # tiny, subnormal-in-fp16 and large entries
    q = O.synth_fill(O.I8, 0, 3, 11, 0, n * k).reshape(n, k)
    s = O.synth_fill(O.F32, 1, 3, 12, 0, n * (k // 32), 1e-3, 1e-2).reshape(n, k // 32)
    before = llm.launchCounts()
    c = llm.q8GemmF32Host(a, q, s)
    after = llm.launchCounts()
    kind = "q8_gemm_tc" if k % 128 == 0 else "q8_gemm_simt"
    assert after[kind] == before[kind] + 1   # the tcgen05 kernel takes every shape with K % 128 == 0
    ref = O.q8_gemm_f32(a, O.F32, q, s)
    assert llm.kernelStatus() == 0
    assert rel_l2(c, ref) < 2e-6, rel_l2(c, ref)


@pytest.mark.parametrize("simt", [False, True])
def test_q8_gemm_epilogues(llm, oracle, golden, simt):
    O = oracle
    a, q, s, aux = golden["gemm_a"], golden["gemm_q"], golden["gemm_s"], golden["gemm_aux"]
    c1 = llm.q8GemmHost(a, q, s, epilogue=1, aux=aux, simt=simt)
    assert np.mean(c1 != O.q8_gemm(a, q, s, 1, aux)) < 0.01
    assert rel_l2(O.bf16_to_f32(c1), golden["gemm_res"]) < 3e-3
    c2 = llm.q8GemmHost(a, q, s, epilogue=2, simt=simt)
    assert c2.shape == (a.shape[0], q.shape[0] // 2)
    assert rel_l2(O.bf16_to_f32(c2), golden["gemm_swiglu"]) < 5e-3
    m, n, k = 64, 512, 1024
    a, q, s = _gemm_inputs(O, m, n, k, seed=4)
    c2 = llm.q8GemmHost(a, q, s, epilogue=2, simt=simt)
    assert np.mean(c2 != O.q8_gemm(a, q, s, 2)) < 0.01


@pytest.mark.parametrize("m,n,k", [
    (1, 128, 160),        # K a tail of one Q8 block past a whole stage: scales brought to the tile-major form
    (17, 5000, 1056),     # a last row tile of 8 rows, a tail of 32 columns
    (64, 3584, 2368),     # K splits and a tail of 64 columns
    (65, 300, 256),       # the first count past one 64-token tile
    (96, 384, 384),       # one full 96-token tile, an odd number of row tiles
    (97, 130, 992),       # a second token tile of one token, two rows in the last row tile
    (64, 55196, 256),     # pairs of row tiles first, then single ones, on the same CTAs
    (200, 20000, 128),    # several token tiles of 96, one stage
])
def test_q8_gemm_tiles_tails_and_units(llm, oracle, m, n, k):
    """Edges of the tensor-core kernel's tiles and work units, f32 and bf16, against the oracle; repeated
    calls give the same bits (the kernel's sums have a fixed order)."""
    O = oracle
    a = O.synth_fill(O.F32, 2, 6, 10, 0, m * k, 0.0, 1.0).reshape(m, k)
    q = O.synth_fill(O.I8, 0, 6, 11, 0, n * k).reshape(n, k)
    s = O.synth_fill(O.F32, 1, 6, 12, 0, n * (k // 32), 1e-3, 1e-2).reshape(n, k // 32)
    before = llm.launchCounts()["q8_gemm_tc"]
    c = llm.q8GemmF32Host(a, q, s)
    assert llm.launchCounts()["q8_gemm_tc"] == before + 1
    # f32 sums over k terms in another order: about sqrt(k) roundings of 2^-24, and planes of 22 bits
    assert rel_l2(c, O.q8_gemm_f32(a, O.F32, q, s)) < 2e-6
    for _ in range(3):
        assert np.array_equal(llm.q8GemmF32Host(a, q, s), c)
    ab = O.f32_to_bf16(a)
    got, want = O.bf16_to_f32(llm.q8GemmHost(ab, q, s)), O.q8_gemm_f32(ab, O.BF16, q, s)
    assert rel_l2(got, want) < 3e-3     # bf16 results: half a last place is 2^-9 of the value
    assert llm.kernelStatus() == 0


# m, n, k and the tokens of the unit that it is for
WIDE_UNITS = [
    (128, 18944, 128, 128),    # one full tile of 128 tokens, one stage
    (129, 37000, 160, 192),    # a tile of 192 that is mostly full, a K tail of one Q8 block, a last row tile of 8 rows
    (192, 18946, 384, 0),      # two rows in the last row tile, which make pairs of 64 tokens the cheaper form
    (193, 37888, 288, 128),    # a second tile of one token, several units a CTA
    (460, 19000, 1152, 128),   # tiles of 128 and a tail, more stages than any ring has slots
    (384, 18944, 1152, 192),   # two full tiles of 192, two units a CTA, more stages than any ring has slots
    (387, 18944, 1024, 192),   # a third tile of three tokens (fewer are not the GEMM's), an even number of stages
    (383, 18930, 1056, 192),   # tails of tokens, rows and K
]


@pytest.mark.parametrize("m,n,k", [shape[:3] for shape in WIDE_UNITS])
def test_q8_gemm_wide_units_give_the_same_bits(llm, oracle, m, n, k):
    """Many tokens run in larger units than 64: the order of a sum, and so its bits, are those of 64 tokens at a time."""
    O = oracle
    a = O.synth_fill(O.F32, 2, 8, 10, 0, m * k, 0.0, 1.0).reshape(m, k)
    q = O.synth_fill(O.I8, 0, 8, 11, 0, n * k).reshape(n, k)
    s = O.synth_fill(O.F32, 1, 8, 12, 0, n * (k // 32), 1e-3, 1e-2).reshape(n, k // 32)
    ab = O.f32_to_bf16(a)
    c, cb, cs = llm.q8GemmF32Host(a, q, s), llm.q8GemmHost(ab, q, s), llm.q8GemmHost(ab, q, s, epilogue=2)
    for i in range(0, m, 64):
        assert np.array_equal(c[i:i + 64], llm.q8GemmF32Host(a[i:i + 64], q, s)), i
        assert np.array_equal(cb[i:i + 64], llm.q8GemmHost(ab[i:i + 64], q, s)), i
        assert np.array_equal(cs[i:i + 64], llm.q8GemmHost(ab[i:i + 64], q, s, epilogue=2)), i
    assert llm.kernelStatus() == 0


@pytest.mark.parametrize("m,n,k", [
    (65, 130, 1536),      # the first count past the other rule, three splits of four stages
    (129, 1000, 2080),    # a K tail of one Q8 block, splits of unequal length
    (300, 520, 4096),     # several token tiles
])
def test_q8_gemm_many_tokens_in_k_splits(llm, oracle, m, n, k):
    """Few row tiles and more than 64 tokens: every epilogue behind the fold, and the same bits from call to call."""
    O = oracle
    a = O.synth_fill(O.F32, 2, 9, 10, 0, m * k, 0.0, 1.0).reshape(m, k)
    q = O.synth_fill(O.I8, 0, 9, 11, 0, n * k).reshape(n, k)
    s = O.synth_fill(O.F32, 1, 9, 12, 0, n * (k // 32), 1e-3, 1e-2).reshape(n, k // 32)
    before = llm.launchCounts()
    c = llm.q8GemmF32Host(a, q, s)
    after = llm.launchCounts()
    # the preparation, the product, and the fold that only K splits have
    assert after["q8_gemm_tc"] == before["q8_gemm_tc"] + 1 and after["elementwise"] == before["elementwise"] + 2
    assert rel_l2(c, O.q8_gemm_f32(a, O.F32, q, s)) < 2e-6   # as above: sqrt(k) roundings of 2^-24, planes of 22 bits
    assert np.array_equal(llm.q8GemmF32Host(a, q, s), c)
    ab = O.f32_to_bf16(a)
    aux = O.f32_to_bf16(O.synth_fill(O.F32, 2, 9, 13, 0, m * n, 0.0, 1.0).reshape(m, n))
    for epilogue in (0, 1, 2):
        got = llm.q8GemmHost(ab, q, s, epilogue=epilogue, aux=aux if epilogue == 1 else None)
        # one rounding to bf16 of sums in another order: last-place differences of few elements
        assert np.mean(got != O.q8_gemm(ab, q, s, epilogue, aux if epilogue == 1 else None)) < 0.01, epilogue
    assert llm.kernelStatus() == 0


def test_q8_gemm_config1_slice(llm, oracle):
    """Config 1 shapes (M=64, K=3584) on a 2048-row slice of N, both kernels."""
    O = oracle
    a, q, s = _gemm_inputs(O, 64, 2048, 3584, seed=1)
    ref = O.bf16_to_f32(O.q8_gemm(a, q, s))
    for simt in (False, True):
        c = O.bf16_to_f32(llm.q8GemmHost(a, q, s, simt=simt))
        assert rel_l2(c, ref) < TOL


def test_q8_gemm_config1_full_size(llm, oracle):
    """The FFN up-projection at its full size: M=64 tokens x K=3584 x N=18944 (Qwen-7B FFN up-proj),
    bf16 activations, bf16 output, compared with the oracle's bf16-rounded result and, before
    the rounding hides it, with the oracle's f32 sums."""
    O = oracle
    m, n, k = 64, 18944, 3584
    a, q, s = _gemm_inputs(O, m, n, k, seed=1)
    c_bits = llm.q8GemmHost(a, q, s)
    assert llm.kernelStatus() == 0
    c = O.bf16_to_f32(c_bits)
    ref_bits = O.q8_gemm(a, q, s)
    ref = O.bf16_to_f32(ref_bits)
    assert rel_l2(c, ref) < TOL
    assert np.mean(c_bits != ref_bits) < 5e-3          # only last-place bf16 flips
    assert rel_l2(c, O.q8_gemm_f32(a, O.BF16, q, s)) < 3e-3   # bf16 output rounding alone is ~1.7e-3
    # every row tile and every token took part: no row or column of the output is left at zero
    assert (np.abs(c).max(axis=0) > 0).all() and (np.abs(c).max(axis=1) > 0).all()


@pytest.mark.parametrize("n,k", [
    (1, 32), (5, 544), (149, 2080),       # less than a stage; columns and rows that end inside one
    ("warps", 128), ("warps+1", 96), (7109, 544),   # one row a warp while every SM's 24 warps suffice, then two
    (300, 16384), (301, 16416),           # x beside the larger CTA's rings, and the smaller one's
    (9, 30208), (9, 30240), ("warps+1", 30240),   # x in shared memory, and in global: one row a warp, two
])
def test_q8_gemv_edges(llm, oracle, n, k):
    O = oracle
    if isinstance(n, str):
        import torch
        n = 24 * torch.cuda.get_device_properties(0).multi_processor_count + n.endswith("+1")
    q = O.synth_fill(O.I8, 0, 5, 1, 0, n * k).reshape(n, k)
    s = O.synth_fill(O.F32, 1, 5, 2, 0, n * (k // 32), 1e-3, 1e-2).reshape(n, k // 32)
    x = O.synth_fill(O.F32, 2, 5, 3, 0, k, 0.0, 1.0)
    y = llm.q8GemvHost(q, s, x)
    w = q.astype(np.float64) * np.repeat(s.astype(np.float64), 32, axis=1)
    # f32 sums of k terms in any order: k roundings of at most 2^-24 of the sum of magnitudes
    bound = k * 2.0 ** -24 * (np.abs(w) @ np.abs(x.astype(np.float64)))
    assert (np.abs(y - w @ x.astype(np.float64)) <= bound).all()


@pytest.mark.parametrize("n,k", [
    (2, 128), (301, 384),                     # one pair of rows; less than a stage a row, an odd number of rows
    ("warps", 640), ("warps+2", 640),         # one row a warp while every SM's 24 warps suffice, then two
    (66, 8192), (66, 8320), (66, 14848),      # two vectors beside the larger CTA's rings, and the smaller one's
    (66, 14976), (66, 30208), (66, 30336),    # one vector still, two in the GEMM; one too
    (8192, 6144), (8194, 6144),               # the most weights of two vectors
])
@pytest.mark.parametrize("m", [1, 2])
def test_q8_gemm_of_one_or_two_tokens(llm, oracle, m, n, k):
    """The GEMV kernel's form of the GEMM operators: every epilogue, f32 and bf16."""
    O = oracle
    if isinstance(n, str):
        import torch
        n = 24 * torch.cuda.get_device_properties(0).multi_processor_count + (2 if n.endswith("+2") else 0)
    a = O.synth_fill(O.F32, 2, 7, 10, 0, m * k, 0.0, 1.0).reshape(m, k)
    q = O.synth_fill(O.I8, 0, 7, 11, 0, n * k).reshape(n, k)
    s = O.synth_fill(O.F32, 1, 7, 12, 0, n * (k // 32), 1e-3, 1e-2).reshape(n, k // 32)
    before = llm.launchCounts()["q8_gemv"]
    c = llm.q8GemmF32Host(a, q, s)
    takes = k <= 30208 if m == 1 else k <= 14848 and n * k <= 48 << 20
    assert llm.launchCounts()["q8_gemv"] == before + takes
    w = q.astype(np.float64) * np.repeat(s.astype(np.float64), 32, axis=1)
    # f32 sums of k terms in any order: k roundings of at most 2^-24 of the sum of magnitudes, and 22-bit planes in the GEMM
    bound = (k + 8) * 2.0 ** -24 * (np.abs(a.astype(np.float64)) @ np.abs(w.T))
    assert (np.abs(c - a.astype(np.float64) @ w.T) <= bound).all()
    ab = O.f32_to_bf16(a)
    aux = O.f32_to_bf16(O.synth_fill(O.F32, 2, 7, 13, 0, m * n, 0.0, 1.0).reshape(m, n))
    for epilogue in (0, 1, 2) if n % 2 == 0 else (0, 1):
        got = O.bf16_to_f32(llm.q8GemmHost(ab, q, s, epilogue=epilogue, aux=aux if epilogue == 1 else None))
        want = O.bf16_to_f32(O.q8_gemm(ab, q, s, epilogue, aux if epilogue == 1 else None))
        # two f32 sums of k terms, each off by at most k roundings of the sum of magnitudes, then rounded to bf16 (2^-8 of the value
        # where they straddle); SwiGLU passes an error on times at most 1.1 (its slope) and the other factor
        e = 2 * (k + 8) * 2.0 ** -24 * (np.abs(O.bf16_to_f32(ab).astype(np.float64)) @ np.abs(w.T))
        if epilogue == 2:
            exact = np.abs(O.bf16_to_f32(ab).astype(np.float64) @ w.T)
            e = 1.1 * (e[:, ::2] * exact[:, 1::2] + e[:, 1::2] * exact[:, ::2] + e[:, ::2] * e[:, 1::2])
        assert (np.abs(got - want) <= 2.0 ** -8 * np.abs(want) + e).all() and np.mean(got != want) < 0.02, epilogue
    assert llm.kernelStatus() == 0


@pytest.mark.parametrize("m", [1, 2, 3, 200])   # the GEMV's token counts, and the GEMM's without and with K splits
@pytest.mark.parametrize("n,k", [(2048, 2048), (3072, 1024)])   # results of the activations' size, and of a larger one
def test_q8_gemm_results_over_the_activations(llm, oracle, m, n, k):
    """A product into the buffer that its activations are in, with the residual there too where it fits: what only kernels that
    have read all activations before the first result is written can give."""
    O = oracle
    a = O.synth_fill(O.F32, 2, 17, 10, 0, m * n, 0.0, 1.0)   # the product's are the first m * k
    q = O.synth_fill(O.I8, 0, 17, 11, 0, n * k).reshape(n, k)
    s = O.synth_fill(O.F32, 1, 17, 12, 0, n * (k // 32), 1e-3, 1e-2).reshape(n, k // 32)
    w = q.astype(np.float64) * np.repeat(s.astype(np.float64), 32, axis=1)
    dq, ds, db = _dev(llm, q), _dev(llm, s), _dev(llm, a)
    gemv = llm.launchCounts()["q8_gemv"]
    llm.q8GemmF32(db, dq, ds, db, m, n, k)
    x = a[:m * k].reshape(m, k).astype(np.float64)
    # f32 sums of k terms in any order: k roundings of at most 2^-24 of the sum of magnitudes, and 22-bit planes
    bound = (k + 8) * 2.0 ** -24 * (np.abs(x) @ np.abs(w.T))
    assert (np.abs(db.download(np.float32, (m, n)) - x @ w.T) <= bound).all()
    for epilogue in (0, 1, 2):
        ab = O.f32_to_bf16(a)
        db = _dev(llm, ab)
        aux = ab.reshape(m, n) if epilogue == 1 else None
        llm.q8Gemm(db, dq, ds, db, m, n, k, epilogue, db if epilogue == 1 else None)
        got = db.download(np.uint16, (m, n // 2 if epilogue == 2 else n))
        # one rounding to bf16 of sums in another order: last-place differences of few elements
        assert np.mean(got != O.q8_gemm(ab[:m * k].reshape(m, k), q, s, epilogue, aux)) < 0.01, epilogue
    assert llm.launchCounts()["q8_gemv"] == gemv   # its CTAs read activations while others write
    assert llm.kernelStatus() == 0


@pytest.mark.parametrize("m,n,k", [(96, 19000, 256), (97, 19001, 256), (193, 19004, 160), (100, 200, 128)])
def test_q8_gemm_residual_of_several_token_tiles(llm, oracle, m, n, k):
    """Past one token tile the residual is added by a kernel of its own: ends of its vectors, and of the rule."""
    O = oracle
    a, q, s = _gemm_inputs(O, m, n, k, seed=6)
    aux = O.f32_to_bf16(O.synth_fill(O.F32, 2, 6, 13, 0, m * n, 0.0, 1.0).reshape(m, n))
    c = llm.q8GemmHost(a, q, s, epilogue=1, aux=aux)
    ref = O.q8_gemm(a, q, s, 1, aux)
    assert llm.kernelStatus() == 0
    # f32 sums of k terms in another order, then one rounding to bf16: last-place differences of few elements
    assert np.mean(c != ref) < 0.01
    assert rel_l2(O.bf16_to_f32(c), O.bf16_to_f32(ref)) < 1e-3


@pytest.mark.parametrize("m,n,k", [(1, 128, 160), (17, 300, 1056), (64, 3584, 2368), (100, 19000, 160)])   # K splits and none
def test_q8_gemm_activations_that_fp16_planes_do_not_hold(llm, oracle, m, n, k):
    """K that is no multiple of 128: magnitudes past fp16's range, tiny ones and NaN give what f32 arithmetic gives, for
    every epilogue, a residual in place among them, whatever the calls before and after had."""
    O = oracle
    a = O.synth_fill(O.F32, 2, 6, 10, 0, m * k, 0.0, 1.0).reshape(m, k)
    q = O.synth_fill(O.I8, 0, 6, 11, 0, n * k).reshape(n, k)
    s = O.synth_fill(O.F32, 1, 6, 12, 0, n * (k // 32), 1e-3, 1e-2).reshape(n, k // 32)
    aux = O.f32_to_bf16(O.synth_fill(O.F32, 2, 6, 13, 0, m * n, 0.0, 1.0).reshape(m, n))
    plain = llm.q8GemmF32Host(a, q, s)
    large, tiny, nan = a.copy(), a * np.float32(1e-7), a.copy()
    large[m - 1, k - 1] = 3e5
    nan[m // 2, 5] = np.nan
    for x in (large, tiny, nan):
        rows = np.isfinite(x).all(axis=1)
        got = llm.q8GemmF32Host(x, q, s)
        want = O.q8_gemm_f32(np.where(np.isnan(x), np.float32(0), x), O.F32, q, s)
        for r in np.flatnonzero(rows):
            # f32 sums over k terms in another order: about sqrt(k) roundings of 2^-24
            assert rel_l2(got[r], want[r]) < 2e-6
        assert np.isnan(got[~rows]).all()
        assert np.array_equal(llm.q8GemmF32Host(a, q, s), plain)
        xb = O.f32_to_bf16(x)
        for epi in (0, 1, 2):
            got = O.bf16_to_f32(llm.q8GemmHost(xb, q, s, epilogue=epi, aux=aux if epi == 1 else None))
            want = O.bf16_to_f32(llm.q8GemmHost(xb, q, s, epilogue=epi, aux=aux if epi == 1 else None, simt=True))
            for r in np.flatnonzero(rows):
                assert rel_l2(got[r], want[r]) < 3e-3   # bf16 results: half a last place is 2^-9 of the value
            assert np.isnan(got[~rows]).all()
        da, dq, ds, dc = (_dev(llm, v) for v in (xb, q, s, aux))
        llm.q8Gemm(da, dq, ds, dc, m, n, k, 1, dc)
        got = O.bf16_to_f32(dc.download(np.uint16, (m, n)))
        want = O.bf16_to_f32(llm.q8GemmHost(xb, q, s, epilogue=1, aux=aux, simt=True))
        for r in np.flatnonzero(rows):
            assert rel_l2(got[r], want[r]) < 3e-3
        assert np.isnan(got[~rows]).all()
    assert llm.kernelStatus() == 0


def _in_a_process_of_its_own(code):
    """Runs `code` after the imports it needs in a fresh process, whose library scratch is empty."""
    here = os.path.dirname(os.path.abspath(__file__))
    head = "import sys; sys.path[:0] = [%r, %r]\nimport numpy as np\nfrom logicaffeine_b200 import llm\n" % (here, os.path.dirname(here))
    r = subprocess.run([sys.executable, "-c", head + textwrap.dedent(code)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]


def test_q8_gemm_of_one_token_as_the_first_call_in_a_capture(llm):
    """The GEMV form allocates nothing, so a process's first product can be inside a capture; the status word that it looks at
    exists once a kernel that can give up has run."""
    _in_a_process_of_its_own("""
        import torch
        n, k = 300, 512
        a, q, s, c, want = (llm.DeviceBuffer(b) for b in (k * 4, n * k, n * (k // 32) * 4, n * 4, n * 4))
        llm.synthFill(a, llm.F32, 2, 3, 3, 0, k)
        llm.synthFill(q, llm.I8, 0, 3, 1, 0, n * k)
        llm.synthFill(s, llm.F32, 1, 3, 2, 0, n * (k // 32), 1e-3, 1e-2)
        llm.q8Gemv(q, s, a, want, n, k)
        llm.devSync()
        st, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            llm.q8GemmF32(a, q, s, c, 1, n, k, stream=st.cuda_stream)
        g.replay()
        torch.cuda.synchronize()
        # the same kernel's sums
        assert np.array_equal(c.download(np.uint32, (n,)), want.download(np.uint32, (n,)))
        llm.q8GemmF32(a, q, s, c, 1, n, k)
        assert np.array_equal(c.download(np.uint32, (n,)), want.download(np.uint32, (n,)))
        assert llm.kernelStatus() == 0
    """)


@pytest.mark.parametrize("m,n", [(2048, 37888), (4100, 33000)])   # 310 MB of sums, and more than 2^27 of them
def test_q8_gemm_residual_keeps_little_scratch(llm, m, n):
    _in_a_process_of_its_own("""
        m, n, k = %d, %d, 128
        q, s = llm.DeviceBuffer(n * k), llm.DeviceBuffer(n * (k // 32) * 4)
        a, x, c, want = llm.DeviceBuffer(m * k * 2), llm.DeviceBuffer(m * n * 2), llm.DeviceBuffer(m * n * 2), llm.DeviceBuffer(m * n * 2)
        llm.synthFill(q, llm.I8, 0, 3, 1, 0, n * k)
        llm.synthFill(s, llm.F32, 1, 3, 2, 0, n * (k // 32), 1e-3, 1e-2)
        llm.synthFill(a, llm.BF16, 2, 3, 3, 0, m * k)
        llm.synthFill(x, llm.BF16, 2, 3, 4, 0, m * n)
        llm.q8Gemm(a, q, s, c, 1, 128, k)     # loads the kernels
        llm.q8GemmSimt(a, q, s, want, m, n, k, 1, x)
        assert llm.kernelStatus() == 0
        before, _ = llm.devMemInfo()
        llm.q8Gemm(a, q, s, c, m, n, k, 1, x)
        llm.devSync()
        after, _ = llm.devMemInfo()
        assert before - after <= 80 << 20, before - after    # 64 MB of sums, the activation plane, rounding
        got, want = c.download(np.uint16, (m, n)), want.download(np.uint16, (m, n))
        assert np.mean(got != want) < 0.01     # last places: f32 sums in another order, then one rounding to bf16
        f = lambda b: (b.astype(np.uint32) << 16).view(np.float32)
        assert np.abs(f(got) - f(want)).max() <= 2.0 ** -7 * np.abs(f(want)).max()
        assert llm.kernelStatus() == 0
    """ % (m, n))


def test_q8_gemm_of_any_k_without_room_for_scratch(llm):
    """K that is no multiple of 128 takes the tensor cores where the library has scratch for it, and goes on without: as
    the first call inside a capture, and when the memory is spent.  So does a residual of many tokens."""
    _in_a_process_of_its_own("""
        import torch
        def inputs(m, n, k):
            a, q, s, c = (llm.DeviceBuffer(b) for b in (m * k * 4, n * k, n * (k // 32) * 4, m * n * 4))
            llm.synthFill(a, llm.F32, 2, 3, 3, 0, m * k)
            llm.synthFill(q, llm.I8, 0, 3, 1, 0, n * k)
            llm.synthFill(s, llm.F32, 1, 3, 2, 0, n * (k // 32), 1e-3, 1e-2)
            return a, q, s, c
        def check(a, q, s, c, m, n, k):
            w = q.download(np.int8, (n, k)).astype(np.float64) * np.repeat(s.download(np.float32, (n, k // 32)).astype(np.float64), 32, axis=1)
            for r in {0, m // 2, m - 1}:
                x = a.download(np.float32, (k,), r * k * 4).astype(np.float64)
                y = c.download(np.float32, (n,), r * n * 4)
                # f32 sums of k terms in any order: k roundings of at most 2^-24 of the sum of magnitudes
                assert (np.abs(y - w @ x) <= k * 2.0 ** -24 * (np.abs(w) @ np.abs(x))).all()
        m, n, k = 3, 40, 160
        bufs = inputs(m, n, k)
        warm = [llm.DeviceBuffer(x) for x in (32 * 2, 32, 4, 2)]
        llm.q8GemmSimt(*warm, 1, 1, 32)
        llm.devSync()
        st, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            llm.q8GemmF32(*bufs, m, n, k, stream=st.cuda_stream)
        g.replay()
        torch.cuda.synchronize()
        check(*bufs, m, n, k)
        # with little memory left: 48 MB where 0.9 GB of planes are wanted, and 64 MB of staged sums
        m, n, k = 4096, 64, 27616
        bufs = inputs(m, n, k)
        rm, rn, rk = 2048, 37888, 128
        ra, rq, rs, rc, rx, want = (llm.DeviceBuffer(x) for x in (rm * rk * 2, rn * rk, rn * (rk // 32) * 4, rm * rn * 2, rm * rn * 2, rm * rn * 2))
        llm.synthFill(rq, llm.I8, 0, 3, 1, 0, rn * rk)
        llm.synthFill(rs, llm.F32, 1, 3, 2, 0, rn * (rk // 32), 1e-3, 1e-2)
        llm.synthFill(ra, llm.BF16, 2, 3, 3, 0, rm * rk)
        llm.synthFill(rx, llm.BF16, 2, 3, 4, 0, rm * rn)
        llm.q8GemmSimt(ra, rq, rs, want, rm, rn, rk, 1, rx)
        llm.q8Gemm(ra, rq, rs, rc, 97, 128, rk, 0)      # loads the kernel of large tiles and its plane
        assert llm.kernelStatus() == 0
        rest = llm.DeviceBuffer(llm.devMemInfo()[0] - (48 << 20))
        llm.q8GemmF32(*bufs, m, n, k)
        check(*bufs, m, n, k)
        llm.q8Gemm(ra, rq, rs, rc, rm, rn, rk, 1, rx)
        got, want = rc.download(np.uint16, (rm, rn)), want.download(np.uint16, (rm, rn))
        assert np.mean(got != want) < 0.01     # last places: f32 sums in another order, then one rounding to bf16
        assert llm.kernelStatus() == 0
    """)


def _attn_inputs(O, b, hq, hkv, d, lmax, lens, seed=0):
    kc = O.synth_fill(O.F16, 2, seed, 20, 0, b * hkv * lmax * d, 0.0, 1.0).reshape(b, hkv, lmax, d)
    vc = O.synth_fill(O.F16, 2, seed, 21, 0, b * hkv * lmax * d, 0.0, 1.0).reshape(b, hkv, lmax, d)
    q = O.synth_fill(O.F16, 2, seed, 22, 0, b * hq * d, 0.0, 1.0).reshape(b, hq, d)
    kn = O.synth_fill(O.F16, 2, seed, 23, 0, b * hkv * d, 0.0, 1.0).reshape(b, hkv, d)
    vn = O.synth_fill(O.F16, 2, seed, 24, 0, b * hkv * d, 0.0, 1.0).reshape(b, hkv, d)
    return q, kn, vn, kc, vc, np.asarray(lens, np.int32)


def test_kv_append_rope_bit_exact(llm, oracle):
    O = oracle
    b, hq, hkv, d, lmax = 5, 8, 2, 128, 96
    q, kn, vn, kc, vc, seq = _attn_inputs(O, b, hq, hkv, d, lmax, [0, 1, 50, 95, 96])
    tab = O.rope_table(lmax, d, 1e6)
    dkc, dvc, dkn, dvn, dtab, dseq = (_dev(llm, x) for x in (kc, vc, kn, vn, tab, seq))
    llm.kvAppendRope(dkc, dvc, dkn, dvn, dtab, dseq, b, hkv, d, lmax)
    O.kv_append_rope(kc, vc, kn, vn, tab, seq)
    assert np.array_equal(dkc.download(np.uint16, kc.shape), kc)
    assert np.array_equal(dvc.download(np.uint16, vc.shape), vc)
    assert np.array_equal(dseq.download(np.int32, (b,)), seq)  # the full sequence stays at l_max


@pytest.mark.parametrize("b,hq,hkv,d,lmax,lens", [
    (3, 6, 2, 64, 40, [0, 17, 39]),
    (4, 28, 4, 128, 700, [1, 64, 65, 699]),
    (2, 14, 2, 64, 384, [128, 383]),
    (2, 16, 1, 128, 300, [299, 130]),
    (1, 8, 8, 128, 129, [128]),
])
def test_gqa_decode_attn(llm, oracle, b, hq, hkv, d, lmax, lens):
    O = oracle
    q, kn, vn, kc, vc, seq = _attn_inputs(O, b, hq, hkv, d, lmax, lens)
    scale = 1.0 / np.sqrt(d)
    dq, dkc, dvc, dseq = (_dev(llm, x) for x in (q, kc, vc, seq))
    do = llm.DeviceBuffer(b * hq * d * 2)
    llm.gqaDecodeAttn(dq, dkc, dvc, dseq, do, b, hq, hkv, d, lmax, scale)
    o = O.f16_to_f32(do.download(np.uint16, (b, hq, d)))
    ref = O.f16_to_f32(O.gqa_decode_attn(q, kc, vc, seq, scale))
    assert llm.kernelStatus() == 0
    assert rel_l2(o, ref) < 1e-3
    assert np.mean(o != ref) < 0.02  # fp16 outputs: only last-place differences


@pytest.mark.parametrize("b,hq,hkv,d,lmax,lens", [
    (3, 6, 2, 64, 40, [0, 17, 39]),
    (4, 28, 4, 128, 700, [0, 63, 64, 698]),
    (3, 14, 2, 64, 200, [127, 128, 199]),
    (2, 28, 4, 128, 130, [129, 130]),   # second sequence is already full
])
def test_gqa_decode_attn_fused_kv_bit_exact(llm, oracle, b, hq, hkv, d, lmax, lens):
    O = oracle
    q, kn, vn, kc, vc, seq = _attn_inputs(O, b, hq, hkv, d, lmax, lens, seed=2)
    tab = O.rope_table(lmax, d, 1e6)
    scale = 1.0 / np.sqrt(d)
    dq, dkn, dvn, dkc, dvc, dtab, dseq = (_dev(llm, x) for x in (q, kn, vn, kc, vc, tab, seq))
    do = llm.DeviceBuffer(b * hq * d * 2)
    llm.gqaDecodeAttnFused(dq, dkn, dvn, dkc, dvc, dtab, dseq, do, b, hq, hkv, d, lmax, scale)
    o = O.f16_to_f32(do.download(np.uint16, (b, hq, d)))
    ref = O.f16_to_f32(O.gqa_decode_attn_fused(q, kn, vn, kc, vc, tab, seq, scale))
    assert llm.kernelStatus() == 0
    assert np.array_equal(dkc.download(np.uint16, kc.shape), kc)   # KV cache contents and indexing: bit exact
    assert np.array_equal(dvc.download(np.uint16, vc.shape), vc)
    assert np.array_equal(dseq.download(np.int32, (b,)), seq)
    assert rel_l2(o, ref) < 1e-3


@pytest.mark.parametrize("b,hq,hkv,d,lmax,lens", [
    (1, 2, 1, 64, 64 * 200, [64 * 200 - 2]),           # one pair in eight parts, two rows: most of them finish none
    (1, 12, 2, 128, 64 * 70, [64 * 66 - 1]),           # parts of eight tiles and of nine
    (2, 16, 1, 64, 64 * 64, [64 * 63, 0]),             # eight parts beside a pair of one tile
    (40, 32, 8, 128, 200, [(37 * i) % 199 for i in range(40)]),   # more pairs than run at once, of few tiles
    (1, 16, 1, 128, 64 * 7, [64 * 7 - 2]),             # seven parts of sixteen rows: all of the exchange's room
    (1, 15, 1, 64, 64 * 512, [64 * 512 - 2]),          # sixteen parts
    (3, 16, 1, 64, 64 * 512, [64 * 64 - 3, 64 * 64 + 5, 100]),     # just below and above where all sixteen are used
    (16, 16, 1, 64, 64 * 512, [64 * 39 + 62] + [64 * 40 + i for i in range(8)] + [9000] + [70 * i for i in range(6)]),   # ten parts, 20 rows
    (16, 7, 1, 64, 64 * 512, [64 * 52 - 2, 64 * 52, 20000] + [301 * i for i in range(13)]),                             # thirteen
    (19, 16, 16, 64, 64 * 40, [64 * 32 - 2, 64 * 32, 64 * 40 - 2] + [11 * i for i in range(16)]),    # more pairs than run at once, two parts
])
def test_gqa_decode_attn_cut_pairs_fold_the_same_every_time(llm, oracle, b, hq, hkv, d, lmax, lens):
    O = oracle
    q, kn, vn, kc, vc, seq = _attn_inputs(O, b, hq, hkv, d, lmax, lens, seed=4)
    tab = O.rope_table(lmax, d, 1e6)
    scale = 1.0 / np.sqrt(d)
    dq, dkn, dvn, dkc, dvc, dtab, dseq = (_dev(llm, x) for x in (q, kn, vn, kc, vc, tab, seq))
    do = llm.DeviceBuffer(b * hq * d * 2)
    for _ in range(2):   # the second call finds the arrival counter and the lengths as the first left them
        llm.gqaDecodeAttnFused(dq, dkn, dvn, dkc, dvc, dtab, dseq, do, b, hq, hkv, d, lmax, scale)
        o = O.f16_to_f32(do.download(np.uint16, (b, hq, d)))
        ref = O.f16_to_f32(O.gqa_decode_attn_fused(q, kn, vn, kc, vc, tab, seq, scale))
        assert llm.kernelStatus() == 0
        assert np.array_equal(dseq.download(np.int32, (b,)), seq)
        # both sides round to fp16 (2^-11 relative at most, each); the sums before it differ by some f32 roundings
        assert rel_l2(o, ref) < 1e-3
    # nothing appended: the same inputs again and again, bit for bit
    llm.gqaDecodeAttn(dq, dkc, dvc, dseq, do, b, hq, hkv, d, lmax, scale)
    first = do.download(np.uint16, (b, hq, d))
    for _ in range(20):
        llm.gqaDecodeAttn(dq, dkc, dvc, dseq, do, b, hq, hkv, d, lmax, scale)
    assert np.array_equal(do.download(np.uint16, (b, hq, d)), first)


def test_gqa_decode_attn_batches_of_several_threads(llm, oracle):
    """Each thread's calls go on working whatever batch sizes the other threads have: the kernel's shared-memory limit and
    the table of the clusters that fit belong to the process."""
    O = oracle
    hq, hkv, d, lmax = 4, 2, 64, 70
    scale = 1.0 / np.sqrt(d)
    wants, gots = {}, []
    for b in (64, 1):
        q, _, _, kc, vc, seq = _attn_inputs(O, b, hq, hkv, d, lmax, [(17 * i) % 70 for i in range(1, b + 1)], seed=9)
        wants[b] = (q, kc, vc, seq, O.f16_to_f32(O.gqa_decode_attn(q, kc, vc, seq, scale)))

    def call(b):
        q, kc, vc, seq, _ = wants[b]
        do = llm.DeviceBuffer(b * hq * d * 2)
        llm.gqaDecodeAttn(*(_dev(llm, x) for x in (q, kc, vc, seq)), do, b, hq, hkv, d, lmax, scale)
        gots.append((b, O.f16_to_f32(do.download(np.uint16, (b, hq, d)))))

    with ThreadPoolExecutor(1) as one, ThreadPoolExecutor(1) as other:
        one.submit(call, 64).result()
        other.submit(call, 1).result()
        one.submit(call, 64).result()
    assert [b for b, _ in gots] == [64, 1, 64]
    for b, o in gots:
        assert rel_l2(o, wants[b][-1]) < 1e-3   # both sides round to fp16


def test_gqa_decode_attn_config2_full_size(llm, oracle):
    """Decode attention at its full size: batch 32, 28 query / 4 KV heads, head_dim 128, 4096
    cached positions, one token appended per sequence with RoPE theta 1e6: the KV cache after the
    call is bit-equal to the oracle's, the lengths advance, the output is within tolerance."""
    O = oracle
    b, hq, hkv, d, ctx = 32, 28, 4, 128, 4096
    lmax = ctx + 1
    q, kn, vn, kc, vc, seq = _attn_inputs(O, b, hq, hkv, d, lmax, [ctx] * b, seed=5)
    tab = O.rope_table(lmax, d, 1e6)
    scale = 1.0 / np.sqrt(d)
    dq, dkn, dvn, dkc, dvc, dtab, dseq = (_dev(llm, x) for x in (q, kn, vn, kc, vc, tab, seq))
    do = llm.DeviceBuffer(b * hq * d * 2)
    llm.gqaDecodeAttnFused(dq, dkn, dvn, dkc, dvc, dtab, dseq, do, b, hq, hkv, d, lmax, scale)
    o = O.f16_to_f32(do.download(np.uint16, (b, hq, d)))
    ref = O.f16_to_f32(O.gqa_decode_attn_fused(q, kn, vn, kc, vc, tab, seq, scale))   # appends to kc, vc, seq in place
    assert llm.kernelStatus() == 0
    assert np.array_equal(dkc.download(np.uint16, kc.shape), kc)
    assert np.array_equal(dvc.download(np.uint16, vc.shape), vc)
    assert np.array_equal(dseq.download(np.int32, (b,)), seq) and (seq == ctx + 1).all()
    assert rel_l2(o, ref) < 1e-3
    for x in (dq, dkn, dvn, dkc, dvc, dtab, dseq, do):
        x.free()


def test_gqa_golden(llm, oracle, golden):
    O = oracle
    g = golden
    b, hq, d = g["att_q"].shape
    hkv, lmax = g["att_kc"].shape[1], g["att_kc"].shape[2]
    scale = float(g["att_scale"][0])
    dq, dkn, dvn, dkc, dvc, dtab, dseq = (_dev(llm, g[k]) for k in
                                          ("att_q", "att_kn", "att_vn", "att_kc", "att_vc", "rope_tab", "att_seq"))
    do = llm.DeviceBuffer(b * hq * d * 2)
    llm.gqaDecodeAttn(dq, dkc, dvc, dseq, do, b, hq, hkv, d, lmax, scale)
    assert rel_l2(O.f16_to_f32(do.download(np.uint16, (b, hq, d))), g["att_o_plain"]) < 1e-3
    llm.gqaDecodeAttnFused(dq, dkn, dvn, dkc, dvc, dtab, dseq, do, b, hq, hkv, d, lmax, scale)
    assert np.array_equal(dkc.download(np.uint16, g["att_kc"].shape), g["att_kc_after"])
    assert np.array_equal(dvc.download(np.uint16, g["att_vc"].shape), g["att_vc_after"])
    assert rel_l2(O.f16_to_f32(do.download(np.uint16, (b, hq, d))), g["att_o_fused"]) < 1e-3


def test_rmsnorm_and_swiglu(llm, oracle, golden):
    O = oracle
    x, g = golden["norm_x"], golden["norm_g"]
    dx, dg, dy = _dev(llm, x), _dev(llm, g), llm.DeviceBuffer(x.nbytes)
    llm.rmsNorm(dx, dg, dy, x.shape[0], x.shape[1], 1e-6)
    assert rel_l2(dy.download(np.float32, x.shape), O.rmsnorm(x, g, 1e-6)) < 1e-6
    a, b = golden["swi_g"], golden["swi_u"]
    da, db, dc = _dev(llm, a), _dev(llm, b), llm.DeviceBuffer(a.nbytes)
    llm.swiGlu(da, db, dc, a.size)
    assert rel_l2(dc.download(np.float32, a.shape), O.swiglu(a, b)) < 1e-6


def test_out_of_bounds_buffers_are_refused(llm):
    small = llm.DeviceBuffer(64)
    with pytest.raises(llm.LogosError) as e:
        llm.q8Gemv(small, small, small, small, 64, 64)
    assert e.value.status == 4
    small.free()
    with pytest.raises(llm.LogosError) as e:
        llm.q8Gemv(small, small, small, small, 1, 32)
    assert e.value.status in (3, 6)


def test_gemm_with_one_token_equals_gemv(llm, oracle):
    """Metamorphic: the tensor-core GEMM at M = 1 and the GEMV kernel compute the same product."""
    O = oracle
    n, k = 1000, 2048
    q = O.synth_fill(O.I8, 0, 4, 21, 0, n * k).reshape(n, k)
    s = O.synth_fill(O.F32, 1, 4, 22, 0, n * (k // 32), 1e-3, 1e-2).reshape(n, k // 32)
    x = O.synth_fill(O.F32, 2, 4, 23, 0, k, 0.0, 1.0)
    y = llm.q8GemvHost(q, s, x)
    c = llm.q8GemmF32Host(x.reshape(1, k), q, s).reshape(n)
    assert rel_l2(c, y) < 2e-6


def test_gemv_chain_in_a_dependent_launch_scope(llm, oracle):
    """Launches inside the scope may overlap their predecessor's tail; results must not change."""
    O = oracle
    n, k = 512, 4096
    q = O.synth_fill(O.I8, 0, 5, 31, 0, n * k).reshape(n, k)
    s = O.synth_fill(O.F32, 1, 5, 32, 0, n * (k // 32), 1e-3, 1e-2).reshape(n, k // 32)
    xs = [O.synth_fill(O.F32, 2, 5, 40 + i, 0, k, 0.0, 1.0) for i in range(3)]
    dq, ds = llm.DeviceBuffer.from_host(q), llm.DeviceBuffer.from_host(s)
    dx = [llm.DeviceBuffer.from_host(x) for x in xs]
    dy = [llm.DeviceBuffer(n * 4) for _ in xs]
    want = []
    for x_, y_ in zip(dx, dy):
        llm.q8Gemv(dq, ds, x_, y_, n, k)
        want.append(y_.download(np.float32, (n,)))
    prev = llm.dependentLaunchScope(True)
    try:
        for rep in range(4):
            for x_, y_ in zip(dx, dy):
                llm.q8Gemv(dq, ds, x_, y_, n, k)
    finally:
        assert llm.dependentLaunchScope(prev) is True
    llm.devSync()
    for y_, w in zip(dy, want):
        assert np.array_equal(y_.download(np.float32, (n,)), w)
    for b in [dq, ds] + dx + dy:
        b.free()


def _sequences_in_a_scope(llm, O, scoped):
    """Attention calls whose inputs the calls before them write, on one stream: what is left of each sequence."""
    b, hq, hkv, d, lmax, n, k = 6, 14, 2, 64, 700, 512, 4096
    lens = [0, 63, 64, 400, 690, 127]
    q, kn, vn, kc, vc, seq = _attn_inputs(O, b, hq, hkv, d, lmax, lens, seed=12)
    tab = O.rope_table(lmax, d, 1e6)
    scale = 1.0 / np.sqrt(d)
    dw = [_dev(llm, x) for x in (O.synth_fill(O.I8, 0, 5, 31, 0, n * k), O.synth_fill(O.F32, 1, 5, 32, 0, n * (k // 32), 1e-3, 1e-2),
                                 O.synth_fill(O.F32, 2, 5, 33, 0, k, 0.0, 1.0))]
    dy = llm.DeviceBuffer(n * 4)
    left = []
    for between in ("nothing", "gemv", "append"):
        dq, dkn, dvn, dkc, dvc, dtab, dseq = (_dev(llm, x) for x in (q, kn, vn, kc, vc, tab, seq))
        outs = [llm.DeviceBuffer(b * hq * d * 2) for _ in range(8)]
        llm.devSync()
        prev = llm.dependentLaunchScope(scoped)
        try:
            for do in outs:
                if between == "append":
                    llm.kvAppendRope(dkc, dvc, dkn, dvn, dtab, dseq, b, hkv, d, lmax)
                    llm.gqaDecodeAttn(dq, dkc, dvc, dseq, do, b, hq, hkv, d, lmax, scale)
                    continue
                llm.gqaDecodeAttnFused(dq, dkn, dvn, dkc, dvc, dtab, dseq, do, b, hq, hkv, d, lmax, scale)
                if between == "gemv":
                    llm.q8Gemv(*dw, dy, n, k)
        finally:
            llm.dependentLaunchScope(prev)
        llm.devSync()
        left.append([do.download(np.uint16, (b, hq, d)) for do in outs] + [dkc.download(np.uint16, kc.shape),
                    dvc.download(np.uint16, vc.shape), dseq.download(np.int32, (b,))])
    assert llm.kernelStatus() == 0
    return left


def test_attention_in_a_dependent_launch_scope(llm, oracle):
    """A scope only promises that nothing writes weights: lengths and cache rows that the call before an attention call
    wrote, or one two calls before it behind a kernel that lets its successor start early, are waited for."""
    plain = _sequences_in_a_scope(llm, oracle, False)
    for _ in range(3):
        for got, want in zip(_sequences_in_a_scope(llm, oracle, True), plain):
            for g, w in zip(got, want):
                assert np.array_equal(g, w)


def _freshly_written(llm, wait):
    """Products whose weights and activations the calls just before them write, on one stream; bits of all results."""
    n, k, m, rounds = 1184, 4096, 40, 6
    dq, ds, other = llm.DeviceBuffer(n * k), llm.DeviceBuffer(n * (k // 32) * 4), llm.DeviceBuffer(n * k)
    dx, dxb, scratch = llm.DeviceBuffer(m * k * 4), llm.DeviceBuffer(m * k * 2), llm.DeviceBuffer(n * 4)
    sizes = [n * 4, n * 4, m * n * 4, m * n * 2]
    outs = [[llm.DeviceBuffer(b) for b in sizes] for _ in range(rounds)]
    llm.synthFill(other, llm.I8, 0, 99, 1, 0, n * k, 0.0, 1.0)

    def then():
        if wait:
            llm.devSync()

    for i, (y0, y1, c0, c1) in enumerate(outs):
        llm.synthFill(dx, llm.F32, 2, 60 + i, 3, 0, m * k, 0.0, 1.0)
        llm.synthFill(dxb, llm.BF16, 2, 60 + i, 4, 0, m * k, 0.0, 1.0)
        llm.synthFill(ds, llm.F32, 1, 60 + i, 2, 0, n * (k // 32), 1e-3, 1e-2)
        llm.synthFill(dq, llm.I8, 0, 60 + i, 1, 0, n * k, 0.0, 1.0)
        then()
        if i % 2:                       # a call between the writer and one that reads its weights early
            llm.q8Gemv(other, ds, dx, scratch, n, k)
            prev = llm.dependentLaunchScope(True)
            llm.q8Gemv(dq, ds, dx, y0, n, k)
            llm.dependentLaunchScope(prev)
            then()
        for call in (lambda: llm.q8Gemv(dq, ds, dx, y0 if not i % 2 else y1, n, k), lambda: llm.q8GemmF32(dx, dq, ds, c0, m, n, k),
                     lambda: llm.q8Gemm(dxb, dq, ds, c1, m, n, k)):
            call()
            then()
    llm.devSync()
    return [b.download(np.uint8, (size,)) for row in outs for b, size in zip(row, sizes)][: 4 * rounds]


def test_operators_behind_calls_that_write_their_weights(llm, oracle):
    """Outside a scope a product reads nothing before the calls ahead of it have ended, and a scope's early reads behind
    such a product do not pass it."""
    want = _freshly_written(llm, True)
    for _ in range(3):
        for i, (got, w) in enumerate(zip(_freshly_written(llm, False), want)):
            if i % 4 != 1 or i // 4 % 2:   # (a second vector in odd rounds only)
                assert np.array_equal(got, w), i


def _chained(llm, wait):
    """Operators outside a scope whose inputs are the results of the calls just before them, over buffers that every round
    uses again; all bits that the last rounds leave, and those of every round's ends."""
    def sync(call, *args):
        call(*args)
        if wait:
            llm.devSync()

    def weights(i, n, k):
        q, s = llm.DeviceBuffer(n * k), llm.DeviceBuffer(n * (k // 32) * 4)
        llm.synthFill(q, llm.I8, 0, 40, 2 * i, 0, n * k, 0.0, 1.0)
        llm.synthFill(s, llm.F32, 1, 40, 2 * i + 1, 0, n * (k // 32), 1e-4, 1e-3)
        return q, s

    rounds, b, hq, hkv, d, lmax = 5, 4, 8, 2, 64, 256
    x0, y, s2, c, e = (llm.DeviceBuffer(4 * count) for count in (512, 3168, 2368 * 33, 3 * 2368, 3072))
    xb, cb, hb, gb, o1, o2 = (llm.DeviceBuffer(2 * count) for count in (65 * 1024, 65 * 2177, 69 * 1536, 69 * 1024, 2048, 2048))
    kc, vc = llm.DeviceBuffer(2 * b * hkv * lmax * d), llm.DeviceBuffer(2 * b * hkv * lmax * d)
    tab, seq = _dev(llm, llm.ropeTable(lmax, d, 1e6)), _dev(llm, np.array([3, 64, 127, 200], np.int32))
    wy, ws, w2, wd, we, wf = (weights(i, *shape) for i, shape in enumerate([(3168, 512), (2368 * 33, 512), (2368, 1056), (1024, 2368),
                                                                          (512, 512), (640, 3072)]))
    wc, wh, wg, wo, wp = (weights(10 + i, *shape) for i, shape in enumerate([(2177, 1024), (1536, 2048), (2048, 1536), (300, 1024), (700, 512)]))
    dd = llm.DeviceBuffer(4 * 3072)
    llm.synthFill(cb, llm.BF16, 2, 41, 1, 0, 65 * 2177, 0.0, 1.0)
    for i, cache in enumerate((kc, vc)):
        llm.synthFill(cache, llm.F16, 2, 41, 2 + i, 0, b * hkv * lmax * d, 0.0, 1.0)
    ends = [[llm.DeviceBuffer(n) for n in (3072 * 4, 640 * 4, 2 * 300 * 2, 4 * 700 * 2)] for _ in range(rounds)]
    llm.devSync()
    for r, (end_e, end_f, end_o, end_p) in enumerate(ends):
        llm.synthFill(x0, llm.F32, 2, 50 + r, 1, 0, 512, 0.0, 1.0)
        llm.synthFill(xb, llm.BF16, 2, 50 + r, 2, 0, 65 * 1024, 0.0, 1.0)
        # f32: vectors by the GEMV, activations and scales of a K that is no multiple of 128, then planes, then one token
        sync(llm.q8Gemv, *wy, x0, y, 3168, 512)
        sync(llm.q8Gemv, *ws, x0, s2, 2368 * 33, 512)
        sync(llm.q8GemmF32, y, w2[0], s2, c, 3, 2368, 1056)
        sync(llm.q8GemmF32, c, *wd, dd, 3, 1024, 2368)
        sync(llm.q8GemmF32, dd, *we, e, 6, 512, 512)
        sync(llm.q8GemmF32, e, *we, end_e, 6, 512, 512)
        sync(llm.q8GemmF32, end_e, *wf, end_f, 1, 640, 3072)
        # bf16: a residual in place with an odd number of columns, then products of what it left
        sync(llm.q8Gemm, xb, *wc, cb, 65, 2177, 1024, 1, cb)
        sync(llm.q8Gemm, cb, *wh, hb, 69, 1536, 2048)
        sync(llm.q8Gemm, hb, *wg, gb, 69, 2048, 1536, 2)
        # attention over those bits as f16 rows: append, attend, both in one call, and products of its result
        sync(llm.kvAppendRope, kc, vc, gb, gb, tab, seq, b, hkv, d, lmax)
        sync(llm.gqaDecodeAttn, gb, kc, vc, seq, o1, b, hq, hkv, d, lmax, 0.125)
        sync(llm.gqaDecodeAttnFused, o1, gb, o1, kc, vc, tab, seq, o2, b, hq, hkv, d, lmax, 0.125)
        sync(llm.q8Gemm, o2, *wo, end_o, 2, 300, 1024)
        sync(llm.q8Gemm, o2, *wp, end_p, 4, 700, 512)
    llm.devSync()
    assert llm.kernelStatus() == 0
    return [buf.download(np.uint8, (buf.nbytes,)) for buf in [y, s2, c, dd, e, cb, hb, gb, o1, o2, kc, vc, seq] + [x for row in ends for x in row]]


def test_operators_behind_operators_that_write_their_operands(llm, oracle):
    """An operator that starts while the one before it ends reads what that one wrote: activations, scales, residuals, cache
    rows, lengths and queries."""
    want = _chained(llm, True)
    assert all(w.any() for w in want)
    for _ in range(4):
        for i, (got, w) in enumerate(zip(_chained(llm, False), want)):
            assert np.array_equal(got, w), i


def test_products_in_a_scope_behind_one_that_writes_their_scales(llm, oracle):
    """q8_gemm of any number of tokens reads nothing before the calls ahead of it have ended, in a caller's scope too: here the
    scales are the results of a long product that was still running when the scope was opened."""
    n, k, nw, kw, m, rounds = 1184, 4096, 2368, 8192, 64, 4    # m * nw results are the n * k / 32 scales
    dq, wq, ws = llm.DeviceBuffer(n * k), llm.DeviceBuffer(nw * kw), llm.DeviceBuffer(nw * (kw // 32) * 4)
    wx, ds, dx, dxb = (llm.DeviceBuffer(b) for b in (m * kw * 4, m * nw * 4, 3 * k * 4, 3 * k * 2))
    llm.synthFill(dq, llm.I8, 0, 5, 1, 0, n * k, 0.0, 1.0)
    llm.synthFill(wq, llm.I8, 0, 5, 2, 0, nw * kw, 0.0, 1.0)
    llm.synthFill(ws, llm.F32, 1, 5, 3, 0, nw * (kw // 32), 1e-5, 1e-4)
    llm.synthFill(dx, llm.F32, 2, 5, 4, 0, 3 * k, 0.0, 1.0)
    llm.synthFill(dxb, llm.BF16, 2, 5, 4, 0, 3 * k, 0.0, 1.0)

    def results(wait):
        outs = []
        for i in range(rounds):
            for tokens in (1, 2, 3):
                c, cb = llm.DeviceBuffer(tokens * n * 4), llm.DeviceBuffer(tokens * n * 2)
                for call in (lambda: llm.q8GemmF32(dx, dq, ds, c, tokens, n, k), lambda: llm.q8Gemm(dxb, dq, ds, cb, tokens, n, k)):
                    llm.synthFill(wx, llm.F32, 2, 70 + 3 * i + tokens, 5, 0, m * kw, 0.0, 1.0)
                    llm.q8GemmF32(wx, wq, ws, ds, m, nw, kw)
                    if wait:
                        llm.devSync()
                    prev = llm.dependentLaunchScope(True)
                    call()
                    llm.dependentLaunchScope(prev)
                outs += [(c, tokens * n * 4), (cb, tokens * n * 2)]
        llm.devSync()
        return [b.download(np.uint8, (size,)) for b, size in outs]

    for got, want in zip(results(False), results(True)):
        assert np.array_equal(got, want)


def test_waits_inside_kernels_end_in_seconds(tmp_path):
    """A wait for a barrier that nothing completes returns and says so, in seconds: the limit is of time, whatever a
    poll takes."""
    here = os.path.dirname(os.path.abspath(__file__))
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "wait_limit")
    subprocess.run([nvcc, "-ccbin", "/usr/bin/g++", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3",
                    "--expt-relaxed-constexpr", "-I", os.path.join(here, "..", "logicaffeine_b200", "csrc"), "-o", exe,
                    os.path.join(here, "wait_limit.cu")], check=True, capture_output=True)
    lines = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout.split("\n")
    for form, line in enumerate(lines[:3]):
        f, ms, gave_up = line.split()
        assert int(f) == form and int(gave_up) == 1, line
        assert 1000 < float(ms) < 12000, line   # 2^32 to 2^33 cycles: 2.2 to 4.4 s at 1965 MHz


@pytest.fixture(scope="module")
def native(tmp_path_factory):
    """Runs a program beside this file that is linked with the operators, and returns its output's lines."""
    here = os.path.dirname(os.path.abspath(__file__))
    csrc = os.path.join(here, "..", "logicaffeine_b200", "csrc")
    out = str(tmp_path_factory.mktemp("native"))
    nvcc = [shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc", "-ccbin", "/usr/bin/g++", "-gencode", "arch=compute_100a,code=sm_100a",
            "-std=c++17", "-O3", "--expt-relaxed-constexpr", "-I", csrc]

    def compiled(sources):
        objects = [os.path.join(out, os.path.basename(s) + ".o") for s in sources]
        with ThreadPoolExecutor(len(sources)) as ex:
            list(ex.map(lambda so: subprocess.run(nvcc + ["-c", so[0], "-o", so[1]], check=True, capture_output=True), zip(sources, objects)))
        return objects

    operators = compiled([os.path.join(csrc, f + ".cu") for f in ("attention", "elementwise", "q8_gemm", "q8_gemm_tc", "q8_gemv", "q8_narrow",
                                                                  "runtime", "synth", "tma_host")])

    def run(program, *args):
        exe = os.path.join(out, program)
        subprocess.run(nvcc + ["-o", exe] + compiled([os.path.join(here, program + ".cu")]) + operators + ["-ldl"], check=True, capture_output=True)
        r = subprocess.run([exe] + [str(a) for a in args], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stdout
        return r.stdout.split("\n")[:-1]

    return run


def test_kernels_behind_a_failure_write_nothing(native):
    """With a code in the status word a kernel leaves its outputs, the cache and the lengths as they are; once the code has
    been read and cleared the same launch writes them all."""
    lines = native("after_failure")
    assert lines
    for line in lines:
        what, behind, after = line.rsplit(" ", 2)
        assert (behind, after) == ("0", "1"), line


def test_forms_of_products_of_many_tokens(native):
    """What the bits above are compared for does run in the wide form."""
    lines = native("gemm_forms", *[x for shape in WIDE_UNITS for x in shape[:3]])
    assert [int(line) for line in lines] == [shape[3] for shape in WIDE_UNITS]


def test_narrow_products_bit_for_bit(native):
    lines = native("narrow_products")
    assert lines and not [line for line in lines if not line.endswith(" 0")]


def test_short_division_of_swiglu_gives_the_same_bits(native):
    """All gates that it takes (0, and every finite float of at least 2^-100) against the division that rounds correctly."""
    taken, other = map(int, native("silu_gates")[0].split())
    assert taken == 2 * (0x7f800000 - 0x0d800000) + 1 and other == 0
