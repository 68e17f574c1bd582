"""The CUDA-core and split-BF16 GRM builds, which a cohort takes whose 1/sd^2 spans too much for the exact integers of the
FP4 build: here a marker carried once, with no frequency bound."""
import numpy as np
import pytest

from oracle import aireml, plink
from saigegpu import GRM_BF16X3_TC, GRM_FP32_SIMT, MV_FP32_SIMT, TC_SYRK_GROUP, TC_SYRK_PAIR, synth

pytestmark = pytest.mark.gpu


def load(ctx, seed, n, m):
    """A cohort whose first marker has one copy, in its first sample; its image."""
    bed, _ = synth.synth_bed(seed, n, m, 0.01)
    raw = np.frombuffer(bed, np.uint8).copy()
    nb = (n + 3) // 4
    raw[3:3 + nb] = 0xFF
    raw[3] = 0xFE
    ctx.set_matvec_mode(MV_FP32_SIMT)
    ctx.setgeno(raw, n, m, min_maf=0.0)
    return raw


def build(ctx, precision):
    ctx.grm_build(precision)
    assert ctx.build_timing()["zbuild_ms"] > 0  # standardised genotypes were written out, as the FP4 build does not
    return ctx.grm_get()


def oracle(raw, n, m):
    return plink.setgeno(raw.tobytes(), n, m, np.arange(1, n + 1), np.ones(n, bool), 0.0, 0.15)


def bf16(x):
    u = np.asarray(x, np.float32).view(np.uint32).astype(np.uint64)
    u = (u + 0x7FFF + ((u >> 16) & 1)) & 0xFFFF0000
    return u.astype(np.uint32).view(np.float32)


def test_split_bf16_sums_four_products(gpu_ctx):
    """K against the FP64 GRM, and on the sum of all four products of 16-bit genotypes: within its FP32 accumulation
    (~2e-9 off the diagonal), a tenth of what the smallest product adds."""
    n, m = 700, 1900
    raw = load(gpu_ctx, 31, n, m)
    K = build(gpu_ctx, GRM_BF16X3_TC).astype(np.float64)
    np.testing.assert_array_equal(K, K.T)
    g = oracle(raw, n, m)
    ref = aireml.DenseGRM(g).K
    assert np.abs(K - ref).max() < 2e-5 * np.abs(ref).max()
    Z = plink.std_geno(g)
    Zh = bf16(Z)
    Zl = bf16(Z - Zh).astype(np.float64)
    Zh = Zh.astype(np.float64)
    off = ~np.eye(n, dtype=bool)
    rms = lambda a: float(np.sqrt(np.mean(a[off] ** 2)))  # noqa: E731
    assert rms(K - (Zh + Zl).T @ (Zh + Zl) / len(Z)) < 0.1 * rms(Zl.T @ Zl / len(Z))


@pytest.mark.parametrize("n,m", [(700, 1900), (600, 1300)])
def test_split_bf16_shape_variants_bit_identical(gpu_ctx, n, m):
    """Single CTAs and CTA pairs, any raster group, 6 and 5 row blocks of 128: the same K."""
    ctx = gpu_ctx
    load(ctx, 33, n, m)
    prev = ctx.tc_options()
    try:
        K = None
        for pair, group in ((0, 16), (0, 1), (1, 1), (1, 2), (1, 16)):
            ctx.set_tc_option(TC_SYRK_PAIR, pair)
            ctx.set_tc_option(TC_SYRK_GROUP, group)
            got = build(ctx, GRM_BF16X3_TC)
            K = got if K is None else K
            np.testing.assert_array_equal(got, K)
    finally:
        ctx.set_tc_options(prev)


@pytest.mark.parametrize("precision,mean,worst", [(GRM_BF16X3_TC, 5e-6, 2e-5), (GRM_FP32_SIMT, 5e-6, 2e-5)])
def test_diagonals_carry_no_accumulation_bias(gpu_ctx, precision, mean, worst):
    """The diagonal over 30,000 markers against the exact sums of z^2: a long reduction, drained (split BF16) or in one
    FP32 chain of 30,000 (2^-24 of each partial sum, 30,000^0.5 of them at random)."""
    n, m = 5000, 30000
    load(gpu_ctx, 35, n, m)
    K = build(gpu_ctx, precision)
    rel = np.diag(K).astype(np.float64) / (gpu_ctx.grm_diag() / gpu_ctx.dims()["m_qc"]) - 1.0
    assert abs(rel.mean()) < mean and np.abs(rel).max() < worst


def test_fp32_grm_at_size(gpu_ctx):
    """K of the FP32 CUDA-core build at 3,000 x 8,000, entry by entry: an FP32 chain of 8,000 terms, 2^-24 of partial sums
    that grow to at most the diagonal's (8,000^0.5 of them at random, 5 sigma)."""
    n, m = 3000, 8000
    raw = load(gpu_ctx, 36, n, m)
    K = build(gpu_ctx, GRM_FP32_SIMT)
    ref = aireml.DenseGRM(oracle(raw, n, m)).K
    np.testing.assert_array_equal(K, K.T)
    assert np.abs(K - ref).max() < 5 * 2.0 ** -24 * np.sqrt(m) * np.abs(ref).max()
