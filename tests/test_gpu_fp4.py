"""Exact-integer genotype GEMMs (csrc/k_fp4.cu) through the subset-exact engine's FP32 drop-ins, at the
edges of its row blocks (256), K stages (192), column tiles (16, 32, 48, 64) and of the exact range of
one accumulation (2^20 elements)."""
import numpy as np
import pytest

from oracle import aireml, plink
from saigegpu import GRM_BF16X3_TC, GRM_FP32_SIMT, MV_BF16X3_TC, MV_FP32_SIMT, MV_SUBSET_EXACT, synth

pytestmark = pytest.mark.gpu

# A product's entries carry a bounded number of FP32 roundings (the column's fixed-point quantisation
# at 2^-25 of its largest entry, T, d' T, 2p', U, the difference U - c and its scale): fewer than 64
# of 2^-24, relative to the largest entry
TOL = 64 * 2.0 ** -24


@pytest.mark.parametrize("n,m", [(33, 40), (128, 191), (129, 193), (256, 384), (385, 577), (1000, 2100)])
def test_products_match_fp64_at_tile_edges(gpu_ctx, n, m):
    """K b of one column, and two PCG iterations over 1 to 130 columns (a fixed count: the columns'
    products enter with coefficients of order one, so twice two products' bound holds)."""
    bed, _ = synth.synth_bed(500 + n, n, m, 0.03)
    ctx = gpu_ctx
    ctx.set_matvec_mode(MV_FP32_SIMT)
    ctx.setgeno(bed, n, m)
    g = plink.setgeno(bed, n, m, np.arange(1, n + 1), np.ones(n, bool), 0.01, 0.15)
    grm = aireml.DenseGRM(g)
    rng = np.random.default_rng(n)
    V = (rng.standard_normal((n, 130)) + 0.3).astype(np.float32)
    V[:, 3] = 0.0
    V[n // 2, 5] = 3000.0      # one entry far above the rest
    V[:, 7] *= np.float32(1e-12)
    V[:, 9] *= np.float32(1e12)
    w, tau = np.ones(n, np.float32), np.array([0.5, 0.5], np.float32)
    ref = aireml.pcg(grm, w, tau, V, 2, 0.0)
    ctx.set_matvec_mode(MV_SUBSET_EXACT)
    try:
        for j in (0, 5, 9):
            y, want = ctx.getCrossprodMatAndKin(V[:, j]), grm.K @ V[:, j].astype(np.float64)
            assert np.abs(y - want).max() < TOL * np.abs(want).max(), j
        first = None
        for k in (1, 15, 16, 17, 32, 33, 48, 49, 64, 65, 130):
            X = ctx.getSigma_X(w, tau, V[:, :k], 2, 0.0)
            err = np.abs(X - ref[:, :k]).max(0) / (np.abs(ref[:, :k]).max(0) + 1e-300)
            assert err.max() < 4 * TOL, (k, err.argmax(), err.max())
            first = X[:, 0] if first is None else first
            np.testing.assert_array_equal(X[:, 0], first)  # whatever the tile
            if k > 3:
                assert not X[:, 3].any()
    finally:
        ctx.set_matvec_mode(MV_FP32_SIMT)


def test_reduction_longer_than_one_exact_accumulation(gpu_ctx):
    """1,050,000 markers: the second product's K is accumulated in two segments."""
    n, m = 192, 1_050_000
    rng = np.random.default_rng(3)
    p = rng.uniform(0.05, 0.5, (m, 1))
    u = rng.random((m, n), dtype=np.float32)
    g = (u >= (1 - p) ** 2).astype(np.uint8) + (u >= 1 - p * p).astype(np.uint8)
    field = np.array([3, 2, 0], np.uint8)[g].reshape(m, n // 4, 4)
    body = field[..., 0] | (field[..., 1] << 2) | (field[..., 2] << 4) | (field[..., 3] << 6)
    bed = np.concatenate([np.array([0x6C, 0x1B, 0x01], np.uint8), body.ravel()])
    ctx = gpu_ctx
    ctx.set_matvec_mode(MV_FP32_SIMT)
    ctx.setgeno(bed, n, m)
    V = rng.standard_normal((n, 3)).astype(np.float32)
    ref, used = np.zeros((n, 3)), 0
    for i in range(0, m, 50_000):
        x = g[i:i + 50_000].astype(np.float64)
        f = x.mean(1, keepdims=True) / 2
        ok = (np.minimum(f, 1 - f) >= 0.01)[:, 0]
        z = (x - 2 * f) / np.sqrt(2 * f * (1 - f))
        ref += z[ok].T @ (z[ok] @ V)
        used += int(ok.sum())
    ref /= used
    assert used == ctx.dims()["m_qc"]
    ctx.set_matvec_mode(MV_SUBSET_EXACT)
    try:
        Y = np.column_stack([ctx.getCrossprodMatAndKin(V[:, j]) for j in range(3)])
    finally:
        ctx.set_matvec_mode(MV_FP32_SIMT)
    assert (np.abs(Y - ref).max(0) / np.abs(ref).max(0)).max() < TOL


def test_refused_memory_falls_back(gpu_ctx):
    """A budget without room for the E2M1 matrix: the drop-ins run on the BF16 products instead."""
    from saigegpu import Context
    n, m = 500, 900
    bed, _ = synth.synth_bed(9, n, m, 0.02)
    b = np.random.default_rng(1).standard_normal(n).astype(np.float32)
    out = []
    for budget in (0, None):
        with Context(0, 0 if budget == 0 else tight) as ctx:
            ctx.setgeno(bed, n, m)
            ctx.set_matvec_mode(MV_SUBSET_EXACT)
            ctx.engine_reserve(128, 1)
            ctx.grm_matmul(b)  # the BF16 products' scratch
            tight = ctx.bytes_in_use() + (1 << 16)
            out.append(ctx.getCrossprodMatAndKin(b))
            if budget is None:
                np.testing.assert_array_equal(out[1], ctx.grm_matmul(b).astype(np.float32))
    np.testing.assert_allclose(out[0], out[1], rtol=0, atol=6e-5 * np.abs(out[0]).max())


@pytest.mark.parametrize("precision,tol", [(GRM_FP32_SIMT, 4 * 2.0 ** -23), (GRM_BF16X3_TC, 2.0 ** -16)])
@pytest.mark.parametrize("n,m", [(33, 40), (64, 192), (65, 193), (256, 700), (300, 191), (641, 1500)])
def test_grm_matches_fp64_at_tile_edges(gpu_ctx, n, m, precision, tol):
    """Every entry of K against the FP64 GRM.  FP32: its own rounding (2^-24) and the oracle's, whose
    standardised genotypes are FP32 values (2^-23 of each term).  Split BF16: genotypes of 16 bits
    (2^-17 of each of a term's two factors)."""
    bed, _ = synth.synth_bed(900 + n, n, m, 0.02)
    ctx = gpu_ctx
    ctx.set_matvec_mode(MV_FP32_SIMT)
    ctx.setgeno(bed, n, m)
    ref = aireml.DenseGRM(plink.setgeno(bed, n, m, np.arange(1, n + 1), np.ones(n, bool), 0.01, 0.15)).K
    ctx.grm_build(precision)
    K = ctx.grm_get()
    assert np.abs(K - ref).max() < tol * np.abs(ref).max()
    np.testing.assert_array_equal(K, K.T)
    ctx.grm_build(precision)  # over the resident K
    np.testing.assert_array_equal(ctx.grm_get(), K)


@pytest.mark.parametrize("precision,tol", [(GRM_FP32_SIMT, 2e-6), (GRM_BF16X3_TC, 2e-5)])
def test_grm_of_a_wide_frequency_range_takes_the_other_builds(gpu_ctx, precision, tol):
    """A marker carried once among 3,000 samples: 1/sd^2 spans a factor of 1,500."""
    n, m = 3000, 400
    bed, _ = synth.synth_bed(77, n, m, 0.0)
    raw = np.frombuffer(bed, np.uint8).copy()
    nb = (n + 3) // 4
    raw[3:3 + nb] = 0xFF
    raw[3] = 0xFE  # the first sample of the first marker has one copy
    ctx = gpu_ctx
    ctx.set_matvec_mode(MV_FP32_SIMT)
    ctx.setgeno(raw, n, m, min_maf=0.0)
    g = plink.setgeno(raw.tobytes(), n, m, np.arange(1, n + 1), np.ones(n, bool), 0.0, 0.15)
    ref = aireml.DenseGRM(g).K
    ctx.grm_build(precision)
    assert np.abs(ctx.grm_get() - ref).max() < tol * np.abs(ref).max()


@pytest.mark.parametrize("mode,n,m", [(MV_BF16X3_TC, 500, 900), (MV_BF16X3_TC, 700, 1900), (MV_FP32_SIMT, 129, 300),
                                      (MV_FP32_SIMT, 1030, 700)])
def test_drop_ins_on_a_resident_grm(gpu_ctx, mode, n, m):
    """Two PCG iterations over 1 to 70 columns in the resident-GRM engines: through the genotypes (split BF16, M
    <= 2.4 N), through K (M above), and through the few-column FP32 kernel.  Split BF16 keeps 16 bits of K and
    P (2^-17 of each factor, entering twice with coefficients of order one)."""
    bed, _ = synth.synth_bed(40 + n, n, m, 0.02)
    ctx = gpu_ctx
    ctx.set_matvec_mode(MV_FP32_SIMT)
    ctx.setgeno(bed, n, m)
    grm = aireml.DenseGRM(plink.setgeno(bed, n, m, np.arange(1, n + 1), np.ones(n, bool), 0.01, 0.15))
    V = np.random.default_rng(n).standard_normal((n, 70)).astype(np.float32)
    w, tau = np.ones(n, np.float32), np.array([0.5, 0.5], np.float32)
    ref = aireml.pcg(grm, w, tau, V, 2, 0.0)
    ctx.grm_build(GRM_BF16X3_TC if mode == MV_BF16X3_TC else GRM_FP32_SIMT)
    ctx.set_matvec_mode(mode)
    try:
        first = None
        for k in (1, 2, 3, 5, 8, 9, 16, 17, 33, 70):
            X = ctx.getSigma_X(w, tau, V[:, :k], 2, 0.0)
            err = np.abs(X - ref[:, :k]).max(0) / np.abs(ref[:, :k]).max(0)
            assert err.max() < (8 * 2.0 ** -17 if mode == MV_BF16X3_TC else 4 * TOL), (k, err.argmax(), err.max())
            first = X[:, 0] if first is None else first
            np.testing.assert_array_equal(X[:, 0], first)  # whatever its neighbours
        y, want = ctx.getCrossprodMatAndKin(V[:, 0]), grm.K @ V[:, 0].astype(np.float64)
        assert np.abs(y - want).max() < (4 * 2.0 ** -17 if mode == MV_BF16X3_TC else TOL) * np.abs(want).max()
    finally:
        ctx.set_matvec_mode(MV_FP32_SIMT)


def test_refused_scratch_gives_the_matrix_back():
    """A larger engine whose FP4 scratch no longer fits the budget: the E2M1 matrix, built for the smaller one, goes too
    and the drop-ins run on the BF16 products."""
    from saigegpu import Context
    n, m = 500, 900
    bed, _ = synth.synth_bed(9, n, m, 0.02)
    b = np.random.default_rng(1).standard_normal(n).astype(np.float32)

    def run(budget):
        with Context(0, budget) as ctx:
            ctx.setgeno(bed, n, m)
            ctx.set_matvec_mode(MV_SUBSET_EXACT)
            used, out = [], []
            for cols in (128, 256):
                ctx.engine_reserve(cols, 1)
                ctx.grm_matmul(b)  # the BF16 products' scratch
                used.append(ctx.bytes_in_use())
                out.append(ctx.getCrossprodMatAndKin(b))
                used.append(ctx.bytes_in_use())
            assert not budget or np.array_equal(out[1], ctx.grm_matmul(b).astype(np.float32))
            return used, out

    used, out = run(0)
    np.testing.assert_array_equal(out[0], out[1])
    tight = run(used[3] - 16)
    assert tight[0][:2] == used[:2]
    np.testing.assert_array_equal(tight[1][0], out[0])
    matrix = 12288 * (8 * 3 + 4 * 5)  # row blocks of 128 (markers, samples) x stages of 192 (samples, markers)
    assert tight[0][2] == used[2] and tight[0][3] == used[2] - matrix


@pytest.mark.parametrize("mode", [MV_SUBSET_EXACT, MV_FP32_SIMT])
def test_drop_ins_leave_no_products_in_the_probe_cache(gpu_ctx, mode):
    """K u of a drop-in's probes, computed in its own form, does not answer an FP64 caller of the engine."""
    n, m, seed = 300, 500, 17
    bed, _ = synth.synth_bed(61, n, m, 0.02)
    ctx = gpu_ctx
    ctx.set_matvec_mode(MV_FP32_SIMT)
    ctx.setgeno(bed, n, m)
    ctx.grm_build(GRM_FP32_SIMT)
    X = np.column_stack([np.ones(n), np.random.default_rng(0).standard_normal(n)]).astype(np.float32)
    w, tau = np.ones(n, np.float32), np.array([0.6, 0.4], np.float32)
    cov = np.linalg.inv(X.T @ X).astype(np.float32)
    ctx.set_matvec_mode(mode)
    try:
        ctx.GetTrace_q(X, X, w, tau, cov, 10, seed=seed)
        assert not any(ctx.engine_probe_cached(0, seed, r) for r in range(10))
        ctx.getAIScore_q(X[:, 1], X, w, tau, X[:, 1], X, cov, 10, seed=seed)
        assert not any(ctx.engine_probe_cached(0, seed, r) for r in range(10))
    finally:
        ctx.set_matvec_mode(MV_FP32_SIMT)


@pytest.mark.parametrize("mode", [MV_SUBSET_EXACT, MV_BF16X3_TC])
@pytest.mark.parametrize("scale", [1e-34, 1e-30, 1e30])
def test_columns_of_extreme_magnitude(gpu_ctx, mode, scale):
    """A column's digits scale with it over FP32's range, so K (s b) = s K b as far as FP32 holds both."""
    n, m = 400, 700
    bed, _ = synth.synth_bed(67, n, m, 0.02)
    ctx = gpu_ctx
    ctx.set_matvec_mode(MV_FP32_SIMT)
    ctx.setgeno(bed, n, m)
    b = np.random.default_rng(5).standard_normal(n).astype(np.float32)
    if mode == MV_BF16X3_TC:
        ctx.grm_build(GRM_BF16X3_TC)
    ctx.set_matvec_mode(mode)
    try:
        y = ctx.getCrossprodMatAndKin(b).astype(np.float64)
        z = ctx.getCrossprodMatAndKin((b * np.float64(scale)).astype(np.float32)) / np.float64(scale)
    finally:
        ctx.set_matvec_mode(MV_FP32_SIMT)
    assert np.abs(z - y).max() < 2 * TOL * np.abs(y).max()


@pytest.mark.parametrize("singles", [0, 20])
def test_rare_markers_keep_the_engine_products(gpu_ctx, singles):
    """1/sd^2 of markers carried once among 6,000 samples is 3,000 times the others': the drop-ins' products stay with
    the engine's BF16 halves, which keep each entry's own bits."""
    n, m = 6000, 400
    bed, _ = synth.synth_bed(78, n, m, 0.0)
    raw = np.frombuffer(bed, np.uint8).copy()
    rows = raw[3:].reshape(m, n // 4)
    for k in range(singles):
        rows[k] = 0xFF
        rows[k, 7 * k] = 0xFE  # one copy
    b = np.random.default_rng(6).standard_normal(n).astype(np.float32)
    ctx = gpu_ctx
    ctx.set_matvec_mode(MV_FP32_SIMT)
    ctx.setgeno(raw, n, m, min_maf=0.0)
    ctx.set_matvec_mode(MV_SUBSET_EXACT)
    try:
        y, z = ctx.getCrossprodMatAndKin(b), ctx.grm_matmul(b).astype(np.float32)
    finally:
        ctx.set_matvec_mode(MV_FP32_SIMT)
    assert np.array_equal(y, z) == (singles > 0)
    assert np.abs(y - z).max() < 6e-5 * np.abs(z).max()


@pytest.mark.parametrize("m,rare", [(40, 0), (300, 1)])
def test_fp32_grm_of_few_markers_keeps_the_weights_precision(gpu_ctx, m, rare):
    """Few markers, one of them near the frequency bound: 1/sd^2 as integers of one exponent would cost the common
    markers' bits, so FP32 genotypes are multiplied.  Off-diagonal entries: 2^-24 on each of a term's two factors and of
    the chain's sums, over M terms of order one (a root of M over M), with room for the oracle's FP32 genotypes."""
    n = 2000
    bed, _ = synth.synth_bed(88, n, m, 0.0)
    raw = np.frombuffer(bed, np.uint8).copy()
    rows = raw[3:].reshape(m, n // 4)
    for k in range(rare):
        rows[k] = 0xFF
        rows[k, :6] = 0xFE  # one copy in six samples: MAF 0.0015
    ctx = gpu_ctx
    ctx.set_matvec_mode(MV_FP32_SIMT)
    ctx.setgeno(raw, n, m, min_maf=0.001)
    g = plink.setgeno(raw.tobytes(), n, m, np.arange(1, n + 1), np.ones(n, bool), 0.001, 0.15)
    ref = aireml.DenseGRM(g).K
    ctx.grm_build(GRM_FP32_SIMT)
    assert ctx.build_timing()["zbuild_ms"] > 0  # FP32 genotypes were written out
    off = ~np.eye(n, dtype=bool)
    err = (ctx.grm_get() - ref)[off]
    assert np.sqrt((err ** 2).mean()) < 16 * 2.0 ** -24 / np.sqrt(m)


def test_products_over_changed_fills(gpu_ctx):
    """setgeno with a sample list but every sample in the phenotype mask: its fills of missing calls are counted over all
    of them, and the drop-ins' subset, the listed samples, has its own at some markers (the fill-change terms)."""
    n_fam, m = 1000, 1500
    bed, _ = synth.synth_bed(93, n_fam, m, 0.1)
    sub = np.sort(np.random.default_rng(8).permutation(n_fam)[:517]).astype(np.int32) + 1
    codes = plink.decode_bed(bed, n_fam, m)  # 3: missing
    miss, allele = (codes == 3).sum(1), np.where(codes == 3, 0, codes).sum(1)
    fill_all = np.floor(2 * (allele / (2.0 * (len(sub) - miss))) + 0.5)
    c = codes[:, sub - 1]
    miss, allele = (c == 3).sum(1), np.where(c == 3, 0, c).sum(1)
    fill = np.floor(2 * (allele / (2.0 * (len(sub) - miss))) + 0.5)
    assert ((fill_all != fill) & (miss > 0)).sum() > 100  # more than one word of the fill-change bit map
    mask = np.zeros(n_fam, bool)
    mask[sub - 1] = True
    g = plink.setgeno(bed, n_fam, m, sub, mask, 0.01, 0.15)
    b = np.random.default_rng(9).standard_normal(len(sub)).astype(np.float32)
    ctx = gpu_ctx
    ctx.set_matvec_mode(MV_FP32_SIMT)
    ctx.setgeno(bed, n_fam, m, sub)
    ctx.set_matvec_mode(MV_SUBSET_EXACT)
    try:
        y, z = ctx.getCrossprodMatAndKin(b), ctx.grm_matmul(b)
    finally:
        ctx.set_matvec_mode(MV_FP32_SIMT)
    want = aireml.DenseGRM(g).K @ b.astype(np.float64)
    assert np.abs(y - want).max() < TOL * np.abs(want).max()
    assert np.abs(z - want).max() < 8 * 2.0 ** -17 * np.abs(want).max()


def test_other_slots_fill_changes_launch_nothing(gpu_ctx):
    """A drop-in beside a slot that holds a masked subset with fill changes: as many kernels as without it."""
    n, m = 600, 900
    bed, _ = synth.synth_bed(95, n, m, 0.1)
    ctx = gpu_ctx
    ctx.set_matvec_mode(MV_FP32_SIMT)
    ctx.setgeno(bed, n, m)
    b = np.random.default_rng(2).standard_normal(n).astype(np.float32)
    ctx.set_matvec_mode(MV_SUBSET_EXACT)
    try:
        ctx.engine_reserve(128, 2)
        count, out = [], []
        for masked in (False, True):
            if masked:
                ctx.engine_set_pheno(1, np.ones(n), np.array([0.6, 0.4]), np.arange(n) % 3 > 0)
            for _ in range(2):
                before = ctx.kernel_launches()
                out.append(ctx.getCrossprodMatAndKin(b))
                count.append(ctx.kernel_launches() - before)
        assert count[1] == count[3]
        for y in out:
            np.testing.assert_array_equal(y, out[0])
    finally:
        ctx.set_matvec_mode(MV_FP32_SIMT)
