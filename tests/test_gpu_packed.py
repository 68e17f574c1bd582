"""Products of few columns through two-bit genotypes (csrc/k_tc.cu, tc_packed_kernel) against the BF16 genotype matrix
on CTA pairs: the same products in the same order, so the same bits."""
import numpy as np
import pytest

from saigegpu import MV_FP32_SIMT, MV_SUBSET_EXACT, TC_DRAIN_BYTES, TC_SUBSET_PAIR, Context, SaigeGpuError, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(40, 30), (128, 128), (129, 257), (511, 1300), (1025, 640)])
def test_same_bits_as_bf16(gpu_ctx, n, m):
    """One to nine stages, fewer and more than the kernel has buffers; rows, samples and markers past a tile."""
    ctx = gpu_ctx
    bed, _ = synth.synth_bed(40 + n, n, m, 0.05)
    ctx.set_matvec_mode(MV_FP32_SIMT)
    ctx.setgeno(bed, n, m)
    mask = np.random.default_rng(n).uniform(size=n) > 0.2  # fills that differ from the cohort's
    try:
        ctx.set_matvec_mode(MV_SUBSET_EXACT)
        ctx.engine_reserve(128, 1)
        ctx.engine_set_pheno(0, np.ones(n), np.array([1.0, 0.5]), mask)
        for k in (1, 33, 64, 65, 96):
            V = np.random.default_rng(k).standard_normal((n, k)) * 10.0 ** np.linspace(-18, 18, k)
            V[~mask] = 0.0
            out = []
            for pair in (0, 1):
                ctx.set_tc_option(TC_SUBSET_PAIR, pair)
                ids = [int(i) for i in ctx.engine_submit(0, 1, V)]
                got = {}
                for _ in range(1000):
                    if len(got) == k:
                        break
                    ctx.engine_run()
                    got.update({i: r[0] for i in ids if i not in got and (r := ctx.engine_try_fetch(i)) is not None})
                out.append(np.column_stack([got[i] for i in ids]))
            np.testing.assert_array_equal(out[0], out[1])
            assert np.isfinite(out[0]).all() and np.abs(out[0]).max(0).min() > 0
    finally:
        ctx.set_tc_option(TC_SUBSET_PAIR, 2)
        ctx.set_matvec_mode(MV_FP32_SIMT)


def test_gives_way_to_other_memory():
    """Under a budget the two-bit copy is left out, or given back for what has to be allocated."""
    n, m = 500, 900
    bed, _ = synth.synth_bed(9, n, m, 0.02)
    V = np.random.default_rng(1).standard_normal((n, 8))

    def run(budget, grow=True):
        with Context(0, budget) as ctx:
            ctx.setgeno(bed, n, m)
            ctx.set_matvec_mode(MV_SUBSET_EXACT)
            ctx.engine_reserve(128, 1)
            a = ctx.grm_matmul(V)
            used1 = ctx.bytes_in_use()
            if grow:
                ctx.engine_reserve(256, 1)
            b = ctx.grm_matmul(V)
            return a, b, used1, ctx.bytes_in_use()

    a, b, used1, used2 = run(0)
    packed = 2 * 1024 * 512 // 4
    c = run(used1 - packed, False)  # left out
    d = run(used2 - packed)  # taken, then given back or left out for the larger engine
    for o in (b, c[0], d[0], d[1]):
        np.testing.assert_array_equal(o, a)
    assert c[3] == used1 - packed
    assert d[2] == used1 and d[3] == used2 - packed


def test_a_read_back_leaves_the_copies(gpu_ctx):
    """packed_geno()'s staging buffer only saves time: under a budget with no room for it the two-bit and E2M1 copies
    stay, and the rows are copied without it."""
    n, m = 500, 900
    bed, _ = synth.synth_bed(9, n, m, 0.02)
    b = np.random.default_rng(1).standard_normal(n).astype(np.float32)

    def run(budget):
        with Context(0, budget) as ctx:
            ctx.setgeno(bed, n, m)
            ctx.set_matvec_mode(MV_SUBSET_EXACT)
            ctx.engine_reserve(128, 1)
            y = ctx.grm_matmul(b), ctx.getCrossprodMatAndKin(b)
            used = ctx.bytes_in_use()
            packed = ctx.packed_geno()
            assert ctx.bytes_in_use() == used
            return used, packed, y, (ctx.grm_matmul(b), ctx.getCrossprodMatAndKin(b))

    used, packed, y, again = run(0)
    tight = run(used)
    assert tight[0] == used
    np.testing.assert_array_equal(tight[1], packed)
    for got in (again, tight[2], tight[3]):
        for a, o in zip(got, y):
            np.testing.assert_array_equal(a, o)


def test_a_request_that_cannot_fit_leaves_the_copies():
    """An allocation beyond the budget even without the copies is refused and takes nothing from them."""
    n, m = 500, 900
    bed, _ = synth.synth_bed(9, n, m, 0.02)
    b = np.random.default_rng(1).standard_normal(n).astype(np.float32)
    with Context(0, 1 << 30) as ctx:
        ctx.setgeno(bed, n, m)
        ctx.set_matvec_mode(MV_SUBSET_EXACT)
        ctx.engine_reserve(128, 1)
        y, z = ctx.grm_matmul(b), ctx.getCrossprodMatAndKin(b)
        used = ctx.bytes_in_use()
        with pytest.raises(SaigeGpuError) as ei:
            ctx.synth_bed(1, 1 << 20, 1 << 14, 0.0)  # 4 GB
        assert ei.value.code == 3  # SG_ERR_NOMEM
        assert ctx.bytes_in_use() == used
        np.testing.assert_array_equal(ctx.grm_matmul(b), y)
        np.testing.assert_array_equal(ctx.getCrossprodMatAndKin(b), z)
        assert ctx.bytes_in_use() == used


def test_copies_come_back_with_the_memory():
    """What made the copies give way is freed: the next products build them again, and give the same bits."""
    n, m, big = 500, 900, 2 << 20
    bed, _ = synth.synth_bed(9, n, m, 0.02)
    b = np.random.default_rng(1).standard_normal(n).astype(np.float32)

    def run(budget):
        with Context(0, budget) as ctx:
            ctx.setgeno(bed, n, m)
            ctx.set_matvec_mode(MV_SUBSET_EXACT)
            ctx.engine_reserve(128, 1)
            used, out = [], []
            for size in (16, big, 16):
                ctx.synth_bed(1, 4, size, 0.0)  # ``size`` bytes that have to be there
                out.append((ctx.grm_matmul(b), ctx.getCrossprodMatAndKin(b)))
                used.append(ctx.bytes_in_use())
            return used, out

    used, out = run(0)
    assert used[1] == used[0] + big - 16 and used[2] == used[0]
    tight, got = run(used[0] + 1024)
    assert tight[0] == used[0] and tight[1] < used[1] and tight[2] == used[2]
    for i in range(3):
        np.testing.assert_array_equal(got[i][0], out[0][0])
    np.testing.assert_array_equal(got[1][1], got[1][0].astype(np.float32))  # the BF16 products meanwhile
    for i in (0, 2):
        np.testing.assert_array_equal(got[i][1], out[0][1])


def test_more_row_blocks_than_a_grid_has_rows(gpu_ctx):
    """8.4 million markers of a few samples: 65,537 blocks of 128 rows."""
    n, m = 8, 65536 * 128 + 5
    ctx = gpu_ctx
    body = np.random.default_rng(2).choice(np.array([0, 2, 3], np.uint8), (m, n))
    body = body[:, 0::4] | (body[:, 1::4] << 2) | (body[:, 2::4] << 4) | (body[:, 3::4] << 6)
    ctx.set_matvec_mode(MV_FP32_SIMT)
    ctx.setgeno(np.concatenate([np.array([0x6C, 0x1B, 0x01], np.uint8), body.ravel()]), n, m)
    V = np.random.default_rng(3).standard_normal((n, 5))
    try:
        ctx.set_matvec_mode(MV_SUBSET_EXACT)
        ctx.engine_reserve(32, 1)
        out = []
        for pair in (0, 1):
            ctx.set_tc_option(TC_SUBSET_PAIR, pair)
            out.append(ctx.grm_matmul(V))
        np.testing.assert_array_equal(out[0], out[1])
        assert np.abs(out[0]).max(0).min() > 0
    finally:
        ctx.set_tc_option(TC_SUBSET_PAIR, 2)
        ctx.set_matvec_mode(MV_FP32_SIMT)
        bed, _ = synth.synth_bed(9, 64, 90, 0.02)
        ctx.setgeno(bed, 64, 90)  # the 4 GB of genotypes leave the shared context


@pytest.mark.parametrize("drain", [256, 512, 2048])
def test_same_bits_at_several_column_tiles(gpu_ctx, drain):
    """Three column tiles of 96 (single CTAs asked for) and other drain lengths, past a whole number of drains."""
    n, m, k = 900, 1500, 288
    ctx = gpu_ctx
    bed, _ = synth.synth_bed(51, n, m, 0.05)
    ctx.set_matvec_mode(MV_FP32_SIMT)
    ctx.setgeno(bed, n, m)
    V = np.random.default_rng(k).standard_normal((n, k)) * 10.0 ** np.linspace(-18, 18, k)
    prev = ctx.tc_options()
    try:
        ctx.set_matvec_mode(MV_SUBSET_EXACT)
        ctx.engine_reserve(320, 1)
        ctx.set_tc_option(TC_DRAIN_BYTES, drain)
        out = []
        for pair in (1, 0):
            ctx.set_tc_option(TC_SUBSET_PAIR, pair)
            ctx.engine_set_pheno(0, np.ones(n), np.array([1.0, 0.5]))
            ids = [int(i) for i in ctx.engine_submit(0, 1, V)]
            ctx.engine_reset_timing()
            ctx.engine_hold_results(True)
            ctx.engine_run()
            assert len(ctx.engine_step_trace()) == 1  # one launch over all of them
            out.append(np.column_stack([ctx.engine_fetch(i)[0] for i in ids]))
        np.testing.assert_array_equal(out[0], out[1])
        assert np.isfinite(out[0]).all() and np.abs(out[0]).max(0).min() > 0
    finally:
        ctx.engine_hold_results(False)
        ctx.set_tc_options(prev)
        ctx.set_matvec_mode(MV_FP32_SIMT)
