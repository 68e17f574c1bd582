"""Failure detection without faulting the GPU: bounded device waits, host-side refusals and
per-request failures that leave the other requests running."""
import ctypes as C

import numpy as np
import pytest

from saigegpu import GRM_FP32_SIMT, MV_FP32_SIMT, MV_SUBSET_EXACT, Context, SaigeGpuError, prep, serve, synth

pytestmark = pytest.mark.gpu


def test_bounded_device_wait_reports_timeout_and_context_survives():
    with Context(0) as ctx:
        with pytest.raises(SaigeGpuError) as ei:
            ctx._call("sg_selftest_wait_timeout", 50.0)
        assert ei.value.code == 8  # SG_ERR_TIMEOUT
        n, m = 128, 200
        bed, _ = synth.synth_bed(2, n, m, 0.0)
        ctx.setgeno(bed, n, m)  # the context is still usable
        ctx.grm_build(GRM_FP32_SIMT)
        x, it = ctx.pcg_solve(np.full(n, 0.2), np.array([1.0, 0.3]), np.ones(n), 50, 1e-8)
        assert np.isfinite(x).all() and it > 0


def test_hbm_budget_refusal():
    n, m = 4000, 3000
    bed, _ = synth.synth_bed(3, n, m, 0.0)
    with Context(0, hbm_budget_bytes=8 << 20) as ctx:
        with pytest.raises(SaigeGpuError) as ei:
            ctx.setgeno(bed, n, m)
            ctx.grm_build(GRM_FP32_SIMT)
        assert ei.value.code == 3  # SG_ERR_NOMEM


def test_nan_inputs_are_rejected():
    n, m = 256, 300
    bed, _ = synth.synth_bed(4, n, m, 0.0)
    with Context(0) as ctx:
        ctx.setgeno(bed, n, m)
        ctx.grm_build(GRM_FP32_SIMT)
        w = np.full(n, 0.2)
        b = np.ones(n)
        b[7] = np.nan
        with pytest.raises(SaigeGpuError) as ei:
            ctx.pcg_solve(w, np.array([1.0, 0.3]), b)
        assert ei.value.code == 6
        w[3] = np.nan
        with pytest.raises(SaigeGpuError):
            ctx.engine_set_pheno(0, w, np.array([1.0, 0.3]))


def test_failing_and_cancelled_fits_do_not_stop_the_others():
    n, m = 500, 900
    bed, codes = synth.synth_bed(5, n, m, 0.01)
    with Context(0) as ctx:
        ctx.set_matvec_mode(MV_FP32_SIMT)
        ctx.setgeno(bed, n, m)
        ctx.grm_build(GRM_FP32_SIMT)
        gv = synth.genetic_value_from_codes(codes, 2)
        good = []
        for k in range(3):
            y, C = synth.simulate_pheno(gv, 20 + k, "binary", tau=0.5, prevalence=0.3)
            good.append(serve.FitSpec(prep.make_fit0(y, C, "binary", True), "binary"))
        yq = np.random.default_rng(0).standard_normal(n) * 0.01  # var(Y) < 0.1: the fit must stop
        bad = serve.FitSpec(prep.make_fit0(yq, None, "quantitative", False), "quantitative")
        r = serve.Runner(ctx, 512, 4)
        ids = [r.submit(s) for s in good[:2]] + [r.submit(bad), r.submit(good[2])]
        r.step()
        r.cancel(ids[1])
        r.run()
        by = {j.jid: j for j in r.finished}
        assert isinstance(by[ids[2]].error, ValueError)
        assert str(by[ids[1]].error) == "cancelled"
        for i in (ids[0], ids[3]):
            assert by[i].error is None and by[i].result["converged"]


@pytest.mark.parametrize("cleared", [False, True])
def test_a_step_whose_wait_ran_out_fails(cleared):
    """The flag the tcgen05 kernels set when a wait runs out, set from the host before a step: the step fails, also
    when the process-wide flag has been read and cleared (as another context's check does) before it is finished."""
    n, m = 256, 300
    bed, _ = synth.synth_bed(6, n, m, 0.0)
    V = np.random.default_rng(0).standard_normal((n, 2))
    cuda = C.CDLL("libcuda.so.1")
    with Context(0) as ctx:
        flag = ctx._L._ZN2sg16tc_error_addressEv
        flag.restype = C.c_void_p
        address = C.c_uint64(flag())
        assert address.value

        def put(v):
            assert cuda.cuMemcpyHtoD_v2(address, C.byref(C.c_int(v)), C.c_size_t(4)) == 0

        ctx.setgeno(bed, n, m)
        ctx.set_matvec_mode(MV_SUBSET_EXACT)
        ctx.engine_reserve(32, 1)
        ctx.engine_set_pheno(0, np.ones(n), np.array([1.0, 0.3]))
        ids = ctx.engine_submit(0, 1, V)
        put(3)
        try:
            ctx.engine_launch()
            ctx.engine_wait()
            if cleared:
                put(0)
            with pytest.raises(SaigeGpuError) as ei:
                ctx.engine_finish()
            assert ei.value.code == 2  # SG_ERR_CUDA
        finally:
            put(0)
        for i in ids:
            ctx.engine_cancel(i)
        np.testing.assert_allclose(ctx.grm_matmul(V), ctx.grm_matmul(V), rtol=0, atol=0)  # still usable


def test_a_launch_that_failed_is_reported_by_the_next_one():
    """A launch with too many grid rows (refused by the runtime: nothing runs) before one that first sets its kernel's
    shared memory, which would clear the error unread."""
    torch = pytest.importorskip("torch")
    with Context(0) as ctx:
        ctx.make_current()
        lib, buf = ctx._L, torch.zeros(4 << 16, dtype=torch.uint8, device="cuda:0")
        torch.cuda.synchronize()
        at = [C.c_void_p(buf.data_ptr() + (k << 16)) for k in range(4)]
        gemv = lib._ZN2sg17launch_gemv_multiEPKflS1_PKilPfP11CUstream_st
        gemv.restype = None
        build = lib._ZN2sg17launch_fp4_gbuildEPKhlPKillPvS4_P11CUstream_st
        # one marker of 16 samples: one stage of two row blocks each way, 24,576 bytes
        args = (at[0], C.c_int64(16), at[1], C.c_int64(1), C.c_int64(16), at[2], at[3], C.c_void_p(0))
        assert build(*args) == 0
        gemv(at[0], C.c_int64(128), at[1], at[2], C.c_int64(8 * 65536), at[3], C.c_void_p(0))
        assert build(*args) != 0
        assert build(*args) == 0
        torch.cuda.synchronize()
