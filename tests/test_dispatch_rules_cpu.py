"""Rules that choose a product's form by its sizes, as plain functions of the library (no GPU needed)."""
import ctypes as C

import pytest


def rule(name, *args):
    from saigegpu import build
    fn = getattr(C.CDLL(build.build_lib()), name)
    fn.restype = C.c_bool
    return fn(*args)


def i64(*v):
    return [C.c_int64(x) for x in v]


@pytest.mark.parametrize("n,m,cols,want", [
    (20000, 30000, 1, True), (20000, 48000, 64, True), (20000, 48001, 64, False), (1000, 2400, 63, True), (1023, 2000, 256, True), (1024, 2000, 65, False),
    (20000, 30000, 65, False), (20000, 12000, 65, True), (20000, 12000, 512, True), (20000, 12001, 65, False),
    (6000, 3600, 128, True), (5999, 3000, 128, False)])
def test_drop_ins_on_split_bf16_through_genotypes(n, m, cols, want):
    """Wide calls leave the genotypes where K's GEMM is the faster one."""
    assert rule("_ZN2sg22fp32_through_genotypesElll", *i64(n, m, cols)) is want


@pytest.mark.parametrize("np_,cols,want", [
    (128, 1, True), (24576, 16, True), (24576, 17, False), (8192, 64, True), (8192, 65, False), (8320, 17, False),
    (4096, 128, True), (4096, 129, False), (2048, 192, True), (2048, 193, False), (1024, 512, False)])
def test_drop_ins_on_fp32_by_gemv(np_, cols, want):
    """Wide calls leave the few-column kernel where the GEMM is the faster one."""
    assert rule("_ZN2sg12fp32_by_gemvEll", *i64(np_, cols)) is want


@pytest.mark.parametrize("cols,two_bit,want", [(32, True, False), (96, True, False), (128, True, True), (32, False, True),
                                               (96, False, True), (160, False, True), (512, True, True)])
def test_pairs_wherever_the_two_bit_form_does_not_serve(cols, two_bit, want):
    """Without the two-bit copy (refused memory, or the FP16 / E4M3 form) single CTAs are the slower ones."""
    assert rule("_ZN2sg14tc_subset_pairElb", C.c_int64(cols), C.c_bool(two_bit)) is want


@pytest.mark.parametrize("kind,where,want", [(2, 1, True), (2, 0, False), (3, 0, True), (1, 1, False), (0, -2, False)])
def test_which_images_a_kernel_reads(kind, where, want):
    """A .bed image in this device's memory or in managed memory is re-pitched in place; one on another device, or in host
    memory, goes through a copy.  kind: cudaMemoryType (0 unregistered, 1 host, 2 device, 3 managed)."""
    assert rule("_ZN2sg12kernel_readsEiii", C.c_int(kind), C.c_int(where), C.c_int(1)) is want
