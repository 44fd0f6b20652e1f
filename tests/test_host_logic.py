"""Host logic without a GPU: the launch planner and the kernels' per-thread tile routines,
executed thread by thread on the CPU by tests/emul/bfly_emul.cpp behind the same driver
that plans the GPU launches, compared with the oracle.  This checks panels, unit
decomposition, twiddle addressing, padding/slicing and the phase plan of the backward; it
is a test of index arithmetic, not a CPU implementation of the product."""
import ctypes
import math
import os
import subprocess

import pytest
import torch

from conftest import ROOT, assert_rtol_atol, golden_files, load_golden, rel_err, unitary_chain

EMUL_SRC = os.path.join(ROOT, "tests", "emul", "bfly_emul.cpp")
EMUL_LIB = os.path.join(ROOT, "tests", "emul", "libbfly_emul.so")
CSRC = os.path.join(ROOT, "butterfly_b200", "csrc")


@pytest.fixture(scope="module")
def emul():
    deps = [EMUL_SRC] + [os.path.join(CSRC, f) for f in sorted(os.listdir(CSRC)) if f.endswith(".h")]
    if not os.path.exists(EMUL_LIB) or os.path.getmtime(EMUL_LIB) < max(os.path.getmtime(f) for f in deps):
        subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-Wno-unknown-pragmas", "-I", CSRC,
                               EMUL_SRC, "-o", EMUL_LIB])
    return ctypes.CDLL(EMUL_LIB)


def emul_option(lib, name, value):
    from conftest import library_option
    return library_option(lambda n, v: lib.bfly_emul_set_option(n.encode(), int(v)),
                          lambda n: lib.bfly_emul_get_option(n.encode()), name, value)


def P(t):
    return ctypes.c_void_p(t.data_ptr() if t is not None and t.numel() else 0)


I64 = ctypes.c_int64


def emul_fw(lib, tw2, tw4, x, inc, out_size, log_n, nblocks, base4, threads=64, tail_untouched=True):
    B, S, insz = x.shape
    n = 1 << log_n
    out = torch.full((B, S, n), float("nan"), dtype=x.dtype)
    rc = lib.bfly_emul_fw(int(x.is_complex()), int(base4), P(tw2), P(tw4), P(x), I64(x.stride(0)), I64(x.stride(1)),
                          P(out), B, S, log_n, nblocks, insz, out_size, int(inc), threads)
    assert rc == 0, rc
    # columns >= out_size must stay untouched (a product that runs in several passes uses them as
    # working space)
    if tail_untouched:
        assert torch.isnan(out[:, :, out_size:]).all()
    return out[:, :, :out_size]


def emul_bw(lib, tw2, tw4, x, g, inc, log_n, nblocks, base4, threads=64, sms=7):
    B, S, insz = x.shape
    n = 1 << log_n
    d2 = torch.full_like(tw2, float("nan")) if tw2 is not None else None
    d4 = torch.full_like(tw4, float("nan")) if tw4 is not None else None
    dx = torch.full((B, S, max(insz, n)), float("nan"), dtype=x.dtype)
    g = g.contiguous()
    rc = lib.bfly_emul_bw(int(x.is_complex()), int(base4), P(tw2), P(tw4), P(x), I64(x.stride(0)), I64(x.stride(1)),
                          P(g), I64(g.stride(0)), I64(g.stride(1)), P(d2), P(d4), P(dx), B, S, log_n, nblocks, insz,
                          g.shape[2], int(inc), threads, sms)
    assert rc == 0, rc
    return d2, d4, dx[:, :, :insz]


@pytest.mark.parametrize("dtype", [torch.float32, torch.complex64], ids=["f32", "c64"])
@pytest.mark.parametrize("log_n", [1, 2, 3, 4, 5, 7, 9, 10, 11, 12])
def test_radix2_plan_and_indexing(emul, oracle_mod, dtype, log_n):
    torch.manual_seed(log_n)
    n = 1 << log_n
    shapes = [(n, n), (max(1, n // 2 - 1), max(1, n - 5)), (2 * n + 7, max(1, n // 2 - 2))] if log_n <= 7 else [(n, n)]
    for nb, inc in [(1, True), (1, False), (2, True), (3, False)]:
        if log_n >= 11 and nb == 3:
            continue
        S = 2 if log_n < 8 else 1
        B = 5 if log_n < 10 else 3
        for insz, outsz in shapes:
            tw = torch.randn(S, nb, log_n, n // 2, 2, 2, dtype=dtype) / 2 ** 0.5
            x = torch.randn(B, S, insz, dtype=dtype)
            g = torch.randn(B, S, outsz, dtype=dtype)
            thr = 64 if log_n < 10 else 256
            y = emul_fw(emul, tw, None, x, inc, outsz, log_n, nb, False, thr)
            assert rel_err(y, oracle_mod.multiply_fw(tw, x, inc, outsz)) < 2e-5
            d2, _, dx = emul_bw(emul, tw, None, x, g, inc, log_n, nb, False, thr)
            dtr, dxr = oracle_mod.multiply_bw(tw, x, g, inc)
            assert rel_err(d2, dtr) < 2e-5 and rel_err(dx, dxr) < 2e-5


@pytest.mark.parametrize("dtype", [torch.float32, torch.complex64], ids=["f32", "c64"])
@pytest.mark.parametrize("log_n", [1, 2, 3, 4, 5, 6, 7, 10, 11])
def test_base4_plan_and_indexing(emul, oracle_mod, log_n, dtype):
    torch.manual_seed(100 + log_n)
    n = 1 << log_n
    for nb, inc in [(1, True), (1, False), (2, True), (3, False)]:
        S, B = 2, 4
        for insz, outsz in [(n, n), (max(1, n // 2 - 1), max(1, n - 5)), (2 * n + 7, max(1, n // 2 - 2))]:
            tw4 = torch.randn(S, nb, log_n // 2, n // 4, 4, 4, dtype=dtype) / 2
            tw2 = torch.randn(S, nb, log_n % 2, n // 2, 2, 2, dtype=dtype) / 2 ** 0.5
            x = torch.randn(B, S, insz, dtype=dtype)
            g = torch.randn(B, S, outsz, dtype=dtype)
            y = emul_fw(emul, tw2, tw4, x, inc, outsz, log_n, nb, True)
            assert rel_err(y, oracle_mod.base4_fw(tw4, tw2, x, inc, outsz)) < 2e-5
            d2, d4, dx = emul_bw(emul, tw2, tw4, x, g, inc, log_n, nb, True)
            d4r, d2r, dxr = oracle_mod.base4_bw(tw4, tw2, x, g, inc)
            assert rel_err(dx, dxr) < 2e-5
            if tw4.numel():
                assert rel_err(d4, d4r) < 2e-5
            if tw2.numel():
                assert rel_err(d2, d2r) < 2e-5


def test_stack_broadcast_and_ragged_slices(emul, oracle_mod):
    torch.manual_seed(7)
    tw = torch.randn(3, 2, 6, 32, 2, 2) / 2 ** 0.5
    x = torch.randn(11, 1, 64).expand(11, 3, 64)  # stride 0 over stacks
    g = torch.randn(11, 3, 64)
    y = emul_fw(emul, tw, None, x, True, 64, 6, 2, False)
    assert rel_err(y, oracle_mod.multiply_fw(tw, x, True)) < 2e-5
    for sms in (1, 3, 7, 64):  # different row-slice splits must give the same sums
        d2, _, dx = emul_bw(emul, tw, None, x, g, True, 6, 2, False, sms=sms)
        dtr, dxr = oracle_mod.multiply_bw(tw, x, g, True)
        assert rel_err(d2, dtr) < 2e-5 and rel_err(dx, dxr) < 2e-5


@pytest.mark.parametrize("logc", [6, 7, 8])
def test_forward_passes_over_panels(emul, oracle_mod, logc):
    """Rows wider than a tile run as several forward launches over panels, in place; the
    fw_logcmax switch forces that path at sizes the emulator handles (the product path takes
    it for rows beyond one SM's shared memory)."""
    with emul_option(emul, "fw_logcmax", logc):
        _forward_passes_over_panels(emul, oracle_mod, logc)


def _forward_passes_over_panels(emul, oracle_mod, logc):
    torch.manual_seed(40 + logc)
    for dtype in (torch.float32, torch.complex64):
        for log_n, nb, inc in [(9, 1, True), (9, 2, False), (10, 2, True), (11, 1, False)]:
            n = 1 << log_n
            for insz, outsz in [(n, n), (n // 2 + 32, n - 64)]:
                S, B = 2, 3
                tw = torch.randn(S, nb, log_n, n // 2, 2, 2, dtype=dtype) / 2 ** 0.5
                x = torch.randn(B, S, insz, dtype=dtype)
                g = torch.randn(B, S, outsz, dtype=dtype)
                y = emul_fw(emul, tw, None, x, inc, outsz, log_n, nb, False, 64, tail_untouched=False)
                assert rel_err(y, oracle_mod.multiply_fw(tw, x, inc, outsz)) < 2e-5
                d2, _, dx = emul_bw(emul, tw, None, x, g, inc, log_n, nb, False, 64)
                dtr, dxr = oracle_mod.multiply_bw(tw, x, g, inc)
                assert rel_err(d2, dtr) < 2e-5 and rel_err(dx, dxr) < 2e-5
    # base-4, odd and even log_n (a radix-4 stage needs two panel bits plus 32-column segments)
    for log_n, nb, inc in ([(9, 2, True), (10, 1, False)] if logc >= 7 else []):
        n = 1 << log_n
        tw4 = torch.randn(1, nb, log_n // 2, n // 4, 4, 4) / 2
        tw2 = torch.randn(1, nb, log_n % 2, n // 2, 2, 2) / 2 ** 0.5
        x = torch.randn(3, 1, n)
        y = emul_fw(emul, tw2, tw4, x, inc, n, log_n, nb, True, tail_untouched=False)
        assert rel_err(y, oracle_mod.base4_fw(tw4, tw2, x, inc, n)) < 2e-5


@pytest.mark.parametrize("dtype", [torch.float32, torch.complex64], ids=["f32", "c64"])
def test_forward_that_saves_snapshots_feeds_the_backward(emul, oracle_mod, dtype):
    """bfly_fw_*_saving + bfly_bw_*_saved: the forward leaves the phase-boundary activations, the
    backward starts from them; results as from the recomputing pair."""
    torch.manual_seed(77)
    for log_n, nb, inc, thr in [(6, 3, True, 64), (10, 2, False, 256), (11, 2, True, 256), (4, 1, True, 64)]:
        n = 1 << log_n
        for insz, outsz in [(n, n), (max(1, n // 2 - 1), max(1, n - 5))]:
            S, B = 2, 5
            tw = torch.randn(S, nb, log_n, n // 2, 2, 2, dtype=dtype) / 2 ** 0.5
            x = torch.randn(B, S, insz, dtype=dtype)
            g = torch.randn(B, S, outsz, dtype=dtype)
            out = torch.full((B, S, n), float("nan"), dtype=dtype)
            d_tw = torch.full_like(tw, float("nan"))
            dx = torch.full((B, S, max(insz, n)), float("nan"), dtype=dtype)
            rc = emul.bfly_emul_fw_bw_saved(int(dtype.is_complex), P(tw), P(x), I64(x.stride(0)), I64(x.stride(1)), P(out),
                                            P(g), I64(g.stride(0)), I64(g.stride(1)), P(d_tw), P(dx), B, S, log_n, nb,
                                            insz, outsz, int(inc), thr, 7)
            assert rc == 0, rc
            assert rel_err(out[:, :, :outsz], oracle_mod.multiply_fw(tw, x, inc, outsz)) < 2e-5
            dtr, dxr = oracle_mod.multiply_bw(tw, x, g, inc)
            assert rel_err(d_tw, dtr) < 2e-5 and rel_err(dx[:, :, :insz], dxr) < 2e-5


def test_backward_in_chunks_of_phases(emul, oracle_mod):
    """More phases than one forward launch has snapshot slots for (here 9 and 11 blocks of 8 stages
    at n = 256): the backward runs in chunks, each with its own forward pass from the input."""
    torch.manual_seed(3)
    log_n, S, B = 8, 2, 5
    n = 1 << log_n
    for nb, inc in [(11, True), (9, False), (19, True)]:
        tw = torch.randn(S, nb, log_n, n // 2, 2, 2) / 2 ** 0.5
        x = torch.randn(B, S, n - 3)
        g = torch.randn(B, S, n - 7)
        # products of more than 40 stage groups run as several forward launches, in place on `out`
        y = emul_fw(emul, tw, None, x, inc, n - 7, log_n, nb, False, 64, tail_untouched=False)
        assert rel_err(y, oracle_mod.multiply_fw(tw, x, inc, n - 7)) < 5e-5
        d2, _, dx = emul_bw(emul, tw, None, x, g, inc, log_n, nb, False, 64)
        dtr, dxr = oracle_mod.multiply_bw(tw, x, g, inc)
        assert rel_err(d2, dtr) < 5e-5 and rel_err(dx, dxr) < 5e-5
    ws = ctypes.c_int64(0)
    assert emul.bfly_emul_bw_plan(0, 0, 16, 1, 10, 9, 1, ctypes.byref(ws)) > 9  # 90 stages: chunked
    assert ws.value == 9 * 16 * 1024 * 4 + 9 * 10 * 512 * 16  # 9 planes + the forward pass's re-ordered twiddles


def test_backward_phase_plan_sizes(emul):
    ws = ctypes.c_int64(0)
    # float: a phase holds at most 8 stages (4 sub-groups of 2) on a panel of 1024 columns
    assert emul.bfly_emul_bw_plan(0, 0, 64, 1, 8, 1, 1, ctypes.byref(ws)) == 1 and ws.value == 0
    assert emul.bfly_emul_bw_plan(0, 0, 64, 1, 10, 1, 1, ctypes.byref(ws)) == 2 and ws.value == 64 * 1024 * 4 + 10 * 512 * 16
    # n = 4096, two blocks: 24 stages = three phases of 8 -> two (B,S,n) float snapshots
    assert emul.bfly_emul_bw_plan(0, 0, 16384, 1, 12, 2, 1, ctypes.byref(ws)) == 3
    assert ws.value == 2 * 16384 * 4096 * 4 + 24 * 2048 * 16  # two snapshots + re-ordered twiddles of the forward pass
    # complex, n >= 1024: panels of 1024 columns, two 2-stage sub-groups (4 stages) per phase
    nph = emul.bfly_emul_bw_plan(1, 0, 8192, 1, 11, 1, 1, ctypes.byref(ws))
    assert nph == 3 and ws.value == 2 * 8192 * 2048 * 8
    # complex, n < 1024: panels of 512 columns, up to 10 one-stage sub-groups per phase
    nph = emul.bfly_emul_bw_plan(1, 0, 64, 1, 9, 2, 1, ctypes.byref(ws))
    assert nph == 2 and ws.value == 64 * 512 * 8
    with emul_option(emul, "bw_c64_kw2", 0):
        nph = emul.bfly_emul_bw_plan(1, 0, 8192, 1, 11, 1, 1, ctypes.byref(ws))
        assert nph == 2 and ws.value == 8192 * 2048 * 8


def test_complex_backward_on_two_stage_subgroups(emul, oracle_mod):
    """complex64 products of n >= 1024 run their backward phases on the tensor-memory kernel's step
    routines with 2-bit windows (two sub-groups of two stages); emulated here against the oracle."""
    torch.manual_seed(13)
    for log_n, nb, B, S, inc in ((10, 1, 9, 1, True), (11, 2, 6, 1, False), (12, 1, 5, 2, True)):
        n = 1 << log_n
        tw = torch.randn(S, nb, log_n, n // 2, 2, 2, dtype=torch.complex64) / 2 ** 0.5
        x = torch.randn(B, S, n - 5, dtype=torch.complex64)
        g = torch.randn(B, S, n - 9, dtype=torch.complex64)
        d2, _, dx = emul_bw(emul, tw, None, x, g, inc, log_n, nb, False, 256)
        dtr, dxr = oracle_mod.multiply_bw(tw, x, g, inc)
        assert rel_err(d2, dtr) < 2e-5 and rel_err(dx, dxr) < 2e-5, (log_n, nb)


def test_twiddle_stacks_beyond_32bit_offsets_are_refused(emul):
    """The kernels address twiddles with 32-bit element offsets inside a stack: the planner and
    the library's size queries refuse a stack of 2^31 elements or more instead of wrapping."""
    from butterfly_b200 import abi
    ws = ctypes.c_int64(0)
    # n = 2^20: a stack holds nblocks * 20 * 2^21 elements -- 51 blocks fit under 2^31, 52 do not
    assert emul.bfly_emul_bw_plan(0, 0, 4, 1, 20, 51, 1, ctypes.byref(ws)) > 0
    assert emul.bfly_emul_bw_plan(0, 0, 4, 1, 20, 52, 1, ctypes.byref(ws)) == -2
    assert emul.bfly_emul_bw_plan(1, 0, 4, 1, 24, 6, 1, ctypes.byref(ws)) == -2
    assert abi.bw_workspace_bytes(torch.float32, 4, 1, 20, 51) > 0
    assert abi.bw_workspace_bytes(torch.float32, 4, 1, 20, 52) == -2
    assert abi.fw_workspace_bytes(torch.float32, 4, 1, 20, 52) == -2
    assert abi.bw_workspace_bytes(torch.float32, 4, 1, 24, 3, base4=True) == -2  # 3 * 12 * 2^22 * 16 elements


@pytest.mark.parametrize("path", golden_files("radix2")[::4], ids=lambda p: p.split("/")[-1])
def test_emulated_kernels_on_golden(emul, path):
    d = load_golden(path)
    y = emul_fw(emul, d["twiddle"], None, d["input"], d["increasing_stride"], d["output_size"], d["log_n"],
                d["nblocks"], False)
    assert rel_err(y, d["output"]) < 2e-5
    d2, _, dx = emul_bw(emul, d["twiddle"], None, d["input"], d["grad"], d["increasing_stride"], d["log_n"],
                        d["nblocks"], False)
    assert rel_err(d2, d["d_twiddle"]) < 2e-5 and rel_err(dx, d["d_input"]) < 2e-5


def test_shared_memory_accesses_are_bank_conflict_free(emul):
    """With 256 threads per CTA, every register-window access of the planned groups (forward) and
    sub-groups (backward) must hit 32 distinct banks per wavefront, for the window widths the
    kernels use by default (3 bits float / 2 bits complex) at the benchmark sizes."""
    for dtype, kmax in ((0, 3), (1, 2)):
        for log_n in (10, 11, 12, 13):
            for nblocks, inc in ((1, 1), (2, 1), (2, 0)):
                deg = emul.bfly_emul_max_conflicts(dtype, 0, log_n, nblocks, inc, kmax)
                assert deg == 1, (dtype, log_n, nblocks, inc, deg)
    # base-4 (float): radix-4 windows of 2 bits
    for log_n in (10, 12, 14):
        assert emul.bfly_emul_max_conflicts(0, 1, log_n, 1, 1, 2) == 1


@pytest.mark.parametrize("log_n", [9, 10, 11, 12])
def test_packed_pair_forward_path(emul, oracle_mod, log_n):
    """Float rows of 512 .. 4096 columns take the packed-pair forward kernel (two columns per
    64-bit register, warps that own a 512-column chunk of the tile).  Its per-thread routines run
    here thread by thread; with the kernel switched off the generic kernel must give the same bits
    (both evaluate a butterfly output as fma(own, x, rn(partner * z)))."""
    torch.manual_seed(700 + log_n)
    emul.bfly_emul_fw2_calls.restype = ctypes.c_long
    n = 1 << log_n
    for nb, inc in [(1, True), (2, False), (3, True)]:
        for B, S, insz, outsz in [(2, 1, n, n), (37, 2, n - 32, n - 64), (9, 3, n + 3, 64)]:
            tw = torch.randn(S, nb, log_n, n // 2, 2, 2) / 2 ** 0.5
            x = torch.randn(B, S, insz)
            before = emul.bfly_emul_fw2_calls()
            y = emul_fw(emul, tw, None, x, inc, outsz, log_n, nb, False, 256)
            assert emul.bfly_emul_fw2_calls() == before + 1
            with emul_option(emul, "fw2", 0):
                y0 = emul_fw(emul, tw, None, x, inc, outsz, log_n, nb, False, 256)
            assert emul.bfly_emul_fw2_calls() == before + 1
            assert torch.equal(y, y0)
            assert rel_err(y, oracle_mod.multiply_fw(tw, x, inc, outsz)) < 2e-5
    # a ragged width (not a multiple of 32 columns) cannot be described to the TMA unit: generic kernel
    x = torch.randn(3, 1, n - 5)
    tw = torch.randn(1, 1, log_n, n // 2, 2, 2) / 2 ** 0.5
    before = emul.bfly_emul_fw2_calls()
    y = emul_fw(emul, tw, None, x, True, n, log_n, 1, False, 256)
    assert emul.bfly_emul_fw2_calls() == before
    assert rel_err(y, oracle_mod.multiply_fw(tw, x, True, n)) < 2e-5


@pytest.mark.parametrize("log_n", [10, 11, 12])
def test_packed_pair_backward_path(emul, oracle_mod, log_n):
    """Float radix-2 phases on full 1024-column panels take the packed-pair backward kernel (two
    columns per 64-bit register, twiddles and accumulators paired in tensor memory).  Its step
    routines run here thread by thread; with the kernel switched off the scalar kernels must give
    the same input gradient bits (same rounding order) and the same twiddle gradient up to the
    order of the row sums."""
    torch.manual_seed(800 + log_n)
    emul.bfly_emul_bw3_calls.restype = ctypes.c_long
    n = 1 << log_n
    for nb, inc in [(1, True), (2, False), (2, True)]:
        for B, S, insz, outsz in [(5, 1, n, n), (23, 2, n - 32, n - 64), (9, 1, n + 32, 64)]:
            tw = torch.randn(S, nb, log_n, n // 2, 2, 2) / 2 ** 0.5
            x = torch.randn(B, S, insz)
            g = torch.randn(B, S, outsz)
            before = emul.bfly_emul_bw3_calls()
            with emul_option(emul, "bw3_min_rows", 0):  # small batches would take the scalar kernel otherwise
                d2, _, dx = emul_bw(emul, tw, None, x, g, inc, log_n, nb, False, 256)
            assert emul.bfly_emul_bw3_calls() > before
            with emul_option(emul, "bw3", 0):
                mid = emul.bfly_emul_bw3_calls()
                d2s, _, dxs = emul_bw(emul, tw, None, x, g, inc, log_n, nb, False, 256)
                assert emul.bfly_emul_bw3_calls() == mid
            dtr, dxr = oracle_mod.multiply_bw(tw, x, g, inc)
            assert torch.equal(dx, dxs)
            assert rel_err(d2, d2s) < 1e-5
            assert rel_err(d2, dtr) < 2e-5 and rel_err(dx, dxr) < 2e-5


@pytest.mark.parametrize("log_n,S", [(10, 4), (11, 2), (12, 1)])
def test_fused_linear_layer(emul, oracle_mod, log_n, S):
    """Butterfly as a linear layer, fused: the forward adds the bias in its store epilogue, the backward
    sums the input gradient over the stacks in its last store and collects the bias gradient from
    the gradient tiles -- against the oracle composed with the reference's PyTorch glue
    (torch_butterfly/butterfly.py:152-169: expand, flatten, slice, add bias)."""
    torch.manual_seed(900 + log_n)
    n = 1 << log_n
    for nb, inc in [(1, True), (2, True), (2, False)]:
        for B, in_size in [(5, n), (23, n - 64)]:
            out_total = S * n
            tw = torch.randn(S, nb, log_n, n // 2, 2, 2) / 2 ** 0.5
            x = torch.randn(B, in_size)
            bias = torch.randn(out_total)
            g = torch.randn(B, out_total)
            # the unfused composition on the oracle
            xe = x.unsqueeze(1).expand(B, S, in_size)
            yr = oracle_mod.multiply_fw(tw, xe, inc).reshape(B, S * n) + bias
            dtr, dxr = oracle_mod.multiply_bw(tw, xe, g.reshape(B, S, n), inc)
            dxr, dbr = dxr.sum(1), g.sum(0)
            out = torch.full((B, S * n), float("nan"))
            rc = emul.bfly_emul_linear_fw(P(tw), P(x), I64(x.stride(0)), P(out), P(bias), B, S, log_n, nb, in_size, out_total, int(inc))
            assert rc == 0
            assert rel_err(out, yr) < 2e-5
            d_tw = torch.full_like(tw, float("nan")); d_in = torch.full((B, in_size), float("nan")); d_b = torch.full((out_total,), float("nan"))
            rc = emul.bfly_emul_linear_bw(P(tw), P(x), I64(x.stride(0)), P(g), I64(g.stride(0)), P(d_tw), P(d_in), I64(d_in.stride(0)),
                                          P(d_b), B, S, log_n, nb, in_size, out_total, int(inc), 7)
            if rc == -2:
                # a phase on strided column segments takes only rows that are whole groups of segments
                # (what the TMA descriptors can express): refused before anything is written
                assert in_size != n and torch.isnan(d_in).all() and torch.isnan(d_tw).all()
                continue
            assert rc == 0
            assert rel_err(d_tw, dtr) < 2e-5 and rel_err(d_in, dxr) < 2e-5 and rel_err(d_b, dbr) < 2e-5
    # a ragged input width is refused before anything is written
    x = torch.randn(8, n - 3); g = torch.randn(8, S * n); d_in = torch.full((8, n - 3), 7.0)
    tw = torch.randn(S, 1, log_n, n // 2, 2, 2)
    d_tw = torch.full_like(tw, 7.0)
    rc = emul.bfly_emul_linear_bw(P(tw), P(x), I64(x.stride(0)), P(g), I64(g.stride(0)), P(d_tw), P(d_in), I64(d_in.stride(0)),
                                  P(None), 8, S, log_n, 1, n - 3, S * n, 1, 7)
    assert rc == -2 and (d_in == 7.0).all() and (d_tw == 7.0).all()


def test_unitary_twiddle_arithmetic(emul):
    """The per-block arithmetic of the unitary twiddle kernels against the reference's chain of
    torch operators and autograd's backward of it."""
    torch.manual_seed(2)
    shape = (2, 2, 5, 16)
    angles = torch.cat([torch.asin(torch.sqrt(torch.rand(shape + (1,)))), torch.rand(shape + (3,)) * 2 * math.pi], dim=-1)
    blocks = angles.numel() // 4
    tw = torch.empty(shape + (2, 2), dtype=torch.complex64)
    emul.bfly_emul_unitary_fw(P(angles), P(tw), I64(blocks))
    a = angles.clone().requires_grad_(True)
    ref = unitary_chain(a)
    assert_rtol_atol(tw, ref.detach(), "unitary twiddle", rtol=1e-6, atol=1e-6)
    # unitary blocks: T T^H = I
    eye = tw @ tw.conj().transpose(-1, -2)
    assert (eye - torch.eye(2)).abs().max() < 1e-6
    g = torch.randn(shape + (2, 2), dtype=torch.complex64)
    ref.backward(g)
    d = torch.empty_like(angles)
    emul.bfly_emul_unitary_bw(P(angles), P(g), P(d), I64(blocks))
    assert_rtol_atol(d, a.grad, "unitary twiddle gradient", rtol=1e-5, atol=1e-6)


def _glue_reference(oracle_mod, tw, x, inc, in_perm, out_diag, out_perm, out_real):
    """The pipeline the glue forward replaces, operator by operator on the oracle."""
    xin = x.to(tw.dtype)
    if in_perm is not None:
        xin = xin[..., in_perm.long()]
    y = oracle_mod.multiply_fw(tw, xin.contiguous(), inc)
    if out_diag is not None:
        y = y * out_diag
    if out_perm is not None:
        y = y[..., out_perm.long()]
    return y.real.contiguous() if out_real else y


@pytest.mark.parametrize("cplx", [False, True])
def test_forward_with_glue_operators(emul, oracle_mod, cplx):
    """Gather before, diagonal and gather after, real input / output: the kernel's passes on the
    tile (emulated thread by thread) against the chain of separate operators."""
    torch.manual_seed(8)
    dtype = torch.complex64 if cplx else torch.float32
    for log_n, nb, B, S in ((6, 1, 5, 1), (9, 2, 9, 2), (11, 1, 3, 1)):
        n = 1 << log_n
        tw = torch.randn(S, nb, log_n, n // 2, 2, 2, dtype=dtype) / 2 ** 0.5
        for combo in range(8 if cplx else 4):
            use_in, use_out = bool(combo & 1), bool(combo & 2)
            real_io = bool(combo & 4)
            x = torch.randn(B, S, n, dtype=torch.float32 if real_io else dtype)
            in_perm = torch.randperm(n, dtype=torch.int32) if use_in else None
            out_perm = torch.randperm(n, dtype=torch.int32) if use_out else None
            out_diag = torch.randn(n, dtype=dtype) if use_out else None
            out = torch.full((B, S, n), float("nan"), dtype=torch.float32 if real_io else dtype)
            rc = emul.bfly_emul_fw_glue(int(cplx), P(tw), P(x), int(real_io), I64(x.stride(0)), I64(x.stride(1)), P(out), int(real_io),
                                        P(in_perm), P(out_diag), P(out_perm), B, S, log_n, nb, n, n, 1, 256)
            assert rc == 0, (log_n, combo, rc)
            want = _glue_reference(oracle_mod, tw, x, True, in_perm, out_diag, out_perm, real_io)
            assert_rtol_atol(out, want, "glue forward n=%d combo=%d" % (n, combo), rtol=1e-4, atol=1e-4)
    # rows wider than a tile, gathers on ragged sizes: refused
    n = 1 << 13
    tw = torch.randn(1, 1, 13, n // 2, 2, 2)
    x = torch.randn(2, 1, n)
    perm = torch.randperm(n, dtype=torch.int32)
    assert emul.bfly_emul_fw_glue(0, P(tw), P(x), 0, I64(n), I64(n), P(torch.empty(2, 1, n)), 0, P(perm), None, None,
                                  2, 1, 13, 1, n, n, 1, 256) == -2
    tw = torch.randn(1, 1, 6, 32, 2, 2)
    x = torch.randn(2, 1, 64)
    perm = torch.randperm(64, dtype=torch.int32)
    assert emul.bfly_emul_fw_glue(0, P(tw), P(x), 0, I64(64), I64(64), P(torch.empty(2, 1, 64)), 0, P(perm), None, None,
                                  2, 1, 6, 1, 60, 64, 1, 256) == -1


def test_packed_pair_forward_on_wide_rows(emul, oracle_mod):
    """float32 rows of 8192 columns run the packed-pair forward in one launch (512-thread CTAs); rows of
    16384 columns pass by pass on 4096-column panels (contiguous for the low bits, 32-column blocks at
    a stride for the top bits); both also as the backward's snapshot pass.  Input that the kernel's
    descriptors cannot cover falls back to the generic kernel."""
    torch.manual_seed(21)
    for log_n, nb, B, inc in ((13, 2, 5, True), (13, 1, 3, False), (14, 2, 2, True)):
        n = 1 << log_n
        tw = torch.randn(1, nb, log_n, n // 2, 2, 2) / 2 ** 0.5
        x = torch.randn(B, 1, n)
        calls = emul.bfly_emul_fw2_calls()
        y = emul_fw(emul, tw, None, x, inc, n - 96, log_n, nb, False, 256, tail_untouched=False)
        assert emul.bfly_emul_fw2_calls() - calls == (1 if log_n == 13 else 3), (log_n, nb)
        assert rel_err(y, oracle_mod.multiply_fw(tw, x, inc, n - 96)) < 2e-5
        g = torch.randn(B, 1, n)
        calls = emul.bfly_emul_fw2_calls()
        d2, _, dx = emul_bw(emul, tw, None, x, g, inc, log_n, nb, False, 256)
        assert emul.bfly_emul_fw2_calls() > calls  # the snapshot pass
        dtr, dxr = oracle_mod.multiply_bw(tw, x, g, inc)
        assert rel_err(d2, dtr) < 2e-5 and rel_err(dx, dxr) < 2e-5
    # two stacks of 8192 columns: still one launch; with the one-launch path refused (input not a
    # multiple of 32 columns) a single stack cannot take the panel passes either: generic passes
    n = 1 << 13
    tw2 = torch.randn(2, 1, 13, n // 2, 2, 2) / 2 ** 0.5
    x2 = torch.randn(3, 2, n)
    calls = emul.bfly_emul_fw2_calls()
    y2 = emul_fw(emul, tw2, None, x2, False, n, 13, 1, False, 256)
    assert emul.bfly_emul_fw2_calls() - calls == 1
    assert rel_err(y2, oracle_mod.multiply_fw(tw2, x2, False, n)) < 2e-5
    tw = torch.randn(1, 1, 13, n // 2, 2, 2) / 2 ** 0.5
    x = torch.randn(3, 1, n - 65)
    calls = emul.bfly_emul_fw2_calls()
    y = emul_fw(emul, tw, None, x, True, n, 13, 1, False, 256)
    assert emul.bfly_emul_fw2_calls() == calls
    assert rel_err(y, oracle_mod.multiply_fw(tw, x, True, n)) < 2e-5


@pytest.mark.parametrize("cplx,base4,log_n,S,nblocks,cut,extra", [
    (0, 0, 2, 1, 2, 0, 1), (0, 0, 5, 2, 1, 0, 3), (0, 0, 6, 1, 2, 0, 5), (0, 0, 8, 1, 1, 3, 1), (0, 0, 9, 1, 2, 64, 1),
    (0, 1, 6, 1, 1, 0, 5), (0, 1, 7, 2, 1, 1, 3), (0, 1, 10, 1, 1, 32, 3), (1, 0, 3, 1, 1, 0, 7), (1, 0, 8, 2, 1, 3, 5)])
def test_several_rows_to_a_tile_row(emul, oracle_mod, cplx, base4, log_n, S, nblocks, cut, extra):
    """Narrow rows of 2^21 values and more share a tile row.  A batch that does not fill the last one, cut and unaligned
    widths: against the oracle, and outputs and input gradients bit by bit against the same product row by row."""
    torch.manual_seed(log_n)
    n, dt = 1 << log_n, torch.complex64 if cplx else torch.float32
    B = (1 << 21) // n + extra
    tw2 = torch.randn(S, nblocks, log_n % 2 if base4 else log_n, n // 2, 2, 2, dtype=dt) / 2 ** 0.5
    tw4 = torch.randn(S, nblocks, log_n // 2, n // 4, 4, 4, dtype=dt) / 2 if base4 else None
    x, g = torch.randn(B, S, n - cut, dtype=dt), torch.randn(B, S, n - cut // 2, dtype=dt)
    run = lambda: (emul_fw(emul, tw2, tw4, x, True, g.shape[2], log_n, nblocks, base4, 256),
                   *emul_bw(emul, tw2, tw4, x, g, True, log_n, nblocks, base4, 256))
    y, d2, d4, dx = run()
    with emul_option(emul, "virtual_rows", 0):
        ys, _, _, dxs = run()
    assert torch.equal(y, ys) and torch.equal(dx, dxs)
    wide = torch.complex128 if cplx else torch.float64
    w = lambda t: t.to(wide)
    if base4:
        d4r, d2r, dxr = oracle_mod.base4_bw(w(tw4), w(tw2), w(x), w(g), True)
        yr = oracle_mod.base4_fw(w(tw4), w(tw2), w(x), True, g.shape[2])
    else:
        (d2r, dxr), d4r = oracle_mod.multiply_bw(w(tw2), w(x), w(g), True), None
        yr = oracle_mod.multiply_fw(w(tw2), w(x), True, g.shape[2])
    assert rel_err(y, yr.to(dt)) < 2e-5 and rel_err(dx, dxr.to(dt)) < 2e-5
    for a, b in ((d2, d2r), (d4, d4r)):  # sums over up to 2^19 rows: the emulator adds them one by one, 2^-24 * sqrt(rows) each way
        assert a is None or not a.numel() or rel_err(a, b.to(dt)) < 1e-4


@pytest.mark.parametrize("cplx,log_n,S", [(1, 2, 1), (1, 5, 2), (1, 8, 1), (0, 6, 2), (0, 9, 1)])
def test_glue_of_rows_that_share_a_tile_row(emul, oracle_mod, cplx, log_n, S):
    torch.manual_seed(50 + log_n)
    n, dt = 1 << log_n, torch.complex64 if cplx else torch.float32
    B = (1 << 21) // n + 3
    tw = torch.randn(S, 1, log_n, n // 2, 2, 2, dtype=dt) / 2 ** 0.5
    for combo in (1, 2, 4, 6, 7, 15) if cplx else (1, 4, 7):
        real_io = bool(combo & 8)
        x = torch.randn(B, S, n, dtype=torch.float32 if real_io else dt)
        in_perm, out_perm = (torch.randperm(n, dtype=torch.int32) if combo & bit else None for bit in (1, 2))
        diag = torch.randn(n, dtype=dt) if combo & 4 else None
        out = torch.full((B, S, n), float("nan"), dtype=x.dtype)
        rc = emul.bfly_emul_fw_glue(int(cplx), P(tw), P(x), int(real_io), I64(x.stride(0)), I64(x.stride(1)), P(out), int(real_io),
                                    P(in_perm), P(diag), P(out_perm), B, S, log_n, 1, n, n, 1, 256)
        assert rc == 0
        want = _glue_reference(oracle_mod, tw, x, True, in_perm, diag, out_perm, real_io)
        assert_rtol_atol(out, want, "glue of narrow rows n=%d combo=%d" % (n, combo), rtol=1e-4, atol=1e-4)


def test_glue_of_padded_rows(emul, oracle_mod):
    """Rows narrower than n enter padded where nothing gathers them (circulants of any length), real and complex, with a
    diagonal and a gather behind the product, at widths with and without 16-byte rows."""
    torch.manual_seed(60)
    for log_n, B in ((5, 9), (9, 7), (11, 4), (6, (1 << 21) // 64 + 3)):
        n = 1 << log_n
        tw = torch.randn(1, 1, log_n, n // 2, 2, 2, dtype=torch.complex64) / 2 ** 0.5
        for width, real_in, use_diag, use_perm, real_out in ((n // 2 + 1, 1, 1, 0, 0), (n // 2 + 4, 1, 1, 0, 0), (n - 7, 0, 0, 1, 0), (n - 3, 1, 0, 0, 1),
                                                             (n - 2, 0, 1, 0, 1)):
            x = torch.randn(B, 1, width, dtype=torch.float32 if real_in else torch.complex64)
            diag = torch.randn(n, dtype=torch.complex64) if use_diag else None
            perm = torch.randperm(n, dtype=torch.int32) if use_perm else None
            out = torch.full((B, 1, n), float("nan"), dtype=torch.float32 if real_out else torch.complex64)
            rc = emul.bfly_emul_fw_glue(1, P(tw), P(x), real_in, I64(x.stride(0)), I64(x.stride(1)), P(out), real_out, None, P(diag), P(perm),
                                        B, 1, log_n, 1, width, n, 1, 256)
            assert rc == 0
            xp = torch.zeros(B, 1, n, dtype=torch.complex64)
            xp[..., :width] = x
            want = _glue_reference(oracle_mod, tw, xp, True, None, diag, perm, bool(real_out))
            assert_rtol_atol(out, want, "glue of padded rows n=%d width=%d" % (n, width), rtol=1e-4, atol=1e-4)


def emul_layer(lib, kind, tws, x, bias, g, S, log_n, nblocks, inc, save, threads=256, sms=7):
    """Output, d_input, d_bias and twiddle gradients of a layer through the driver's layer calls."""
    base4, B, n = kind == "base4", x.shape[0], 1 << log_n
    tw4, tw2 = tws if base4 else (None, tws[0])
    out = torch.full((B, S * n), float("nan"), dtype=x.dtype)
    d4, d2 = (None if t is None else torch.full_like(t, float("nan")) for t in (tw4, tw2))
    d_in = torch.full((B, x.shape[1] if S > 1 else max(x.shape[1], n)), float("nan"), dtype=x.dtype)
    d_b = None if bias is None else torch.full_like(bias, float("nan"))
    rc = lib.bfly_emul_layer(int(x.is_complex()), int(base4), P(tw2), P(tw4), P(x), I64(x.stride(0)), P(bias), P(out), P(g), I64(g.stride(0)),
                             P(d2), P(d4), P(d_in), P(d_b), B, S, log_n, nblocks, x.shape[1], g.shape[1], int(inc), int(save), threads, sms)
    return rc, out[:, :g.shape[1]], d_in[:, :x.shape[1]], d_b, [d4, d2] if base4 else [d2]


@pytest.mark.parametrize("save", [0, 1])
@pytest.mark.parametrize("kind,in_size,S,out_size,nblocks,B", [
    ("f32", 1000, 3, 3000, 1, 37), ("f32", 1024, 2, 2048, 2, 60), ("f32", 1023, 2, 1025, 2, 1), ("f32", 5, 1, 2, 1, 1), ("f32", 96, 1, 100, 2, 21),
    ("f32", 8000, 1, 8192, 1, 3), ("f32", 70, 2, 200, 1, (1 << 21) // 128 + 3), ("f32", 64, 2, 128, 1, (1 << 21) // 64 + 3),
    ("c64", 1000, 2, 1500, 2, 9), ("c64", 100, 1, 120, 1, (1 << 21) // 128 + 5), ("base4", 500, 1, 512, 2, 11), ("base4", 1024, 2, 2000, 1, 7),
    ("base4", 100, 1, 120, 1, (1 << 21) // 128 + 5)])
def test_layers(emul, oracle_mod, kind, in_size, S, out_size, nblocks, B, save):
    """A whole layer: padded input shared by the stacks, cut last stack read as one matrix, bias on the tile, input
    gradient summed over the stacks, with and without the forward's snapshots, rows that share a tile row."""
    torch.manual_seed(in_size + nblocks)
    log_n = max(1, (in_size - 1).bit_length())
    n, dt = 1 << log_n, torch.complex64 if kind == "c64" else torch.float32
    wide = torch.complex128 if kind == "c64" else torch.float64
    x, g, bias = torch.randn(B, in_size, dtype=dt), torch.randn(B, out_size, dtype=dt), torch.randn(out_size, dtype=dt)
    xe = x.to(wide).unsqueeze(1).expand(B, S, in_size).contiguous()
    gp = torch.zeros(B, S * n, dtype=wide)
    gp[:, :out_size] = g
    if kind == "base4":
        tws = [torch.randn(S, nblocks, log_n // 2, n // 4, 4, 4) / 2, torch.randn(S, nblocks, log_n % 2, n // 2, 2, 2) / 2 ** 0.5]
        y = oracle_mod.base4_fw(*[t.to(wide) for t in tws], xe, True)
        d4, d2, dx = oracle_mod.base4_bw(*[t.to(wide) for t in tws], xe, gp.view(B, S, n), True)
        dtw = [d4, d2]
    else:
        tws = [torch.randn(S, nblocks, log_n, n // 2, 2, 2, dtype=dt) / 2 ** 0.5]
        y = oracle_mod.multiply_fw(tws[0].to(wide), xe, True)
        d, dx = oracle_mod.multiply_bw(tws[0].to(wide), xe, gp.view(B, S, n), True)
        dtw = [d]
    want = [y.reshape(B, S * n)[:, :out_size] + bias, dx.sum(1), g.to(wide).sum(0)] + dtw
    rc, out, d_in, d_b, d_tw = emul_layer(emul, kind, tws, x, bias, g, S, log_n, nblocks, True, save)
    assert rc == 0
    for got, ref, what in zip([out, d_in, d_b] + d_tw, want, ("output", "d_input", "d_bias", "d_twiddle", "d_twiddle2")):
        assert got.shape == ref.shape and (not got.numel() or rel_err(got, ref.to(dt)) < (2e-5 if B < 1000 else 1e-4)), what


def test_missing_tensors_are_refused(emul):
    """A NULL where the kernels would read or write is an argument error: the odd factors' twiddle2 of a radix-4 product,
    and every tensor of a layer's backward."""
    n, log_n = 32, 5
    tw4, tw2 = torch.randn(1, 1, 2, 8, 4, 4), torch.randn(1, 1, 1, 16, 2, 2)
    x, out = torch.randn(3, 1, n), torch.empty(3, 1, n)
    fw = lambda a, b: emul.bfly_emul_fw(0, 1, P(a), P(b), P(x), I64(n), I64(n), P(out), 3, 1, log_n, 1, n, n, 1, 64)
    assert fw(tw2, tw4) == 0 and fw(None, tw4) == -1 and fw(tw2, None) == -1
    tw = torch.randn(2, 1, log_n, 16, 2, 2)
    x, g, bias = torch.randn(3, n), torch.randn(3, 50), torch.randn(50)
    full = dict(d2=torch.empty_like(tw), d_in=torch.empty(3, n), x=x, g=g, out=torch.empty(3, 2 * n))
    for missing in (None, "d_in", "g", "d2", "x", "out"):
        t = {k: None if k == missing else v for k, v in full.items()}
        rc = emul.bfly_emul_layer(0, 0, P(tw), None, P(t["x"]), I64(n), P(bias), P(t["out"]), P(t["g"]), I64(50), P(t["d2"]), None, P(t["d_in"]),
                                  None, 3, 2, log_n, 1, n, 50, 1, 0, 64, 7)
        assert rc == (-1 if missing else 0), missing


@pytest.mark.parametrize("S", [1, 2])
def test_layer_without_output_columns(emul, S):
    """out_size 0: the gradient matrix has no column, and every gradient is zero."""
    tw, x, g = torch.randn(S, 1, 5, 16, 2, 2), torch.randn(4, 30), torch.full((4, 0), float("nan"))
    rc, out, d_in, _, (d_tw,) = emul_layer(emul, "f32", [tw], x, None, g, S, 5, 1, True, 0)
    assert rc == 0 and out.shape == (4, 0) and (d_in == 0).all() and (d_tw == 0).all()


def test_rows_between_elements_are_refused(emul):
    """Rows that cannot move in 16-byte accesses move one element at a time, complex ones 8 bytes: every complex row tensor
    that starts four bytes off is refused."""
    n, log_n, c64 = 8, 3, torch.complex64
    tw = torch.randn(1, 1, log_n, n // 2, 2, 2, dtype=c64)
    off = lambda t, by: ctypes.c_void_p(t.data_ptr() + by)
    for which in ("none", "x", "out", "g", "dx"):
        t = {k: torch.zeros(3, 1, n + 1, dtype=c64) for k in ("x", "out", "g", "dx")}
        p = {k: off(v, 4 if k == which else 0) for k, v in t.items()}
        d_tw = torch.empty_like(tw)
        s = (I64(n), I64(n))
        fw = emul.bfly_emul_fw(1, 0, P(tw), None, p["x"], *s, p["out"], 3, 1, log_n, 1, n, n, 1, 64)
        bw = emul.bfly_emul_bw(1, 0, P(tw), None, p["x"], *s, p["g"], *s, P(d_tw), None, p["dx"], 3, 1, log_n, 1, n, n, 1, 64, 7)
        both = emul.bfly_emul_fw_bw_saved(1, P(tw), p["x"], *s, p["out"], p["g"], *s, P(d_tw), p["dx"], 3, 1, log_n, 1, n, n, 1, 64, 7)
        layer = emul.bfly_emul_layer(1, 0, P(tw), None, p["x"], I64(n), None, p["out"], p["g"], I64(n), P(d_tw), None, p["dx"], None, 3, 1, log_n, 1,
                                     n, n, 1, 0, 64, 7)
        glue = emul.bfly_emul_fw_glue(1, P(tw), p["x"], 0, *s, p["out"], 0, None, None, None, 3, 1, log_n, 1, n, n, 1, 64)
        bad = lambda *names: -3 if which in names else 0
        assert (fw, bw, both, layer, glue) == (bad("x", "out"), bad("x", "g", "dx"), bad(*p), bad(*p), bad("x", "out")), which


def test_kronecker_twiddle_as_transforms_see_it():
    """The twiddle of a 2-D map is index work, the same on any device: gradients, forward mode and functorch transforms go
    through it, tensors of two devices do not."""
    import butterfly_b200 as bb
    from torch.autograd import forward_ad
    torch.manual_seed(4)
    t1, t2 = (torch.randn(1, 2, l, 1 << (l - 1), 2, 2, dtype=torch.float64) for l in (3, 2))
    v = torch.randn_like(t1)
    for inc in (True, False):
        k = lambda a, b=t2: bb.combine.kronecker_twiddle(a, b, inc)
        want = k(v, torch.zeros_like(t2))  # linear in the pair
        with forward_ad.dual_level():
            assert torch.equal(forward_ad.unpack_dual(k(forward_ad.make_dual(t1, v))).tangent, want)
        assert torch.equal(torch.func.jvp(k, (t1,), (v,))[1], want)
        assert torch.equal(torch.func.vmap(k)(torch.stack([t1, v])), torch.stack([k(t1), k(v)]))
        g = torch.randn_like(want)
        leaf = t1.clone().requires_grad_(True)
        d, = torch.autograd.grad(k(leaf), leaf, g)
        assert torch.allclose(torch.func.vjp(k, t1)[1](g)[0], d)
        assert abs(((d * v).sum() - (want * g).sum()).item()) < 1e-9  # the adjoint of the forward
        assert torch.autograd.gradgradcheck(k, (leaf,))
    with pytest.raises(RuntimeError, match="same device"):
        bb.combine.kronecker_twiddle(t1.to("meta"), t2, True)


@pytest.mark.parametrize("dtype", [0, 1], ids=["f32", "c64"])
@pytest.mark.parametrize("how", ["saved", "recomputed"])
def test_queried_bytes_are_enough_for_what_runs(emul, dtype, how):
    """Training steps under the default options with buffers of exactly the queried sizes, from 16 bytes past a boundary: both
    directions, one to three blocks, up to 2^26 values, on either side of the rule for tensor-core passes.  Nothing is
    refused and no launch leaves a buffer.  (A product may qualify for the passes in one direction and not in the other.)"""
    routes = {}
    for log_n in range(5, 16):
        rows = [300, 777] + [(1 << k) + d for k in range(9, 18) for d in (0, 5)]
        for B in rows:
            for S in (1, 3):
                if B * S << log_n > 1 << 26:
                    continue
                for nb in (1, 2, 3):
                    for base4 in (0, 1):
                        for inc in (0, 1):
                            passes = ctypes.c_int(0)
                            rc = emul.bfly_emul_dry_step(dtype, base4, int(how == "recomputed"), I64(16), B, S, log_n, nb, 1 << log_n, 1 << log_n, inc,
                                                         ctypes.byref(passes))
                            assert rc == 0, (log_n, B, S, nb, base4, inc, rc)
                            routes[log_n, B, S, nb, base4, inc] = passes.value > 0
    one_way = [k for k, v in routes.items() if v and not routes[k[:-1] + (1 - k[-1],)]]
    assert one_way and any(routes.values()) and not all(routes.values())


@pytest.mark.parametrize("dtype", [0, 1], ids=["f32", "c64"])
@pytest.mark.parametrize("save", [0, 1])
def test_queried_bytes_are_enough_for_layers(emul, dtype, save):
    """The same for whole layers: widths that are cut, several stacks, the last one cut short, bias."""
    routes = set()
    for log_n in (6, 9, 10, 12, 14):
        n = 1 << log_n
        for B in (5, 300, 777, 2048, 8192 + 3, 65536):
            for in_size, out_total in ((n, n), (n - 24, n - 20), (n, 4 * n), (n - 24, 3 * n - 72), (n + 5, n), (n, 2 * n + 1)):
                S = -(-out_total // n)
                if B * S << log_n > 1 << 26:
                    continue
                for nb, base4, inc in ((1, 0, 1), (2, 0, 1), (2, 0, 0), (1, 1, 1), (2, 1, 1), (2, 1, 0)):
                    passes = ctypes.c_int(0)
                    rc = emul.bfly_emul_dry_layer(dtype, base4, save, I64(16), B, S, log_n, nb, in_size, out_total, inc, ctypes.byref(passes))
                    assert rc == 0, (log_n, B, in_size, out_total, nb, base4, inc, rc)
                    routes.add(passes.value > 0)
    assert routes == {True, False}


@pytest.mark.parametrize("dtype", [0, 1], ids=["f32", "c64"])
def test_plan_of_the_passes(emul, dtype):
    """Wherever the passes can run: every stage in one group and its bits in the group's window, every column in one block,
    every tile at one CTA, every sum in a slot of its own."""
    assert emul.bfly_emul_set_option(b"mma", 1) == 0
    try:
        groups = set()
        for log_n in range(5, 16):
            for nb in (1, 2, 3):
                for base4 in (0, 1):
                    for inc in (0, 1):
                        for B, S, ctas in ((1, 1, 148), (300, 3, 148), (5000, 1, 148), (4097, 5, 132), (129, 2, 7), (20000, 1, 160), (32768, 1, 148), (32768, 1, 64), (16384, 2, 128),
                                           (1 << 20, 1, 148), (8192 * 128, 1, 64)):
                            if B * S << log_n > 1 << 27 or (B > 1 << 19 and log_n > 7):
                                continue
                            got = emul.bfly_emul_check_mma_plan(dtype, base4, B, S, log_n, nb, inc, ctas)
                            assert got <= 0, (log_n, nb, base4, inc, B, S, ctas, got)
                            groups.add(-got)
        assert {1, 2, 3, 5} <= groups
    finally:
        emul.bfly_emul_set_option(b"mma", -1)


def test_saved_bytes_of_one_direction():
    """What is held between forward and backward is what the direction needs, not the larger of both (three planes of phases
    against two of passes for 16384 rows of 4096 floats, two blocks)."""
    from butterfly_b200 import abi
    lib = abi.lib()
    for name in ("bfly_fw_saving_bytes", "bfly_bw_snapshot_bytes"):
        getattr(lib, name).restype = ctypes.c_int64
    up, down = (lib.bfly_fw_saving_bytes(0, 16384, 1, 12, 2, inc) for inc in (1, 0))
    plane = 16384 * 4096 * 4
    assert 2 * plane < up < 2.1 * plane and 3 * plane < down < 3.1 * plane
    assert lib.bfly_bw_snapshot_bytes(0, 16384, 1, 12, 2) == max(up, down)
    assert lib.bfly_fw_saving_bytes(0, 16384, 1, 40, 2, 1) < 0
