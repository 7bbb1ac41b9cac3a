"""A kernel's shared memory limit is one number for all host threads: a call that set it to its own size
could lower it between another thread's set and launch.  So every call sets the same value, at least what
any launch takes (above the default 48 KB).  The library's host code runs here against recorded CUDA calls."""
import concurrent.futures as cf
import ctypes
import subprocess
from pathlib import Path

import pytest

from segscan_gb300 import build
from segscan_gb300._lib import SsCsr, SsKnobs

HERE = Path(__file__).resolve().parent
PTR = 1 << 20  # device pointers are never dereferenced on the host


@pytest.fixture(scope="module")
def rec(lib, tmp_path_factory):
    out = tmp_path_factory.mktemp("recorded")
    srcs = [s for s in sorted(build.CSRC.glob("*.cu"))
            if s.stem in ("util", "backward", "sddmm") or "smem" in s.read_text()]

    def compile(src):
        obj = out / (src.stem + ".o")
        subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-O0", "-Xcicc", "-O0", "-Xptxas", "-O0", "-Xcompiler",
                        "-fPIC", "--expt-relaxed-constexpr", "-include", str(HERE / "cpp" / "record_launches.h"), "-I",
                        str(build.INCLUDE), "-c", str(src), "-o", str(obj)], check=True)
        return obj

    with cf.ThreadPoolExecutor(8) as ex:
        objs = list(ex.map(compile, srcs))
    rest = [build.BUILD / (s.stem + ".o") for s in sorted(build.CSRC.glob("*.cu")) if s not in srcs]
    so = out / "librecorded.so"
    subprocess.run([build.nvcc(), *build.ARCH, "-shared", "-o", str(so), *map(str, objs + rest)], check=True)
    return ctypes.CDLL(str(so))


def calls(rec, run):
    """[(kernel, bytes, is a launch)] of the CUDA calls that run() makes."""
    lo = rec.recorded_count()
    run()
    out = []
    for i in range(lo, rec.recorded_count()):
        fn, n, launch = ctypes.c_void_p(), ctypes.c_longlong(), ctypes.c_int()
        rec.recorded_get(ctypes.c_longlong(i), ctypes.byref(fn), ctypes.byref(n), ctypes.byref(launch))
        out.append((fn.value, n.value, bool(launch.value)))
    return out


def check(seen):
    """One limit per kernel, above all its launches; returns how many kernels set one."""
    limits, launches = {}, {}
    for fn, n, launch in seen:
        (launches if launch else limits).setdefault(fn, set()).add(n)
    for fn, values in limits.items():
        assert len(values) == 1, f"limits {sorted(values)}"
        assert max(values) <= 227 * 1024
        assert max(launches.get(fn, {0})) <= max(values), "launched above its limit"
    for fn, sizes in launches.items():
        assert fn in limits or max(sizes) <= 48 * 1024, f"{max(sizes)} bytes without a limit"
    return len(limits)


def ok(status, rec):
    rec.ss_last_error.restype = ctypes.c_char_p
    assert status == 0, rec.ss_last_error()


def big(n=1 << 40):
    return ctypes.c_size_t(n)


SIZES = [(1000, 5000), (4000, 60_000), (60_000, 200_000), (300_000, 1_000_000), (1_000_000, 4_600_000),
         (2_000_000, 4_000_000), (16_000_000, 20_000_000)]


def test_coo_to_csr(rec):
    def run():
        for nrow, nnz in SIZES:
            ok(rec.ss_coo_to_csr_values(nrow, nnz, ctypes.c_void_p(PTR), ctypes.c_void_p(PTR), ctypes.c_void_p(PTR), 0,
                                        *[ctypes.c_void_p(PTR)] * 5, big(), None), rec)

    seen = calls(rec, run)
    assert check(seen) == 2
    assert sum(launch for _, _, launch in seen) == 4 * len(SIZES)


def spmm_calls(rec, strategy, **knobs):
    n = ctypes.c_size_t()
    for nrow, nnz in [(100, 700)] + SIZES[:6]:
        for N in (1, 4, 8, 32, 47, 64, 100, 128, 300):
            for dtype in (0, 1):
                for accumulate in (0, 1):
                    A = SsCsr(nrow, nrow, nnz, PTR, PTR, PTR, dtype)
                    k = SsKnobs()
                    ok(rec.ss_default_knobs(strategy, N, ctypes.byref(k)), rec)
                    for name, v in knobs.items():
                        setattr(k, name, v)
                    ok(rec.ss_spmm(strategy, ctypes.byref(A), N, ctypes.c_void_p(PTR), ctypes.c_void_p(PTR), 0,
                                   accumulate, ctypes.byref(k), ctypes.c_void_p(PTR), big(), None), rec)


def test_rbsr(rec):
    assert check(calls(rec, lambda: spmm_calls(rec, 3))) >= 4


@pytest.mark.parametrize("thread_nz", [2, 256])
def test_ebsr_tile_and_group_walk(rec, thread_nz):
    def run():
        for block in (64, 256, 512):
            for gf in (0, 2, 4, 5):
                tnz = thread_nz if thread_nz < 256 else 4096 >> gf
                spmm_calls(rec, 2, thread_nz=tnz, group_factor=gf, thread_per_block=block)

    assert check(calls(rec, run)) > 0


def test_segment(rec):
    def run():
        for n in (100, 5000, 60_000, 1_000_000, 4_600_000):
            for N in (1, 4, 8, 47, 64, 128):
                for dtype in (0, 1):
                    for accumulate in (0, 1):
                        for gf, tnz in ((0, 1), (2, 8), (4, 8), (4, 256), (0, 4096)):
                            k = SsKnobs()
                            ok(rec.ss_default_knobs(2, N, ctypes.byref(k)), rec)
                            k.group_factor, k.thread_nz = gf, tnz
                            ok(rec.ss_segment_coo(1, ctypes.c_void_p(PTR), dtype, ctypes.c_void_p(PTR), n, N, n,
                                                  ctypes.c_void_p(PTR), 0, accumulate, ctypes.byref(k),
                                                  ctypes.c_void_p(PTR), big(), None), rec)

    check(calls(rec, run))


def test_batched(rec):
    def run():
        for sizes in ([(50, 100)] * 3, [(3000, 40_000)] * 40, [(50_000, 300_000)] * 60):
            for N in (1, 4, 8, 32, 64, 128):
                for dtype in (0, 1):
                    for block in (64, 256, 512):
                        for gf, tnz in ((0, 4), (4, 8), (5, 256), (0, 4096)):
                            count = len(sizes)
                            mats = (SsCsr * count)(*[SsCsr(m, m, n, PTR, PTR, PTR, dtype) for m, n in sizes])
                            knobs = (SsKnobs * count)()
                            for k in knobs:
                                ok(rec.ss_default_knobs(2, N, ctypes.byref(k)), rec)
                                k.group_factor, k.thread_nz, k.thread_per_block = gf, tnz, block
                            kinds = (ctypes.c_int * count)(*[2 if i % 3 else 3 for i in range(count)])
                            ptrs = (ctypes.c_void_p * count)(*[PTR] * count)
                            host, dev = ctypes.c_size_t(), ctypes.c_size_t()
                            ok(rec.ss_batch_plan_size_ex(count, mats, N, knobs, kinds, ctypes.byref(host),
                                                         ctypes.byref(dev)), rec)
                            plan = ctypes.create_string_buffer(host.value)
                            ok(rec.ss_batch_plan_ex(count, mats, N, ptrs, ptrs, 0, knobs, kinds, plan, host,
                                                    ctypes.c_void_p(PTR), dev, None), rec)
                            ok(rec.ss_spmm_batched(plan, ctypes.c_void_p(PTR), None), rec)

    assert check(calls(rec, run)) > 0


def test_transpose(rec):
    def run():
        for n, nnz in [(10, 5)] + SIZES:
            A = SsCsr(n, n, nnz, PTR, PTR, PTR, 0)
            ok(rec.ss_csr_transpose(ctypes.byref(A), *[ctypes.c_void_p(PTR)] * 4, big(), None),
               rec)

    seen = calls(rec, run)
    assert check(seen) == 2
    assert sum(launch for _, _, launch in seen) == 4 * (len(SIZES) + 1)
