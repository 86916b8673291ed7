"""Host side of the grid build and of context creation, on a CUDA runtime that
runs nothing (fake_cudart.cpp): a launch that fails ends the build, and the
next build starts from cleared counts; a context is handed out when all that
was cleared and copied for it is done."""

import ctypes as C
import os
import subprocess

import pytest

from fluid_simulation_b200 import _lib, build

HERE = os.path.dirname(os.path.abspath(__file__))
STUB = """
#include "%s/fs_internal.cuh"
namespace fs {
int reduction_blocks(int64_t n) { return (int)(n / 2 + 1); }
size_t metrics_scratch_bytes(int64_t) { return 256; }
}
"""
KERNELS = ["k_cell_keys", "k_scan", "k_scatter", "k_rank"]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("fake")
    stub = d / "stub.cu"
    stub.write_text(STUB % build.CSRC)
    out = d / "libgrid_fake.so"
    flags = [f for f in build.NVCC_FLAGS if f not in ("-O3", "-lineinfo")]
    subprocess.check_call([build.NVCC, *flags, "-O1", "-Xptxas", "-O0", "-cudart", "none", "-Xlinker", "-Bsymbolic",
                           "-o", str(out),
                           os.path.join(build.CSRC, "fs_grid.cu"), str(stub), os.path.join(HERE, "fake_cudart.cpp")])
    lib = C.CDLL(str(out))
    lib.fake_calls.restype = C.c_char_p
    for name in ("fs_context_create", "fs_context_create_worlds", "fs_context_destroy", "fs_grid_build", "fs_grid_tables",
                 "fs_last_error_string"):
        getattr(lib, name).restype, getattr(lib, name).argtypes = _lib.SIGNATURES[name]
    return lib


def calls(lib):
    lines = lib.fake_calls().decode().splitlines()
    lib.fake_clear()
    return lines


def launches(lines):
    return [next(k for k in KERNELS if k in ln) for ln in lines if ln.startswith("launch")]


@pytest.fixture
def ctx(lib):
    p = C.c_void_p()
    assert lib.fs_context_create(C.byref(p), 1000, C.byref(_lib.GridConfig(16, 16, 16, 0)), 0) == _lib.FS_OK
    calls(lib)
    yield p
    lib.fake_fail(b"")
    lib.fs_context_destroy(p)
    calls(lib)


X = C.c_void_p(4096)  # "device" positions: no kernel runs


@pytest.mark.parametrize("failing", KERNELS)
def test_a_failed_launch_ends_the_build_and_the_next_one_clears_the_counts(lib, ctx, failing):
    assert lib.fs_grid_build(ctx, X, 100, 0.1, None) == _lib.FS_OK
    lines = calls(lib)
    assert launches(lines) == KERNELS and not [ln for ln in lines if ln.startswith("memset")]

    lib.fake_fail(failing.encode())
    assert lib.fs_grid_build(ctx, X, 100, 0.1, None) == _lib.FS_ERR_CUDA
    assert b"fake runtime" in lib.fs_last_error_string()
    # the launches after it would write with the offsets of the build before
    assert launches(calls(lib)) == KERNELS[:KERNELS.index(failing)]
    assert lib.fs_grid_tables(ctx, None, None, None, None, None) == _lib.FS_ERR_NOGRID

    lib.fake_fail(b"")
    for n, order in ((100, KERNELS), (0, ["k_scan"])):
        lib.fake_fail(failing.encode())
        lib.fs_grid_build(ctx, X, 100, 0.1, None)
        lib.fake_fail(b"")
        calls(lib)
        assert lib.fs_grid_build(ctx, X, n, 0.1, None) == _lib.FS_OK
        lines = calls(lib)
        first = next(k for k, ln in enumerate(lines) if ln.startswith("launch"))
        cleared = [int(ln.split()[2]) for ln in lines[:first] if ln.startswith("memset")]
        assert cleared[:2] == [4 * (16 ** 3 + 1), 4 * 2 * 8]  # every cell's count; the sums of two tiles, eight copies
        assert launches(lines) == order
    assert lib.fs_grid_build(ctx, X, 100, 0.1, None) == _lib.FS_OK
    assert not [ln for ln in calls(lib) if ln.startswith("memset")]


def test_a_refused_build_changes_nothing(lib, ctx):
    assert lib.fs_grid_build(ctx, X, 100, 0.1, None) == _lib.FS_OK
    calls(lib)
    assert lib.fs_grid_build(ctx, X, 1001, 0.1, None) == _lib.FS_ERR_CAPACITY
    assert lib.fs_grid_build(ctx, X, 100, 0.0, None) == _lib.FS_ERR_INVALID
    assert lib.fs_grid_build(ctx, None, 100, 0.1, None) == _lib.FS_ERR_INVALID
    assert calls(lib) == []
    assert lib.fs_grid_tables(ctx, None, None, None, None, None) == _lib.FS_OK


@pytest.mark.parametrize("batched", [False, True])
def test_a_new_context_waits_for_its_clearing(lib, batched):
    """The legacy stream's clears and copies: a caller's stream need not wait for them."""
    p = C.c_void_p()
    if batched:
        box = _lib.WorldBox()
        box.dims[:] = [4, 4, 4]
        rc = lib.fs_context_create_worlds(C.byref(p), 1000, C.byref(box), 1, 0)
    else:
        rc = lib.fs_context_create(C.byref(p), 1000, C.byref(_lib.GridConfig(16, 16, 16, 0)), 0)
    assert rc == _lib.FS_OK
    lines = calls(lib)
    lib.fs_context_destroy(p)
    assert [ln for ln in lines if ln.startswith("memset")] and lines[-1] == "synchronize"
