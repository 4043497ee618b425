"""Stream operations of the library over a fake CUDA runtime that logs them and
fails one of them (CPU).

An evaluation that ends early, because one of its launches failed, does not
reach into the next one. The accumulators, the tile counts and the charge mesh are zero between
evaluations. After a failed launch the caller's stream first waits for the
kernels already launched on the second stream, then clears the three; the next
evaluation is launched as if nothing had happened. When the clear fails too, the
next evaluation starts with it.

A plan that fails (allocations, sizes) leaves nothing that a later call launches
over: contexts plan again, a failed autotuning goes back to the plan it came
with, and where that fails too every call is refused.

A list build and its set-up (first build, another capacity, another radius) do
everything on the caller's stream.
"""
import ctypes
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CUDA = "/usr/local/cuda/include"

MESH, N = 16, 64


def _libs():
    from esp_hoomd_b200 import _lib
    lib = _lib.get_lib()
    fake = ctypes.CDLL(None)
    fake.fake_log.restype = ctypes.c_char_p
    fake.fake_reset.argtypes = [ctypes.c_long, ctypes.c_long]
    return _lib, lib, fake


def _child_lists():
    _lib, lib, fake = _libs()
    p = _lib.EspParams()
    assert lib.esp_params_default(ctypes.byref(p)) == 0
    p.nx = p.ny = p.nz = MESH
    n = (ctypes.c_int * 2)(N, N)
    boxes = (ctypes.c_double * 6)(*[10.0] * 6)
    b = ctypes.c_void_p()
    assert lib.esp_batch_create(ctypes.byref(p), 2, n, boxes, None, ctypes.byref(b)) == 0, lib.esp_last_error()
    buf = (ctypes.c_double * (64 * N)).from_buffer(bytearray(8 * 64 * N))
    ptr = ctypes.addressof(buf)
    stream = 4711
    for rlist, cap in ((3.0, 8), (3.0, 16), (3.4, 16), (3.4, 16)):
        for build in (lambda: lib.esp_batch_build_nlist(b, stream, ptr, rlist, cap, ptr, ptr, ptr),
                      lambda: lib.esp_batch_build_pairlist(b, stream, ptr, rlist, cap)):
            fake.fake_reset(-1, -1)
            assert build() == 0, lib.esp_last_error()
            ops = [line.split(" ", 2) for line in fake.fake_log().decode().splitlines()]
            assert len(ops) > 5 and {o[1] for o in ops} == {str(stream)}, ops
    lib.esp_batch_destroy(b)
    print("ok")


def _child_plans():
    _lib, lib, fake = _libs()
    fake.fake_fail_mallocs.argtypes = [ctypes.c_long, ctypes.c_long]
    p = _lib.EspParams()
    assert lib.esp_params_default(ctypes.byref(p)) == 0
    p.nx = p.ny = p.nz = MESH
    buf = (ctypes.c_double * (64 * N)).from_buffer(bytearray(8 * 64 * N))
    ptr = ctypes.addressof(buf)
    forever = 1 << 40

    def launches():
        return sum(line.split(" ")[0] == "launch" for line in fake.fake_log().decode().splitlines())

    # a context whose plan for a new particle count fails plans again at the next call
    h = ctypes.c_void_p()
    assert lib.esp_create(ctypes.byref(p), 10.0, 10.0, 10.0, N, ctypes.byref(h)) == 0
    compute = lambda n: lib.esp_compute(h, None, ptr, ptr, n, ptr, ptr, ptr, ptr, None, None, 3)  # noqa: E731
    assert compute(N) == 0
    fake.fake_fail_mallocs(5, forever)
    fake.fake_reset(-1, -1)
    assert [compute(N // 2), compute(N // 2)] == [-3, -3]
    assert lib.esp_get_sort(h, None, ptr, ptr) == -1 and lib.esp_get_potential(h, None, ptr) == -1
    assert compute(1 << 26) == -4 and compute(1 << 26) == -4  # too many particles
    assert launches() == 0
    fake.fake_fail_mallocs(-1, -1)
    assert compute(N // 2) == 0 and compute(N) == 0
    lib.esp_destroy(h)
    # autotuning: the k-th allocation fails alone, then everything from it on
    n = (ctypes.c_int * 1)(N)
    box = (ctypes.c_double * 3)(10.0, 10.0, 10.0)
    b = ctypes.c_void_p()
    assert lib.esp_batch_create(ctypes.byref(p), 1, n, box, None, ctypes.byref(b)) == 0
    tune = lambda: lib.esp_batch_autotune(b, None, ptr, ptr, ptr, ptr, ptr, 3, 1, None, None, 0)  # noqa: E731
    calls = [lambda: lib.esp_batch_compute(b, None, ptr, ptr, ptr, ptr, ptr, ptr, None, None, 3),
             lambda: lib.esp_batch_build_nlist(b, None, ptr, 3.0, 8, ptr, ptr, ptr),
             lambda: lib.esp_batch_build_pairlist(b, None, ptr, 3.0, 8),
             lambda: lib.esp_batch_nve_step1(b, None, ptr, ptr, ptr, 0.1),
             lambda: lib.esp_batch_nve_step2(b, None, ptr, ptr, ptr, 0.1),
             lambda: lib.esp_batch_lj(b, None, ptr, ptr, ptr, ptr, 1.0, 1.0, 2.5, ptr, None),
             lambda: lib.esp_batch_md_run(b, None, ptr, ptr, ptr, ptr, ptr, ptr, ptr, None, None, 1, 0.1, 0)]
    fake.fake_fail_mallocs(-1, -1)
    assert tune() == 0 and [c() for c in calls] == [0] * 7
    for k in (2, 9, 40, 60):  # the trial's outputs and plans
        fake.fake_fail_mallocs(k, k + 1)
        assert tune() == -3
        fake.fake_fail_mallocs(-1, -1)
        assert [c() for c in calls] == [0] * 7, k
    fake.fake_fail_mallocs(9, forever)
    assert tune() == -3
    fake.fake_reset(-1, -1)
    assert [c() for c in calls] == [-1] * 7 and launches() == 0
    fake.fake_fail_mallocs(-1, -1)
    assert tune() == 0 and [c() for c in calls] == [0] * 7
    lib.esp_batch_destroy(b)
    print("ok")


def _child():
    _lib, lib, fake = _libs()
    buf = [(ctypes.c_double * (8 * N)).from_buffer(bytearray(64 * N)) for _ in range(8)]
    pos, q, head, nn, nl, force = (ctypes.addressof(b) for b in buf[:6])

    def log():
        return [tuple(line.split(" ", 2)) for line in fake.fake_log().decode().splitlines()]

    for precision in (0, 1):
        p = _lib.EspParams()
        assert lib.esp_params_default(ctypes.byref(p)) == 0
        p.nx = p.ny = p.nz = MESH
        p.precision = precision
        h = ctypes.c_void_p()
        assert lib.esp_create(ctypes.byref(p), 10.0, 10.0, 10.0, N, ctypes.byref(h)) == 0, lib.esp_last_error()
        compute = lib.esp_compute_f64 if precision else lib.esp_compute

        def run(flags, fail_launch=-1, fail_memset=-1):
            fake.fake_reset(fail_launch, fail_memset)
            rc = compute(h, None, pos, q, N, head, nn, nl, force, None, None, flags)
            return rc, log()

        clears = [str(24 * 8), str(((MESH + 8) // 9) ** 3 * 4), str(MESH ** 3 * 8)]  # 9: the tile edge of support 8
        for flags in (_lib.ESP_ALL, _lib.ESP_LONG_RANGE, _lib.ESP_SHORT_RANGE):
            rc, good = run(flags)
            assert rc == 0
            n = sum(o[0] == "launch" for o in good)
            forks = {o[1] for o in good if o[0] == "wait"} - {"0"}
            assert n >= 3 and len(forks) == (flags == _lib.ESP_ALL)
            for k in range(n):
                rc, ops = run(flags, k)
                assert rc == -2 and b"fake error" in lib.esp_last_error()
                at = [o[0] for o in ops].index("fail")
                forked = [o[1] for o in ops if o[0] == "wait" and o[1] != "0"]
                tail = ops[-3 - 2 * len(forked):]
                assert at < len(ops) - len(tail) and not any(o[0] == "launch" for o in tail)
                if forked:  # the caller's stream waits for what the second stream holds
                    assert tail[0][:2] == ("record", forked[0]) and tail[1] == ("wait", "0", tail[0][2])
                assert [o for o in tail if o[0] == "memset"] == [("memset", "0", c) for c in clears]
                assert run(flags) == (0, good)
            # the clear fails as well: the next evaluation starts with it
            memsets = sum(o[0] == "memset" for o in run(flags, 1)[1])
            rc, _ = run(flags, 1, memsets - 1)
            assert rc == -2 and b"fake error" in lib.esp_last_error()
            rc, ops = run(flags)
            assert rc == 0 and ops[-len(good):] == good
            assert [o for o in ops[:-len(good)] if o[0] == "memset"] == [("memset", "0", c) for c in clears]
            assert run(flags) == (0, good)
        lib.esp_destroy(h)
    print("ok")


def _run(tmp_path, which):
    if not os.path.exists(os.path.join(CUDA, "cuda_runtime.h")):
        pytest.skip("needs the CUDA headers")
    so = str(tmp_path / "libfake_cudart.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I" + CUDA,
                    os.path.join(HERE, "fake_cudart.cpp"), "-o", so], check=True)
    env = dict(os.environ, LD_PRELOAD=so, PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, os.path.abspath(__file__), which], env=env, cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


def test_failed_launch_leaves_clear_state(tmp_path):
    _run(tmp_path, "launches")


def test_list_builds_keep_to_their_stream(tmp_path):
    _run(tmp_path, "lists")


def test_failed_plans_are_not_used(tmp_path):
    _run(tmp_path, "plans")


if __name__ == "__main__":
    {"lists": _child_lists, "plans": _child_plans, "launches": _child}[sys.argv[1]]()
