"""The library's host code without a GPU, against a CUDA runtime in host memory
(tests/host_runtime.cpp; CPU): where device memory runs short, where sizes are
extreme, and which launches a call makes.  Kernels do nothing there; a launch that
is given a freed address is counted."""
import os
import subprocess
import sys

import pytest

from conftest import PKG, ROOT

PRELUDE = """
import ctypes, sys
sys.path.insert(0, {pkg!r})
from dgbgk import _lib
_lib.use_library({lib!r})
import numpy as np
from dgbgk import Batch, Solver, cavity_case
from dgbgk.warmstart import MLP
hr = _lib.lib()
hr.hr_limit.argtypes = hr.hr_block.argtypes = [ctypes.c_size_t]
hr.hr_block.restype = ctypes.c_void_p
hr.hr_fail_at.argtypes = [ctypes.c_long]
hr.hr_last_bad.restype = ctypes.c_char_p
def fails(f, limit):
    # f runs out of device memory in an allocation of more than limit bytes
    hr.hr_limit(limit)
    try:
        f()
    except _lib.DgbgkError as e:
        assert "out of memory" in str(e), e
    else:
        raise AssertionError("did not fail")
    finally:
        hr.hr_limit(0)
def solver(n=4, prec=64, **more):
    s = Solver.from_case(cavity_case(n, 4, 8, mach=0.3, kn=0.1), precision=prec, **more)
    s.init_case()
    return s
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    objs = [os.path.join(PKG, "_build", f"{n}.o") for n in ("dgbgk", "mlp", "plan", "setup_host")]
    cuda = "/usr/local/cuda/include"
    if not all(os.path.exists(p) for p in objs + [os.path.join(cuda, "cuda_runtime_api.h")]):
        pytest.skip("the library's objects and CUDA's headers are needed")
    lib = str(tmp_path_factory.mktemp("hr") / "libhr.so")
    gxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    r = subprocess.run([gxx, "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I", cuda, "-I",
                        os.path.join(PKG, "csrc"), "-o", lib, os.path.join(ROOT, "tests", "host_runtime.cpp")] + objs,
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def go(body):
        code = PRELUDE.format(pkg=PKG, lib=lib) + body + "\nassert hr.hr_bad() == 0, hr.hr_last_bad()\n"
        r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stderr

    return go


@pytest.mark.parametrize("prec", [64, 32])
def test_a_history_that_does_not_fit_leaves_no_freed_one_behind(run, prec):
    run(f"""
s = solver(prec={prec})
assert s.advance(1500)["steps"] == 3
for again in (1200, 1500, 4):           # within what the handle held before
    fails(lambda: s.advance(1_000_000), 4_000_000)
    assert s.advance(again)["steps"] == 3
fails(lambda: s.profile(1_000_000), 4_000_000)
s.profile(2)
assert s.macros()["rho"].size == s.NP
""")


def test_a_history_that_does_not_fit_and_a_batch(run):
    run("""
a, b = solver(), solver(5)
t = Batch([a, b])
t.advance(10)
fails(lambda: a.advance(1_000_000), 4_000_000)
t.advance(10)                           # the batch's table named the old history
fails(lambda: t.advance(1_000_000), 4_000_000)
t.advance(10)
assert a.advance(10)["steps"] == 3
""")


def test_a_shard_without_its_history_is_refused(run):
    run("""
from dgbgk.cases import gll
from dgbgk.solver import setup_mesh, vspace
c = cavity_case(4, 4, 8, mach=0.3, kn=0.1)
m = c.mesh
vc, sw = vspace(c.rorder, c.torder, *gll(c.rorder))
s = Solver(m.intma, m.coord, m.bsido, setup_mesh(m.intma, m.coord, m.bsido), vc, sw, c.rorder, c.torder, c.rv,
           rgas=c.rgas, molar_mass=c.molar_mass, diameter=c.diameter, wall_velocity=m.wall_velocity, shard=1)
L, p = _lib.lib(), ctypes.c_void_p(256)
assert L.dgbgk_shard_begin(s.h, 4, 0.0) == 0 and L.dgbgk_shard_phase(s.h, 4, p, p, p) == 0
fails(lambda: _lib.check(L.dgbgk_shard_begin(s.h, 1_000_000, 0.0)), 4_000_000)
assert L.dgbgk_shard_phase(s.h, 3, p, p, p) == _lib.DGBGK_ECUDA
assert L.dgbgk_shard_phase(s.h, 4, p, p, p) == _lib.DGBGK_ECUDA
assert L.dgbgk_shard_begin(s.h, 4, 0.0) == 0 and L.dgbgk_shard_phase(s.h, 3, p, p, p) == 0
""")


@pytest.mark.parametrize("k", [1, 2])
def test_a_training_call_that_does_not_fit_leaves_the_network_usable(run, k):
    # the k-th buffer that a longer call needs (the rows' indices, the losses)
    run(f"""
m = MLP(3, 128, 1, 128, 128, seed=1)
x, t = np.zeros((128, 3), np.float32), np.zeros((128, 128), np.float32)
m.set_data(x, t)
m.train(4)
for longer in (40, 80):
    hr.hr_fail_at({k})
    try:
        m.train(longer)
    except _lib.DgbgkError as e:
        assert "out of memory" in str(e), e
    else:
        raise AssertionError("did not fail")
    m.gradient(x, t)
    assert m.train(4).size == 4
    hr.hr_fail_at(-1)
assert m.train(40).size == 40
""")


def test_histories_of_a_call_with_a_very_large_step_limit(run):
    # rows of 8 B a step would be further apart than the largest pitch that the
    # device states for a 2-D copy
    run("""
s = solver()
r = s.advance(2 ** 28 + 1, tol=0.5)
assert r["steps"] == 3 and r["res_l2"].size == 3
assert s.advance(5)["steps"] == 3       # the handle keeps the room
""")


@pytest.mark.parametrize("n", [1, 65535, 65536, 65537, 200_000])
def test_histories_come_back_by_kind_and_step(run, n):
    # written where the sweep writes them: three values a step
    run(f"""
s = solver()
hr.hr_steps({n})
s.advance(300_000)
want = np.arange(3.0 * 300_000).reshape(-1, 3)
ctypes.memmove(hr.hr_block(want.nbytes), want.ctypes.data, want.nbytes)
r = s.advance(300_000)
assert r["steps"] == {n}
for k, name in enumerate(("res_linf", "res_l2", "dte")):
    assert np.array_equal(r[name], want[:{n}, k]), name
""")


@pytest.mark.parametrize("tune_steps", [4, 1022, 1023, 1024, 5000])
def test_the_autotuner_has_a_history_for_its_steps(run, tune_steps):
    # tune_steps timed steps after an untimed one, 24 B of history each (room
    # for 1024 steps from the start)
    run(f"""
s = solver()
Batch([s], tune_steps={tune_steps})
assert hr.hr_block(24 * max(1024, {tune_steps} + 1))
""")


@pytest.mark.parametrize("held", [True, False])
def test_an_output_ring_that_does_not_fit_is_off(run, held):
    run(f"""
s = solver()
if {held}:
    s.set_output(2, capacity=4)
s.advance(8)
fails(lambda: s.set_output(2, capacity=1_000_000), 4_000_000)
s.advance(8)
s.advance(2000)                         # the step graphs are captured anew
assert s.outputs() == []
s.set_output(2, capacity=4)
s.advance(8)
""")


@pytest.mark.parametrize("prec", [64, 32])
def test_a_re_blocking_that_does_not_fit_is_made_up_for(run, prec):
    # every allocation of a batch that re-blocks its case fails in turn; the
    # case alone and the batch that held it before go on
    run(f"""
s = solver(prec={prec})
t = Batch([s], tile_elems=64)
for k in range(1, 9):
    hr.hr_fail_at(k)
    try:
        Batch([s], tile_elems=128)
    except _lib.DgbgkError:
        pass
    hr.hr_fail_at(-1)
    if k % 2:
        s.advance(4)
        s.macros()
    t.advance(4)
    s.macros()
    s.profile(2)
""")


@pytest.mark.parametrize("sms", [8, 16, 148])
def test_launch_shapes_follow_the_device(run, sms):
    run(f"""
hr.hr_sms({sms})
# 1024 rows and 128 outputs: 16 tiles of 64 columns, or 32 of 32 where they leave SMs without one
m = MLP(3, 128, 1, 128, 1024, seed=1)
m.forward(np.zeros((1024, 3), np.float32))
narrow, wide = (hr.hr_blocks_of(b"k_gemmILi%dELi%dELi2ELi1E" % t) for t in ((32, 5), (64, 2)))
assert (narrow, wide) == ((32, 0) if 16 < {sms} else (0, 16)), (narrow, wide)
# ALPHA < 1: at most four blocks of k_wspec per SM
c = cavity_case(40, 16, 16, mach=0.3, kn=0.1)
c.alpha = 0.9
s = Solver.from_case(c)
s.init_case()
s.advance(1)
blocks = hr.hr_blocks_of(b"k_wspec")
assert 32 <= blocks <= 4 * {sms} and (blocks == 32) == ({sms} == 8), blocks
""")


@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("k,asked,tile,bufs", [(6, 64, 64, 2), (24, 64, 64, 2), (64, 64, 64, 1), (6, 128, 128, 2),
                                               (24, 128, 128, 1), (64, 128, 64, 1)])
def test_wide_halos_take_the_paths_they_are_run_for(run, k, asked, tile, bufs, prec):
    # the meshes of test_gpu_sweep_tiles.py::test_wide_halos: a 64-element tile
    # has two buffers up to a halo of 160 (162 in FP32), a 128-element one up to
    # 86 (88) and one up to 232 (235); past that 64 elements are taken
    run(f"""
sys.path[:0] = [{os.path.join(ROOT, "tests")!r}, {os.path.join(ROOT, "oracle")!r}]
from test_gpu_sweep_tiles import sheets
s = Solver.from_case(sheets(cavity_case(6, 4, 9, mach=0.3, kn=0.1), {k}), precision={prec}, tile_elems={asked})
s.init_case()
s.advance(1)
i = s.info()
assert (i["tile_elems"], hr.hr_sweep_bufs()) == ({tile}, {bufs}), (i, hr.hr_sweep_bufs())
""")


@pytest.mark.parametrize("alpha", [1.0, 0.9])
@pytest.mark.parametrize("walls", [True, False])
def test_the_profile_names_the_launches_there_are(run, alpha, walls):
    run(f"""
from dgbgk import channel_case
from dgbgk.profile import step_parts
c = channel_case(-2.0, 4.0, -2.0, 2.0, 12, 8, 8, 8, mach=2.0, kn=0.05)
c.alpha = {alpha}
if not {walls}:
    c.mesh.bsido[c.mesh.bsido[:, 3] == 4, 3] = 2
s = Solver.from_case(c)
s.init_case()
s.profile(1)
assert step_parts(c)[:3] == ["k_moments", "k_wall", "k_sweep"]
assert step_parts(c)[3] == ("k_resid" if hr.hr_blocks_of(b"7k_resid") else "gap")
""")
