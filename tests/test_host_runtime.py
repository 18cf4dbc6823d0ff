"""The library's host code against a CUDA runtime that checks it (fake_cudart.c,
preloaded into a process of its own): no GPU, kernels do nothing, and what the
host asks for is refused or noted where the real runtime would refuse it or
where it would be wrong on a machine this suite does not have."""
import os
import subprocess
import sys

import pytest

from gpumetropolis_b200.build import build, nvcc

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PREAMBLE = """
import ctypes, os
import numpy as np
from gpumetropolis_b200 import _native, workloads as W
rt = ctypes.CDLL(os.environ["LD_PRELOAD"])
rt.fake_log.restype = ctypes.c_char_p
rt.fake_pending.restype = ctypes.c_long
for f in (rt.fake_largest_block, rt.fake_live_bytes):
    f.restype = ctypes.c_size_t
rt.fake_block.restype = ctypes.c_void_p
rt.fake_block.argtypes = [ctypes.c_size_t]
def log():
    return rt.fake_log().decode().splitlines()
def wrong():
    return [l for l in log() if l.startswith("VIOLATION")]
def session(p=16, n_obs=1031, engine=0):
    w = W.make("logistic", n_obs=n_obs, p=p)
    m = w.model
    return _native.Session(m.loglik.code, m.loglik.consts, m.prior.code, m.prior.consts,
                           m.n_params, w.data, m.n_cols, w.n_obs, engine=engine)
def start(d, C, n_iter, mode=0):
    L = np.tile(0.1 * np.eye(d), (C, 1, 1)) if mode == 2 else None
    return np.zeros((C, d)), np.full((C, d), 0.1), np.ones(C), n_iter, 1, mode, 0.0, 0.0, L
"""


@pytest.fixture(scope="module")
def runtime(tmp_path_factory):
    lib = str(tmp_path_factory.mktemp("rt") / "fake_cudart.so")
    include = os.path.join(os.path.dirname(os.path.dirname(nvcc())), "include")
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", "-I", include,
                    os.path.join(ROOT, "tests", "fake_cudart.c"), "-o", lib], check=True)
    build()

    def go(text):
        env = dict(os.environ, LD_PRELOAD=lib)
        r = subprocess.run([sys.executable, "-c", PREAMBLE + text], cwd=ROOT, env=env,
                           capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    return go


def test_shared_memory_limits_of_two_sessions(runtime):
    runtime("""
a, b = session(), session()
a.loglik_batch(np.zeros((512, 17)))
b.loglik_batch(np.zeros((10, 17)))
a.loglik_batch(np.zeros((512, 17)))
""")


def test_shared_memory_limits_of_two_prepared_runs(runtime):
    runtime("""
a, b = session(p=64), session(p=54)
a.prepare(*start(65, 594, 6, 2))
b.prepare(*start(55, 594, 6, 2))
a.advance(6)
b.advance(6)
""")


def test_shared_memory_limits_beside_the_no_allocation_entry(runtime):
    # the eight-chain interpreter kernel, of programs that keep seven values
    runtime("""
from gpumetropolis_b200.dsl import gpum_model
X = [f"x{j}" for j in range(16)]
B = [f"b{j}" for j in range(16)]
text = "~ " + "+(".join(f"b{j} * x{j}" for j in range(7)) + ")" * 6
text += " + " + " + ".join(f"{b} * {x}" for b, x in zip(B[7:], X[7:]))
m = gpum_model(text, params=B, data=X)
data = np.zeros((4096, 16))
s = _native.Session(m.loglik.code, m.loglik.consts, m.prior.code, m.prior.consts, 16, data, 16,
                    4096, engine=0)
s.loglik_batch(np.zeros((512, 16)))
lib = s._lib
cols, pts, out = np.zeros((16, 4096), np.float32), np.zeros((1, 16)), np.zeros(1)
cols = cols.ravel()[(-cols.ctypes.data // 4) % 4:]
code = np.ascontiguousarray(m.loglik.code, np.uint32)
consts = np.ascontiguousarray(m.loglik.consts, np.float64)
st, err = ctypes.c_void_p(s.stream), ctypes.create_string_buffer(256)
rc = lib.gpum_b200_loglik_batch_noalloc(
    code.ctypes.data_as(ctypes.POINTER(ctypes.c_uint32)), code.size,
    consts.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), consts.size, 16,
    ctypes.c_void_p(cols.ctypes.data), 4096, 16, 4096, ctypes.c_void_p(pts.ctypes.data), 1,
    ctypes.c_void_p(out.ctypes.data), st, err, 256)
assert rc == 0, err.value
s.loglik_batch(np.zeros((512, 16)))
""")


def test_first_evaluation_has_the_geometry_of_later_ones(runtime):
    # 72 KB a CTA with the static part: three fit an SM, none before the limit is raised
    runtime("""
def grids(s):
    rt.fake_clear()
    s.loglik_batch(np.zeros((512, 17)))
    return [l for l in log() if l.startswith("launch")]
first = grids(session(n_obs=300001))
assert first == grids(session(n_obs=300001)), first
""")


def test_memory_goes_back_without_waiting_for_the_device(runtime):
    # another thread captures a graph: buffers grow with work pending, sessions
    # and surrogates come and go
    runtime("""
s = session()
net = _native.Surrogate(17, hidden=128, batch=256, seed=1)
rt.fake_capture_elsewhere(1)
s.prepare(*start(17, 8, 6))
s.advance(5)
s.prepare(*start(17, 1000, 6))
s.advance(5)
s.loglik_batch(np.zeros((5000, 17)))
net.close()
s.close()
session().close()
assert not wrong(), wrong()
assert rt.fake_live_bytes() == 0
""")


def test_memory_goes_back_to_its_own_device(runtime):
    runtime("""
s = session()
s.loglik_batch(np.zeros((10, 17)))
net = _native.Surrogate(17, hidden=128, batch=256, seed=1)
rt.fake_set_device(1)
other = session()
s.close()
net.close()
assert rt.fake_device() == 1
other.loglik_batch(np.zeros((10, 17)))
rt.fake_set_device(0)
other.close()
assert rt.fake_device() == 0
assert not wrong(), wrong()
assert rt.fake_live_bytes() == 0
""")


def test_a_refused_free_waits_for_the_owner(runtime):
    runtime("""
s = session()
s.prepare(*start(17, 8, 6))
s.advance(5)
rt.fake_fail_frees(1)
s.prepare(*start(17, 1000, 6))
s.close()
assert not wrong(), wrong()
assert rt.fake_live_bytes() == 0
""")


FETCH = """
s = session()
s.prepare(*start(17, {C}, 6))
s.advance(5)
err = ctypes.create_string_buffer(256)
draws = np.full(5 * {C} * 17, 7, np.float32)
acc, last = np.full({C}, 7, np.float32), np.full({C}, 7.0)
n = ctypes.c_uint32(99)
def fetch(*out):
    return s._lib.gpum_b200_session_fetch(s._h, *out, ctypes.byref(n), err, 256)
f32, f64 = ctypes.POINTER(ctypes.c_float), ctypes.POINTER(ctypes.c_double)
everything = [draws.ctypes.data_as(f32), acc.ctypes.data_as(f32), last.ctypes.data_as(f64)]
def fail_kernels():  # as a kernel whose wait ran out does: the session's error word
    ctypes.c_uint32.from_address(rt.fake_block(4)).value = 1
"""


def test_the_count_alone_waits_and_reports_a_failed_run(runtime):
    runtime(FETCH.format(C=8) + """
assert rt.fake_pending() > 0
assert fetch(None, None, None) == 0 and n.value == 5
assert rt.fake_pending() == 0
n.value = 99
fail_kernels()
assert fetch(None, None, None) == _native.ERR_DEVICE, err.value
assert n.value == 99
assert fetch(None, None, None) == 0 and n.value == 5
""")


@pytest.mark.parametrize("C", [8, 2000])
def test_a_failed_run_leaves_the_outputs_alone(runtime, C):
    # draws that share the pinned block, and draws of their own copy
    runtime(FETCH.format(C=C) + """
fail_kernels()
assert fetch(*everything) == _native.ERR_DEVICE, err.value
assert np.all(draws == 7) and np.all(acc == 7) and np.all(last == 7) and n.value == 99
assert fetch(*everything) == 0 and n.value == 5
assert not draws.any() and not acc.any() and not last.any()
""")


@pytest.mark.parametrize("C,arrays", [(444, 7), (445, 5), (20000, 5)])
def test_arrays_of_a_run(runtime, C, arrays):
    # states, proposals, snapshot, scales and scratch, and up to 444 chains the
    # draws made ahead: chains x 17 doubles each; five values of 8 bytes and three
    # of 4 a chain, and 16 alignments, at most beside them
    runtime(f"""
s = session()
s.prepare(*start(17, {C}, 1))
sizes = [int(l.split()[1]) for l in log() if l.startswith("allocated")]
one = {C} * 17 * 8
assert any({arrays} * one <= b < {arrays} * one + 64 * {C} + 16 * 256 for b in sizes), sizes
""")


def test_what_the_pool_keeps_serves_a_large_allocation(runtime):
    runtime("""
session().close()
rt.fake_pool_keeps_last(1)
session(p=64, n_obs=200000)  # 52 MB of data
""")


# Registers of the gradient kernels as compiled for sm_100a: one chain per lane,
# two.  With 148 and 234 two chains per lane keep eight warps on an SM (in one block
# or in two of four warps), with 113 and 196 they halve the sixteen.
@pytest.mark.parametrize("model,regs,n_obs,points,kernel", [
    ("logistic", (148, 234), 600000, 32, "gm_iter_grad"),
    ("logistic", (148, 234), 600000, 33, "gm_iter_grad2h"),
    ("logistic", (148, 234), 600000, 256, "gm_iter_grad2h"),
    ("logistic", (148, 234), 600000, 257, "gm_iter_grad2"),
    ("logistic", (148, 234), 600000, 600, "gm_iter_grad2h"),
    ("logistic", (148, 234), 600000, 2048, "gm_iter_grad2"),
    # a block per SM at most: four warps of it are slower than eight
    ("logistic", (148, 234), 3000, 256, "gm_iter_grad"),
    ("logistic", (148, 234), 3000, 1025, "gm_iter_grad"),
    ("logistic", (148, 234), 0, 300, "gm_iter_grad"),
    ("mixture", (113, 196), 600000, 300, "gm_iter_grad"),
    ("mixture", (113, 196), 600000, 2048, "gm_iter_grad"),
])
def test_choice_of_the_gradient_kernel(runtime, model, regs, n_obs, points, kernel):
    runtime(f"""
for name in ("gm_iter_grad2", "gm_iter_grad2h"):
    rt.fake_registers(name.encode(), {regs[1]})
rt.fake_registers(b"gm_iter_grad", {regs[0]})
kw = dict(p=16) if {model!r} == "logistic" else dict()
m = W.make({model!r}, n_obs=16, **kw).model
data = np.zeros(({n_obs}, m.n_cols))
s = _native.Session(m.loglik.code, m.loglik.consts, m.prior.code, m.prior.consts, m.n_params,
                    data, m.n_cols, {n_obs})
s.grad_batch(np.zeros(({points}, m.n_params)))
names = [l.split()[1] for l in log() if l.startswith("launch")]
assert [n for n in names if n.startswith("gm_iter_grad")] == [{kernel!r}], names
""")


def test_eight_warps_of_two_chains_where_two_blocks_do_not_fit(runtime):
    # 33 parameters: 67 KB of sums and 67 KB of data a block of four warps, so one
    # block an SM; a block of eight warps is as many as with one chain per lane
    runtime("""
for name in ("gm_iter_grad2", "gm_iter_grad2h"):
    rt.fake_registers(name.encode(), 242)
rt.fake_registers(b"gm_iter_grad", 254)
m = W.make("logistic", n_obs=16, p=31).model
s = _native.Session(m.loglik.code, m.loglik.consts, m.prior.code, m.prior.consts, m.n_params,
                    np.zeros((300000, m.n_cols)), m.n_cols, 300000)
for n in (200, 300, 600, 2048):
    s.grad_batch(np.zeros((n, m.n_params)))
names = [l.split()[1] for l in log() if l.startswith("launch gm_iter_grad")]
assert names == ["gm_iter_grad", "gm_iter_grad2", "gm_iter_grad", "gm_iter_grad2"], names
""")
