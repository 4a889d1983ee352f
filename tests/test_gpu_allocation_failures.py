"""A device allocation that fails, and the same call again.

A child process preloads a cudaMalloc whose n-th call fails (the runtime's own
answer to a request larger than the device).  For every n that an action
reaches, the action returns NOSH_ERR_NO_MEMORY, and done again it gives the
bits of an undisturbed run.
"""
import os
import shutil
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

CHILD = r"""
import ctypes
import sys

import numpy as np

import nosh_gb300 as ng
from nosh_gb300 import meshgen

shim = ctypes.CDLL(sys.argv[1])
shim.fail_malloc_at.argtypes = [ctypes.c_long]
shim.fail_malloc_real.argtypes = [ctypes.c_void_p]
ng.lib()
runtime = next(line.split()[-1] for line in open("/proc/self/maps") if "libcudart" in line)
shim.fail_malloc_real(ctypes.cast(ctypes.CDLL(runtime).cudaMalloc, ctypes.c_void_p))
x, cells, psi0 = meshgen.cube(8, 5)
A = meshgen.mvp_constant_curl(x)
p = {"g": 1.0, "mu": 0.3}


def handle():
    model = ng.nls(ng.mesh(x, cells), A, -1.0, 1.0, 1.0, mu=0.3, precision=ng.PREC_FP64)
    model.set_spmv_schedule(ng.SPMV_STAGED)
    return model


def setup(state):
    model = handle()
    return [model.mesh.get_edge_data()[1], model.compute_f(psi0, p)]


def newton(model):
    psi = psi0.copy()
    st = model.newton(psi, p, tol=1e-10)
    assert st["status"] == 0, st
    return [psi]


def union():
    X, C, n = np.concatenate([x, x]), np.concatenate([cells, cells + len(x)]).astype(np.int32), len(x)
    model = ng.nls(ng.mesh(X, C), meshgen.mvp_constant_curl(X), -1.0, 1.0, 1.0, mu=0.3, precision=ng.PREC_FP64)
    model.set_spmv_schedule(ng.SPMV_STAGED)
    return model, np.array([0, n, 2 * n])


def systems(state):
    model, offsets = state
    try:
        model.set_systems(offsets, np.array([0.2, 0.4]))
    except ng.NoshError:
        # the handle is still the single system that it was
        model.newton(np.concatenate([psi0, psi0]), p, tol=1e-10)
        raise
    psi = np.concatenate([psi0, psi0])
    st = model.newton(psi, p, tol=1e-10)
    assert st["status"] == 0, st
    return [psi]


def network():
    model = handle()
    return model, ng.mpnn(model)


def training(state):
    X = np.random.default_rng(1).standard_normal((state[0].mesh.num_vertices, 10)).astype(np.float32)
    return state[1].loss_grad(X, np.array([2.0, 0.5, 1.0]))


def continuation():
    model = handle()
    psi = newton(model)[0]
    go = ng.continuation(model, psi, p["mu"])
    go.learning(4, 2, 1e-3)
    for k in range(3):
        go.advance(p["mu"] + 0.01 * (k + 1))
    return go


def learning_step(go):
    # (the fourth step is the first that trains; its state stands when the
    # training after it fails, so the second try is the step after it)
    st = go.advance(go.mu + 0.01)
    return [st["status"] == 0, np.isfinite(go.last_prediction()["train_loss"])]


ACTIONS = {"setup": (lambda: None, setup), "newton": (handle, newton), "systems": (union, systems),
           "training": (network, training),
           "learning_step": (continuation, learning_step)}
prepare, act = ACTIONS[sys.argv[2]]
reference = act(prepare())
n = 0
while True:
    n += 1
    assert n < 400
    state = prepare()
    shim.fail_malloc_at(n)
    try:
        out = act(state)
        break  # no n-th allocation
    except ng.NoshError as e:
        assert e.code == ng.ERR_NO_MEMORY, (n, e.code, str(e))
    finally:
        shim.fail_malloc_at(0)
    for a, b in zip(reference, act(state)):
        assert np.array_equal(a, b), n
assert n > 1
print("failures", n - 1)
"""


def run_child(tmp_path, action):
    shim = str(tmp_path / "fail_malloc.so")
    subprocess.run([shutil.which("gcc") or "gcc", "-shared", "-fPIC", "-o", shim,
                    os.path.join(HERE, "cpp", "fail_malloc.c")], check=True)
    env = dict(os.environ, LD_PRELOAD=shim)
    r = subprocess.run([sys.executable, "-c", CHILD, shim, action], cwd=ROOT, env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "failures" in r.stdout, r.stdout + r.stderr


@pytest.mark.parametrize("action", ["setup", "newton", "systems", "training", "learning_step"])
def test_a_failed_allocation_leaves_no_trace(tmp_path, action):
    run_child(tmp_path, action)
