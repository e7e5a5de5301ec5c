"""Recordings where device memory runs short: a failed allocation ends the call
it is met in and nothing after it.  The allocations fail in child processes, by
a library loaded ahead of the CUDA runtime that asks it for more than any device
has at the chosen call."""
from __future__ import annotations

import os
import subprocess
import sys
import textwrap
from pathlib import Path

import numpy as np
import pytest

from conftest import fluid_scene

pytestmark = pytest.mark.gpu

TESTS = Path(__file__).resolve().parent

SHIM = r"""
#include <dlfcn.h>
#include <stddef.h>
static long calls, fail_at;  /* the fail_at-th call from now fails; 0: none does */
static size_t above;         /* calls for more bytes than this fail; 0: none does */
static size_t total;         /* bytes asked for since */
void shim_arm(long at, size_t bytes) { calls = 0; total = 0; fail_at = at; above = bytes; }
long shim_calls(void) { return calls; }
size_t shim_bytes(void) { return total; }
int cudaMalloc(void **p, size_t bytes)
{
    static int (*real)(void **, size_t);
    if (!real) real = (int (*)(void **, size_t))dlsym(dlopen("libcudart.so.13", RTLD_LAZY), "cudaMalloc");
    ++calls;
    total += bytes;
    if (calls == fail_at || (above && bytes > above)) bytes = (size_t)1 << 50;
    return real(p, bytes);
}
"""


def run_child(tmp_path, body):
    """Runs body (python, with bp, abi, np, scenes of conftest, shim and arm(at, above)) under the shim."""
    lib = tmp_path / "shim.so"
    (tmp_path / "shim.c").write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", str(tmp_path / "shim.c"), "-o", str(lib), "-ldl"], check=True)
    head = f"""
import ctypes, sys
sys.path.insert(0, {str(TESTS)!r})
import numpy as np
from conftest import entry, fluid_scene
bp = entry.load_package()
abi = bp.abi
shim = ctypes.CDLL({str(lib)!r})
shim.shim_arm.argtypes = [ctypes.c_long, ctypes.c_size_t]
shim.shim_calls.restype = ctypes.c_long
shim.shim_bytes.restype = ctypes.c_size_t
arm = lambda at=0, above=0: shim.shim_arm(at, above)
"""
    code = textwrap.dedent(head) + textwrap.dedent(body)
    r = subprocess.run([sys.executable, "-c", code], env={**os.environ, "LD_PRELOAD": str(lib)}, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    return r.stdout


@pytest.mark.parametrize("kind", ["flag", "fluid"])
def test_gradients_after_a_failed_allocation(bp, gpu, tmp_path, kind):
    """Each allocation of a first recording fails in turn.  The call that met it
    reports it; made again, or from a new recording, the calls give the
    gradients of a solver that met no shortage."""
    out = run_child(tmp_path, f"""
        if {kind!r} == "flag":
            scene = bp.scenes.flag_scene(n=8)
            p = bp.make_params(scene, mode=abi.BP_MODE_TEXTBOOK, wind_drag=1.0, wind_lift=0.3, mass_scaling_k=0.0,
                               wind_velocity=(4.0, 0.0, 0.0),
                               stage_mask=abi.BP_STAGE_PLANES | abi.BP_STAGE_WIND | abi.BP_STAGE_DISTANCE
                               | abi.BP_STAGE_IMMOVABLE)
        else:
            scene = fluid_scene(bp, (5, 5, 5), seed=2, grid_dim=16)
            p = bp.make_params(scene, stage_mask=abi.BP_STAGE_FLUID | abi.BP_STAGE_PLANES | abi.BP_STAGE_XSPH)
        weights = np.random.default_rng(1).normal(size=(scene.num_particles, 3)).astype(np.float32)
        short = 0

        def call(f, again):
            global short
            try:
                return f()
            except Exception as e:
                assert "status 3" in str(e), e  # BP_ERR_OUT_OF_MEMORY
                short += 1
                if not again:
                    raise
                arm()
                return f()

        def record(s, again):
            s.tape_begin(2)
            for _ in range(2):
                call(lambda: s.update(2, 1.0 / 60.0, 2), again)
            g = call(lambda: s.backward(weights, 0.1 * weights), again)
            x = s.positions()
            s.tape_end()
            return dict(g, x=x)

        s = bp.ParticleSolver(scene, p)
        want = record(s, False)
        s.close()
        failed = 0
        for at in range(1, 400):
            again = at % 2 == 0  # the call made again, or a new recording
            s = bp.ParticleSolver(scene, p)
            begin = s.snapshot()
            short = 0
            arm(at)
            try:
                got = record(s, again)
            except Exception:
                arm()
                s.tape_end()
                s.restore(begin)
                got = record(s, False)
            arm()
            s.close()
            if not short:
                break
            failed += short
            for k in want:
                np.testing.assert_array_equal(got[k], want[k], err_msg=f"{{at}} {{k}}")
        assert failed == at - 1 > 40, (failed, at)
        print("failed", failed)
        """)
    assert "failed" in out


def test_a_second_end_gives_the_kept_buffers_back(bp, gpu):
    """An ended recording's buffers stay for the next one until tape_end() is
    called without a recording, which a recording after it does not notice."""
    torch, abi = gpu, bp.abi
    scene = fluid_scene(bp, (32, 32, 32), seed=2, grid_dim=32, box=(4.0, 4.0, 4.0))
    p = bp.make_params(scene, stage_mask=abi.BP_STAGE_FLUID | abi.BP_STAGE_PLANES | abi.BP_STAGE_XSPH)
    s = bp.ParticleSolver(scene, p)
    begin = s.snapshot()
    weights = np.random.default_rng(1).normal(size=(scene.num_particles, 3)).astype(np.float32)
    grads, free = [], []
    for _ in range(2):
        s.restore(begin)
        s.tape_begin(10)
        s.update(2, 1.0 / 60.0, 2)
        grads.append(s.backward(weights, 0.1 * weights))
        s.tape_end()
        free.append(torch.cuda.mem_get_info()[0])
        s.tape_end()
        free.append(torch.cuda.mem_get_info()[0])
    # the adjoint's 13 buffers of 16 bytes a particle are the least it holds
    least = 13 * 16 * scene.num_particles
    assert free[1] - free[0] >= least and free[3] - free[2] >= least, free
    for k, v in grads[0].items():
        np.testing.assert_array_equal(grads[1][k], v, err_msg=k)
    s.close()
