"""The device arithmetic of a grid node's velocity (mpm_lbm_b200/csrc/grid_node.cuh),
compiled as host C++, for node masses down to the smallest number.

Tolerance: the momentum plus dt times the force, the reciprocal, their product and
the sum with dt times gravity are each rounded once, so a component is off by at
most 4 x 2^-24 of the sum of the magnitudes, and by half the smallest number over
the mass where the momentum itself is a multiple of it (given here exactly)."""

import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "grid_node.cuh"
extern "C" float host_component(float P, float m, float f, float g, float dt) {
  FsiMpmParams mp = {};
  mp.dt = dt;
  mp.bound = 0;
  return fsi::grid_node_component(P, fsi::node_mass(m), f, g, 5, 10, mp);
}
"""


@pytest.fixture(scope="module")
def component(tmp_path_factory):
    d = tmp_path_factory.mktemp("gridnode")
    (d / "m.cpp").write_text(SRC)
    so = d / "libm.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "mpm_lbm_b200", "csrc"), str(d / "m.cpp"), "-o", str(so)], check=True)
    fn = ctypes.CDLL(str(so)).host_component
    fn.argtypes, fn.restype = [ctypes.c_float] * 5, ctypes.c_float
    return fn


@pytest.mark.parametrize("exponent", [-149, -148, -140, -130, -129, -128, -127, -126, -125, -60, -20, 0, 60])
def test_velocity_of_small_masses(component, exponent):
    rng = np.random.default_rng(5)
    dt = 1e-4
    for P_of_m in (0.0, 1.0, -3.0, 0.25, rng.uniform(-2, 2)):
        for f_of_m in (0.0, 7.0):
            m = np.float32(2.0 ** exponent * (1.0 if exponent < -140 else rng.uniform(1, 2)))
            P, f = np.float32(P_of_m * float(m)), np.float32(f_of_m * float(m))
            got = component(P, m, f, -9.8, dt)
            dtf = np.float64(np.float32(dt))
            terms = np.array([float(P) / float(m), dtf * float(f) / float(m), dtf * float(np.float32(-9.8))])
            # a momentum near the smallest number 2^-149 is rounded to a multiple of it when dt f is added
            tiny = 2.0 ** -149 / float(m) if f != 0 else 0.0
            assert np.isfinite(got)
            assert abs(got - terms.sum()) <= 4 * 2.0 ** -24 * np.abs(terms).sum() + tiny
