"""The prompt epilogue's sigmoid (csrc/sigmoid.cuh) built with the host compiler, its two approximate instructions replaced by correctly rounded ones:
what is left is the error of the steps themselves."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np

CSRC = Path(__file__).resolve().parents[1] / "mistral_inference_b200" / "csrc"
SOURCE = """
#include "sigmoid.cuh"
extern "C" void run(const float* x, float* y, long long n) {
  for (long long i = 0; i < n; ++i)
    y[i] = mb200::sigmoid_by(x[i], [](float v) { return (float)std::exp2((double)v); }, [](float v) { return (float)(1.0 / (double)v); });
}
"""


def test_sigmoid_is_exact_to_a_few_ulps_over_its_whole_range(tmp_path):
    """Four roundings of 2^-24 (the correction, 1 + e, ex2, rcp) and what the fp32 tail of log2(e) leaves (2^-49 x): within 2^-22 of float64 down to
    e^-x = 2^126, and within the spacing of subnormal numbers (2^-149) below."""
    (tmp_path / "s.cc").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-shared", "-fPIC", "-I", str(CSRC), "-o", str(tmp_path / "s.so"), str(tmp_path / "s.cc")], check=True)
    lib = ctypes.CDLL(str(tmp_path / "s.so"))
    x = np.concatenate([np.linspace(-130, 130, 1_000_001), -np.geomspace(1e-30, 130, 100_000), np.geomspace(1e-30, 130, 100_000), [0.0, -0.0]]).astype(np.float32)
    y = np.empty_like(x)
    lib.run(x.ctypes.data_as(ctypes.c_void_p), y.ctypes.data_as(ctypes.c_void_p), ctypes.c_longlong(len(x)))
    ref = 1 / (1 + np.exp(-x.astype(np.float64)))
    err = np.abs(y.astype(np.float64) - ref)
    normal = x > -87.3
    assert (err[normal] / ref[normal]).max() < 2.0 ** -22
    assert err[~normal].max() <= 2.0 ** -126 * 2.0 ** -22 + 2.0 ** -149 + np.where(x < -88.72, ref, 0).max()
    assert (y[x < -88.8] == 0).all() and (y[x > 20] == 1).all()
    odd = np.array([np.inf, -np.inf, np.nan], dtype=np.float32)
    out = np.empty_like(odd)
    lib.run(odd.ctypes.data_as(ctypes.c_void_p), out.ctypes.data_as(ctypes.c_void_p), ctypes.c_longlong(3))
    assert out[0] == 1 and out[1] == 0
