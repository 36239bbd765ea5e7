"""The block stage's phase factors (csrc/phasor.cuh) against FP64 sines and cosines:
phases inside a turn, at and beside the quadrants' edges, and up to the end of the
range that the reduction is exact for.  Tolerance: the bound its comment derives."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
def test_phasor(tmp_path):
    exe = str(tmp_path / "phasor_driver")
    subprocess.run([os.environ.get("NVCC", "nvcc"), "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "-I" + os.path.join(ROOT, "sfxc-1_gb300", "csrc"), os.path.join(ROOT, "tests", "phasor_driver.cu"),
                    "-o", exe], check=True)
    rng = np.random.Generator(np.random.PCG64(1))
    edges = np.arange(-16, 17, dtype=np.float32) / 4
    x = [rng.uniform(-1, 1, 1 << 20), rng.uniform(-16, 16, 1 << 18), edges, np.nextafter(edges, np.float32(99)),
         np.nextafter(edges, np.float32(-99)), [0.0, -0.0, 1e-30, -1e-20, 2.0**21 - 0.125]]
    x += [rng.uniform(-(2.0**k), 2.0**k, 1 << 12) for k in range(5, 21)]
    x = np.concatenate([np.asarray(a, dtype=np.float32) for a in x])
    x = x[:len(x) // 2 * 2]
    r = subprocess.run([exe], input=x.tobytes(), capture_output=True, check=True)
    got = np.frombuffer(r.stdout, dtype=np.float32).reshape(-1, 2).astype(np.float64)
    a = np.pi * np.fmod(x.astype(np.float64), 2.0)
    assert np.abs(got[:, 0] - np.cos(a)).max() < 1.3e-7
    assert np.abs(got[:, 1] - np.sin(a)).max() < 1.3e-7
