"""FP64 steps on values at the ends of the range that the branch-free quotients are
taken in, bit for bit against the oracle."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from tests.helpers import random_state, temporal_params

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "freeshearlayer_b200", "csrc")
PATHS = ["chosen", "ring", "ppm", "phased", "phased_ppm"]


def _step(path, p, s, n=1):
    import freeshearlayer_b200 as fsl
    from oracle import oracle as orc
    orc.build()
    p = dict(p)
    if path.endswith("ppm"):
        p["recon"] = fsl.RECON_PPM
    o = orc.Oracle(p)
    o.set_state(s)
    o.step(n)
    d = fsl.Domain(p)
    if path == "ring":
        d.tune(d.TUNE_STAGE_ROWS, 16)
    d.upload_state(s)
    (d.step_phased if path.startswith("phased") else d.step)(n)
    return d.download_state(), o.state()


def subnormal_state(p, seed, top):
    """A uniform flow in x, which stays uniform, with transverse momenta that are
    whole multiples of 2^-1074 up to `top` and the only source of themselves.  Its
    density of 6 puts some of their quotients halfway between two such multiples."""
    rng = np.random.default_rng(seed)
    L, H, D = p["LEN"], p["HIG"], p["DEP"]
    s = np.empty((L, H, 5, D))
    s[:, :, 0] = 6.0
    s[:, :, 1] = 6.0 * 120.0
    for v in (2, 3):
        m = rng.integers(0, top, (L, H, D), endpoint=True).view(np.float64)
        s[:, :, v] = np.where(rng.random((L, H, D)) < 0.5, -m, m)
    s[:, :, 4] = 1e5 / 0.4 + 0.5 * 6.0 * 120.0**2
    return s.ravel()


# within one word of the significand, and past it
@pytest.mark.parametrize("path", PATHS)
@pytest.mark.parametrize("top", [60, 2**32 + 2**20])
def test_subnormal_momenta(path, top):
    import freeshearlayer_b200 as fsl
    p = temporal_params(24, 9, 10, deltaT=1e-6, sgs=fsl.SGS_NONE)
    a, b = _step(path, p, subnormal_state(p, 3, top))
    assert np.all(np.isfinite(b))
    m = np.abs(b.reshape(24, 9, 5, 10)[:, :, 2:4])
    assert np.all(m < 2.0**-1000) and np.any(m > 0)  # still subnormal
    assert np.array_equal(a, b)


# a density unit far below and above the range the branch-free quotients are taken in
# (2^-60 .. 2^60), and units that put its ends among the densities and its upper end
# among the pressures (about 1.1e5 times them)
@pytest.mark.parametrize("path", PATHS)
@pytest.mark.parametrize("unit", [1e-30, 1e30, 2.0**-60 * 0.91, 2.0**60 * 0.91, 2.0**60 / 1.05e5])
def test_units_around_the_range(path, unit):
    p = temporal_params(13, 8, 9, deltaT=1e-6)
    p["mu_L"] *= unit  # the same flow in another unit: it stays finite
    a, b = _step(path, p, random_state(p, seed=3) * unit)
    assert np.all(np.isfinite(b))
    assert np.array_equal(a, b)


PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "fsl_phys.cuh"
using namespace fsl;
// n numerators a by m denominators b: quotients taken without a branch that differ
// from the division, and how many are taken; sixths that differ
__global__ void check(const double *a, int n, const double *b, int m, unsigned long long *out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (__double_as_longlong(sixth(a[i])) != __double_as_longlong(a[i] / 6.0)) atomicAdd(&out[2], 1ull);
    if (!zero_or_range_ok(a[i])) return;
    for (int q = 0; q < m; q++) {
        if (!range_ok(b[q]) || ones(b[q])) continue;
        const double x = quot_signed(a[i], b[q], rcp_rn(b[q])), y = a[i] / b[q];
        atomicAdd(&out[0], 1ull);
        if (__double_as_longlong(x) != __double_as_longlong(y)) atomicAdd(&out[1], 1ull);
    }
}
int main(int argc, char **argv)
{
    if (argc != 2) return 2;
    FILE *f = fopen(argv[1], "rb"); // n, m, then the values
    int nm[2];
    if (!f || fread(nm, 4, 2, f) != 2) return 3;
    std::vector<double> v(nm[0] + nm[1]);
    if (fread(v.data(), 8, v.size(), f) != v.size()) return 4;
    fclose(f);
    double *d;
    unsigned long long *o, h[3] = {0, 0, 0};
    if (cudaMalloc(&d, v.size() * 8) || cudaMalloc(&o, sizeof h)) return 5;
    cudaMemcpy(d, v.data(), v.size() * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(o, h, sizeof h, cudaMemcpyHostToDevice);
    check<<<(nm[0] + 127) / 128, 128>>>(d, nm[0], d + nm[0], nm[1], o);
    if (cudaMemcpy(h, o, sizeof h, cudaMemcpyDeviceToHost)) return 6;
    printf("%llu %llu %llu\n", h[0], h[1], h[2]);
    return 0;
}
"""


def test_quotients_by_themselves(tmp_path):
    """Numerators over the whole range, subnormals and zeros of both signs among them."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src = tmp_path / "quot.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "quot"
    subprocess.run([nvcc, "-std=c++17", "--fmad=false", "-gencode", "arch=compute_100a,code=sm_100a", "-I" + CSRC,
                    "-o", str(exe), str(src)], check=True, capture_output=True)
    rng = np.random.default_rng(7)
    tiny = np.arange(0, 4000, dtype=np.int64).view(np.float64)
    wide = rng.integers(0, 0x7FF0000000000000, 20000).view(np.float64)
    ends = np.array([2.0**k * s for k in (-1074, -1042, -1022, -959, -512, 120, 993, 1023) for s in (1, 1.5, 1 - 2.0**-53)])
    a = np.concatenate([tiny, wide, ends, [np.inf]])
    a = np.concatenate([a, -a])
    b = np.concatenate([1 + rng.random(40), 6 * 2.0 ** np.arange(-62, 58, 8), 2.0 ** rng.uniform(-61, 61, 40)])
    data = tmp_path / "values"
    data.write_bytes(np.array([len(a), len(b)], np.int32).tobytes() + a.tobytes() + b.tobytes())
    taken, wrong, sixths = map(int, subprocess.run([str(exe), str(data)], check=True, capture_output=True,
                                                   text=True).stdout.split())
    assert taken > len(a)
    assert (wrong, sixths) == (0, 0)
