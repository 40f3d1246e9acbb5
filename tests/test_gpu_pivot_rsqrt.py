"""The pivots' inverse square root (bl_pivot_rsqrt, bl_math.cuh) by itself, compiled with the library's flags: against
1 / sqrt(s) in 64-bit mantissas over all exponents, with mantissas next to the powers of two, the smallest normal and the
largest number among them - 1.2 ulp, from the roundings of its steps - and against CUDA's own rsqrt(); its special values; and infinite pivots in a frame."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from beamlab_b200 import build, rigs, world_from_rig
from conftest import ROOT

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "bl_math.cuh"
__global__ void k(const double* s, double* r, double* cuda, unsigned char* ok, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    bool good = true;
    r[i] = blg::bl_pivot_rsqrt(s[i], good);
    cuda[i] = rsqrt(s[i]);
    ok[i] = good;
}
extern "C" int run(const double* s, double* r, double* cuda, unsigned char* ok, int n) {
    double* d;
    unsigned char* o;
    if (cudaMalloc(&d, 24 * (size_t)n) != cudaSuccess || cudaMalloc(&o, n) != cudaSuccess) return 1;
    cudaMemcpy(d, s, 8 * (size_t)n, cudaMemcpyHostToDevice);
    k<<<(n + 255) / 256, 256>>>(d, d + n, d + 2 * (size_t)n, o, n);
    cudaMemcpy(r, d + n, 8 * (size_t)n, cudaMemcpyDeviceToHost);
    cudaMemcpy(cuda, d + 2 * (size_t)n, 8 * (size_t)n, cudaMemcpyDeviceToHost);
    cudaMemcpy(ok, o, n, cudaMemcpyDeviceToHost);
    cudaFree(d), cudaFree(o);
    return cudaGetLastError() != cudaSuccess;
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("rsqrt")
    (d / "k.cu").write_text(SOURCE)
    subprocess.run([build.nvcc(), *build.NVCC_FLAGS, "-I", f"{ROOT}/beamlab_b200/csrc", "-o", str(d / "k.so"), str(d / "k.cu")], check=True)
    lib = C.CDLL(str(d / "k.so"))

    def call(s):
        s = np.ascontiguousarray(s, np.float64)
        r, cuda, ok = np.zeros_like(s), np.zeros_like(s), np.zeros(len(s), np.uint8)
        assert lib.run(*(C.c_void_p(a.ctypes.data) for a in (s, r, cuda, ok)), len(s)) == 0
        return r, cuda, ok.astype(bool)
    return call


def test_pivot_rsqrt_within_its_bound(run):
    gen = np.random.default_rng(1)
    m = np.concatenate([gen.uniform(1.0, 2.0, 3000), 1.0 + np.arange(200) * 2.0 ** -52, 2.0 - np.arange(1, 201) * 2.0 ** -52])
    tiny, huge = np.finfo(np.float64).tiny, np.finfo(np.float64).max
    s = np.concatenate([np.ldexp(m[:, None], np.arange(-1022, 1024)[None]).ravel(), [tiny, huge, 1.0, 4.0, 0.25, np.nextafter(4.0, 0.0)]])
    s = s[(s >= tiny) & (s <= huge)]
    r, cuda, ok = run(s)
    exact = 1 / np.sqrt(s.astype(np.longdouble))
    ulp = np.abs(r.astype(np.longdouble) - exact) / np.spacing(exact.astype(np.float64))
    print("greatest error", float(ulp.max()), "ulp; CUDA's", float((np.abs(cuda.astype(np.longdouble) - exact) / np.spacing(exact.astype(np.float64))).max()))
    assert np.finfo(np.longdouble).nmant >= 63 and ok.all()
    assert ulp.max() <= 1.2
    assert np.abs(r - cuda).max() <= 0 or (np.abs(r - cuda) <= 2.2 * np.spacing(cuda)).all()


def test_pivot_rsqrt_special_values(run):
    """Not positive, not a number or subnormal: 1, and the pivot is marked; infinite: no number, which the next pivot's test or
    the block's last one marks."""
    r, _, ok = run([0.0, -0.0, -1.0, -np.inf, np.nan, 5e-324, np.nextafter(np.finfo(np.float64).tiny, 0.0), np.inf])
    assert r[:7].tolist() == [1.0] * 7 and not ok[:7].any() and np.isnan(r[7])


def test_infinite_pivots_fail_their_component():
    """Members so long and dense that their nodes' inertias overflow: the factorization fails, whichever the pivot's place, and
    the step takes the elements' forces, as at a pivot that is not positive."""
    for rails in (2, 3, 5, 9):
        section = rigs.tube_section()
        section["rho"] = 3e38
        rig = rigs.frame_ladder(rails, section=section, spacing=1e5, width=1e5)
        b = rig["bodies"][0]
        b["mass"][:], b["member_mass"][:] = 1.0, 0.5
        w = world_from_rig(rig, fem_dense_front=2)
        w.step_substeps(2)
        assert w.bodies()[0].state()["fem_failures"] == 2, rails
        w.close()
