"""GPU tests of the reciprocals and powers of the pair terms: the FP64 reciprocal and reciprocal square root by
themselves, over the exponent range of the pair terms and to the ends of the range, and damping exponents whose powers
leave the FP64 range, against the FP64 oracle (1e-12, the bound of the other tests)."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

import oracle_ref as O
from test_gpu_molecule_cluster import _param
from test_gpu_twobody import GTOL64, RTOL64

pytestmark = pytest.mark.gpu
CSRC = Path(__file__).resolve().parents[1] / "simple-dftd3_b200" / "csrc"

SOURCE = r"""
#include "d3_math.cuh"
__global__ void k(const double* x, double* r, double* s, int n)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    r[t] = d3::rcp_fast(x[t]);
    s[t] = d3::rsqrt_fast(x[t]);
}
extern "C" int run(const double* x, double* r, double* s, int n)
{
    double* d = nullptr;
    if (cudaMalloc(&d, 3 * sizeof(double) * n) != cudaSuccess) return 1;
    cudaMemcpy(d, x, sizeof(double) * n, cudaMemcpyHostToDevice);
    k<<<(n + 255) / 256, 256>>>(d, d + n, d + 2 * n, n);
    cudaMemcpy(r, d + n, sizeof(double) * n, cudaMemcpyDeviceToHost);
    const cudaError_t e = cudaMemcpy(s, d + 2 * n, sizeof(double) * n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e != cudaSuccess;
}
"""


def test_reciprocals(tmp_path):
    """Series error 2^-60 plus the roundings of the last product and sum: one unit in the last place for 1/x, and for
    1/sqrt(x), whose residual carries the rounding of x y as well, two."""
    (tmp_path / "r.cu").write_text(SOURCE)
    subprocess.run(["nvcc", "-shared", "-Xcompiler", "-fPIC", "-gencode", "arch=compute_100a,code=sm_100a", "-I",
                    str(CSRC), "-o", str(tmp_path / "r.so"), str(tmp_path / "r.cu")], check=True)
    lib = ctypes.CDLL(str(tmp_path / "r.so"))
    rng = np.random.default_rng(0)
    x = np.concatenate([np.exp2(rng.uniform(-40, 40, 1 << 20)), np.exp2(rng.uniform(-1021, 1021, 1 << 18)),
                        1.0 + np.arange(4096) * 2.0 ** -52, 2.0 - np.arange(1, 4096) * 2.0 ** -52])
    r, s = np.empty_like(x), np.empty_like(x)
    ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    assert lib.run(ptr(x), ptr(r), ptr(s), len(x)) == 0
    for got, exact, ulps in ((r, 1.0 / x, 1), (s, (1.0 / np.sqrt(x.astype(np.longdouble))).astype(float), 2)):
        assert np.abs(got.view(np.int64) - exact.view(np.int64)).max() <= ulps


def _system(natoms, periodic):
    from dftd3 import synthetic as S
    rng = np.random.default_rng(natoms)
    num = rng.choice([1, 6, 7, 8], size=natoms).astype(np.int32)
    side = (natoms / 0.012) ** (1 / 3) + 1.0
    return num, S.pack_box(rng, natoms, 0.0, side, 2.0), (np.eye(3) * (side + 1.5) if periodic else None)


# a cluster per molecule; the sweeps of tiles; the warps per atom of small periodic systems
@pytest.mark.parametrize("natoms, periodic", [(40, False), (300, False), (40, True), (300, True)])
@pytest.mark.parametrize("damping", ["zero", "mzero"])
def test_large_exponents(damping, natoms, periodic):
    """alp = 400: the power overflows at r = 1, not at the distances of the atoms; alp = 700: there too, where the
    energy of the pair vanishes (the oracle's gradient is 0 x inf then)."""
    from dftd3.interface import DispersionModel
    num, pos, lat = _system(natoms, periodic)
    cut = (20.0, 15.0, 15.0, 0.0, 0.0)
    for alp in (400.0, 700.0):
        param, par = _param(damping, 0.0, alp)
        model = DispersionModel(num, pos, lat, None if lat is None else np.ones(3, dtype=bool))
        model.set_realspace_cutoff(*cut)
        res = model.get_dispersion(param, grad=True)
        ref = O.dispersion(num, pos, par, lattice=lat, periodic=None if lat is None else [1, 1, 1], cutoff=cut)
        assert abs(float(res["energy"]) - ref["energy"]) <= RTOL64 * abs(ref["energy"])
        for k in ("gradient", "virial"):
            assert np.all(np.isfinite(res[k])), k
            if np.all(np.isfinite(ref[k])):
                # alp times the rounding of R0 / r in the steep part of the damping
                assert np.abs(res[k] - ref[k]).max() <= alp * GTOL64 * np.abs(ref[k]).max(), k


def test_large_exponent_in_a_batch():
    """More molecules than clusters fit: one warp per atom."""
    from dftd3.interface import BatchedDispersion
    mols = [_system(12 + k % 5, False)[:2] for k in range(140)]
    param, par = _param("zero", 0.0, 700.0)
    bat = BatchedDispersion([m[0] for m in mols], [m[1] for m in mols])
    res = bat.get_dispersion(param, grad=True)
    for k in (0, 3, 139):
        ref = O.dispersion(*mols[k], par)
        assert abs(res["energy"][k] - ref["energy"]) <= RTOL64 * abs(ref["energy"])
    assert all(np.all(np.isfinite(g)) for g in res["gradient"])
