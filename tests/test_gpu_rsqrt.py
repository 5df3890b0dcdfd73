"""The FP64 reciprocal square root of the plain form's walks (rsqrt_step): its stated error, and a pair
whose argument it is not made for."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from oracle import oracle as O
from tholedipoleplugin_b200 import build as B
from tholedipoleplugin_b200 import systems as S
from tholedipoleplugin_b200.kernel import CudaCalcTholeDipoleForceKernel

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "tdp_pairs.cuh"
__global__ void k(int n, const double* x, double* y) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = tdp::rsqrt_step(x[i]);
}
extern "C" int run(int n, const double* x, double* y) {
    double* d = nullptr;
    if (cudaMalloc((void**)&d, 2 * n * sizeof(double)) != cudaSuccess) return 1;
    cudaMemcpy(d, x, n * sizeof(double), cudaMemcpyHostToDevice);
    k<<<(n + 127) / 128, 128>>>(n, d, d + n);
    const int rc = cudaMemcpy(y, d + n, n * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(d);
    return rc;
}
"""


def test_error(tmp_path):
    """Half an ulp (2^-53 relative at most) and 3e-20, over both parities of the exponent and the arguments
    that the walks have: squared distances of 1e-6 to 1e4 nm^2, rho^2 from 2e-10, and far beyond either."""
    src, lib = tmp_path / "rsqrt.cu", tmp_path / "rsqrt.so"
    src.write_text(SOURCE)
    subprocess.run([B.nvcc(), "-std=c++17", "-O3", *B.ARCH, "-ftz=true", "-shared", "-Xcompiler", "-fPIC", "-I", B.CSRC,
                    "-o", str(lib), str(src)], check=True)
    rng = np.random.default_rng(3)
    m = np.concatenate([1.0 + rng.random(20000), 1.0 + 2.0 ** -rng.integers(1, 53, 400),
                        2.0 - 2.0 ** -rng.integers(0, 52, 400)])
    x = np.concatenate([np.ldexp(m, e) for e in [*range(-34, 16), -1022, -1021, -501, 500, 1022]])
    y = np.zeros_like(x)
    p = C.POINTER(C.c_double)
    assert C.CDLL(str(lib)).run(len(x), x.ctypes.data_as(p), y.ctypes.data_as(p)) == 0
    ref = np.longdouble(1.0) / np.sqrt(x.astype(np.longdouble))
    assert np.finfo(np.longdouble).eps < 2e-19
    assert float(np.max(np.abs(y - ref) / ref)) < 1.12e-16


@pytest.mark.parametrize("offset", [1e-155, 1e-160, 1e-161])
def test_pair_whose_yz_distance_squared_is_subnormal(offset):
    """Two atoms 5 nm apart along x, in different tiles, whose y differ by so little that the square is
    subnormal: the frame's X is -y for them as for 1e-6 nm (a difference of 1e-6 / 5 of their forces)."""
    n = 64
    rng = np.random.default_rng(1)
    pos = rng.uniform(0.0, 1.0, (n, 3)) * [0.3, 3.0, 3.0] + [0.0, 0.2, 0.2]
    pos[32:, 0] += 5.0
    pos[0] = [0.0, 0.0, 0.0]
    axis = np.full((n, 4), -1, dtype=np.int32)
    axis[:, 0] = S.NOAXISTYPE
    charges, dipoles = rng.permutation(np.resize([0.4, -0.4], n)), rng.normal(scale=0.01, size=(n, 3))
    forces = []
    for y in (offset, 1e-6):
        pos[40] = [5.0, y, 0.0]
        s = S.TholeSystem(positions=pos.copy(), charges=charges, dipoles=dipoles,
                          polarizabilities=np.full(n, 1e-4), tholes=np.full(n, 0.3), axis=axis,
                          cov12=[[] for _ in range(n)], cov13=[[] for _ in range(n)], polarization=S.DIRECT)
        with CudaCalcTholeDipoleForceKernel(s, precision="double") as k:
            forces.append(k.execute(s.positions)[1])
    assert np.all(np.isfinite(forces[0]))
    assert np.abs(forces[0] - forces[1]).max() < 1e-5 * np.abs(forces[1]).max()
    ref = O.compute(s, "port").forces
    assert np.abs(forces[1] - ref).max() < 1e-9 * np.abs(ref).max()
