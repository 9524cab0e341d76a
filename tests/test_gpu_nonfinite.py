"""What is not a number stays visible: a value that has gone bad is passed on, not turned into an
ordinary one, whichever kernel takes it."""
import numpy as np
import pytest

from graphyt_gb300 import scenes

pytestmark = pytest.mark.gpu

STATE_HEADER = 88  # bytes before a saved state's first field, the offset along x of every slot


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_a_nan_offset_reaches_the_nodes(gpu_lib, tmp_path, axis):
    """A particle whose offset is NaN makes its stencil's nodes, and so its neighbours, NaN: the warp
    P2G (p2g_lanes 3) spreads it to the particles that the column kernel (9), with the weights as
    they are defined, does."""
    from graphyt_gb300 import graphyt
    sc = scenes.tiny_block(model=1, n_side=6)
    path = str(tmp_path / "s")
    bad = []
    for lanes in (9, 3):
        s = graphyt.from_scene(sc, options=dict(p2g_lanes=lanes))
        s.iterate_GPU(0.0, 0)
        s.save(path)
        state = np.fromfile(path, np.uint8)
        state[STATE_HEADER:].view(np.float32)[axis * sc.n + sc.n // 2] = np.nan
        state.tofile(path)
        s.load(path)
        assert np.isnan(s._get_particles("pos")[:, axis]).sum() == 1
        s.iterate_GPU(s.dt, 1)
        bad.append(np.isnan(s._get_particles("vel")).any(axis=1))
        s.close()
    assert bad[0].sum() > 1
    # the slots of the two handles hold the particles in the same order: one particle was hit
    assert np.array_equal(bad[0], bad[1])


ACTIVATION = r"""
#include <cuda_bf16.h>
#include "gy_silu.cuh"
__device__ unsigned short bf16(float x) { return __bfloat16_as_ushort(__float2bfloat16_rn(x)); }
// counts over every 32-bit pattern of z: [0] the activation as the layers take it, in BF16, differs
// from the division's, z >= -87; [1] the gradient's 1 / (1 + exp(-z)) does, in FP32; [2] either is off
// by more than 1.1e-36 for a finite z < -87; [3] either differs for an infinite z or NaN
__global__ void k(unsigned long long *bad)
{
    for (unsigned long long u = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; u < (1ull << 32);
         u += (unsigned long long)gridDim.x * blockDim.x) {
        const float z = __uint_as_float((unsigned)u), d = 1.0f + __expf(-z);
        const float s = z / d, g = 1.0f / d, t = gy::silu(z), h = gy::div_ge1(1.0f, d);
        if (isfinite(z) && z >= -87.0f) {
            if (bf16(s) != bf16(t)) atomicAdd(&bad[0], 1ull);
            if (__float_as_uint(g) != __float_as_uint(h)) atomicAdd(&bad[1], 1ull);
        } else if (isfinite(z)) {
            if (!(fabsf(s - t) <= 1.1e-36f) || !(fabsf(g - h) <= 1.1e-36f)) atomicAdd(&bad[2], 1ull);
        } else if (!(s == t || (isnan(s) && isnan(t))) || !(g == h || (isnan(g) && isnan(h)))) {
            atomicAdd(&bad[3], 1ull);
        }
    }
}
extern "C" int count(unsigned long long *out)
{
    unsigned long long *bad;
    if (cudaMalloc(&bad, 32) != cudaSuccess || cudaMemset(bad, 0, 32) != cudaSuccess) return 1;
    k<<<152 * 8, 256>>>(bad);
    const int rc = cudaMemcpy(out, bad, 32, cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(bad);
    return rc;
}
"""


def test_the_activation_is_the_division_it_replaces(gpu_lib, tmp_path):
    import ctypes
    import subprocess

    from graphyt_gb300 import build
    src, lib = tmp_path / "act.cu", tmp_path / "libact.so"
    src.write_text(ACTIVATION)
    subprocess.run([build.nvcc(), *build.ARCH, *build.FLAGS, "-I", build.CSRC, "-shared", str(src), "-o", str(lib)], check=True)
    bad = np.full(4, -1, np.int64)
    assert ctypes.CDLL(str(lib)).count(bad.ctypes.data_as(ctypes.c_void_p)) == 0
    assert bad.tolist() == [0, 0, 0, 0]


def test_an_infinite_activation_stays_infinite(gpu_lib):
    """First-layer biases of +inf under positive weights: every activation and output is +inf."""
    import ctypes

    import torch

    from graphyt_gb300 import _lib
    prm = torch.ones(int(gpu_lib.gy_mlp_param_count()), device="cuda")
    prm[16 * 64:16 * 64 + 64] = float("inf")
    X, Y = torch.zeros(130, 16, device="cuda"), torch.zeros(130, 7, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(gpu_lib.gy_mlp_forward(p(prm), p(X), 130, p(Y), None, stream))
    assert torch.isposinf(Y).all()
