"""The 4-wide nodes as the device fills them (quantise.cuh): every decoded child
box holds its exact box with the room that the walks' rounding needs, unused
slots carry the value that rejects them, and what cannot be quantised is
refused.  The header is compiled into a small kernel of the test; the planes
are decoded here in 64 bits, where they are exact, so the tolerance is zero."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "aviatorengine2_b200", "csrc")
SOURCE = r"""
#include <cstdint>
#include "context.h"
#include "quantise.cuh"
__global__ void k_nodes(const float *box, const int *kids, const uint8_t *valid, int n, ae::QNode *out, uint8_t *good) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float b[4][6], u[6];
    bool v[4];
    for (int k = 0; k < 4; k++) {
        v[k] = valid[4 * i + k] != 0;
        for (int a = 0; a < 6; a++) b[k][a] = box[24 * i + 6 * k + a];
    }
    ae::QNode q;
    good[i] = ae::quantise_node(q, kids[i], b, v, u);
    out[i] = q;
}
extern "C" int run(const float *box, const int *kids, const uint8_t *valid, int n, void *out, uint8_t *good) {
    float *b; int *k; uint8_t *v, *g; ae::QNode *q;
    if (cudaMalloc(&b, n * 96) || cudaMalloc(&k, n * 4) || cudaMalloc(&v, n * 4) || cudaMalloc(&g, n) || cudaMalloc(&q, n * 64)) return 1;
    cudaMemcpy(b, box, n * 96, cudaMemcpyHostToDevice);
    cudaMemcpy(k, kids, n * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(v, valid, n * 4, cudaMemcpyHostToDevice);
    cudaMemset(q, 0, n * 64);
    k_nodes<<<(n + 127) / 128, 128>>>(b, k, v, n, q, g);
    cudaMemcpy(out, q, n * 64, cudaMemcpyDeviceToHost);
    cudaMemcpy(good, g, n, cudaMemcpyDeviceToHost);
    const int e = int(cudaGetLastError());
    cudaFree(b); cudaFree(k); cudaFree(v); cudaFree(g); cudaFree(q);
    return e;
}
"""
ROOM = 2.0 ** -19


@pytest.fixture(scope="module")
def quantise(tmp_path_factory):
    d = tmp_path_factory.mktemp("nodes")
    (d / "nodes.cu").write_text(SOURCE)
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.check_call([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                           "--expt-relaxed-constexpr", "-I" + CSRC, str(d / "nodes.cu"), "-o", str(d / "nodes.so")])
    lib = ctypes.CDLL(str(d / "nodes.so"))

    def run(boxes, kids, valid):
        n = len(boxes)
        boxes, kids = np.ascontiguousarray(boxes, np.float32), np.ascontiguousarray(kids, np.int32)
        valid = np.ascontiguousarray(valid, np.uint8)
        out, good = np.zeros((n, 64), np.uint8), np.zeros(n, np.uint8)
        p = lambda a: ctypes.c_void_p(a.ctypes.data)  # noqa: E731
        assert lib.run(p(boxes), p(kids), p(valid), n, p(out), p(good)) == 0
        org = out[:, :12].copy().view(np.float32).astype(np.float64)
        e = out[:, 12:15].astype(int) - 127
        return org, e, out[:, 16:48].reshape(n, 4, 8), good.astype(bool)
    return run


def plane(q):
    q = q.astype(np.float64)
    return np.where(q < 128, 2.0 + q / 64.0, 4.0 + (q - 128.0) / 32.0)


@pytest.mark.parametrize("extent,at", [(1.0, 0.0), (1e-3, 0.0), (100.0, 37.3), (1.0, 1000.0), (1e-6, 100.0), (3e4, -1e4),
                                       (1e-30, 0.0), (1e30, 0.0), (0.0, 5.0)])
def test_decoded_boxes_hold_the_exact_ones(quantise, extent, at):
    rng = np.random.default_rng(11)
    n = 20_000
    c = rng.uniform(0, 1, (n, 4, 2, 3))
    # Shared faces, flat boxes and planes on the grid among them.
    c = np.where(rng.random((n, 4, 2, 3)) < 0.3, np.round(c * 8) / 8, c)
    c[:, :, 1] = np.where(rng.random((n, 4, 3)) < 0.2, c[:, :, 0], c[:, :, 1])
    c = (c * extent + at).astype(np.float32)
    boxes = np.concatenate([c.min(2), c.max(2)], 2)
    kids = rng.integers(2, 5, n)
    valid = rng.random((n, 4)) < 0.9
    org, e, planes, good = quantise(boxes, kids, valid)
    use = valid & (np.arange(4) < kids[:, None])
    assert good.all()
    assert (planes[..., 6:].reshape(-1, 2)[use.ravel()] == [0x00, 0xC0]).all()
    assert (planes[..., 4:].reshape(-1, 4)[~use.ravel()] == [0x00, 0x00, 0x80, 0x7F]).all()
    s = np.ldexp(1.0, e)[:, None, :]
    lo = org[:, None, :] + plane(planes[..., 0:3]) * s
    hi = org[:, None, :] + plane(planes[..., 3:6]) * s
    # In units of the scale, where the room is stated; the sums of 64-bit values
    # round by 2^-53 of the coordinates, 2^-32 of a scale at most.
    slack = ROOM - 2.0 ** -30
    b = boxes.astype(np.float64)
    assert (((b[..., :3] - lo) / s)[use] >= slack).all()
    assert (((hi - b[..., 3:]) / s)[use] >= slack).all()


def test_what_cannot_be_quantised(quantise):
    inf, big = np.float32(np.inf), np.float32(3e38)
    boxes = np.zeros((4, 4, 6), np.float32)
    boxes[..., 3:] = 1.0
    boxes[0, 1, 3] = inf
    boxes[1, 0, :3], boxes[1, 1, 3:] = -big, big
    boxes[2, 2, 0] = inf  # not among the valid ones
    valid = np.ones((4, 4), bool)
    valid[2, 2] = False
    valid[3] = False
    _, _, planes, good = quantise(boxes, np.full(4, 4), valid)
    assert good.tolist() == [False, False, True, True]
    for node in (0, 1, 3):
        assert (planes[node, :, 4:] == [0x00, 0x00, 0x80, 0x7F]).all()
