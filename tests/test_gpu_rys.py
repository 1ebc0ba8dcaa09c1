"""The device functions of the Rys rule (csrc/jk_device.cuh), compiled here
into a small library of their own (needs a B200)."""
import ctypes
import json
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, 'byteqc_b200', 'csrc')

SOURCE = r'''
#include "jk_device.cuh"
using namespace bqc;
// out: rsqrt_pos(x) and its square, the kernels' 1/x
__global__ void roots_kernel(const double *x, int n, double *out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        out[2 * i] = rsqrt_pos(x[i]);
        out[2 * i + 1] = out[2 * i] * out[2 * i];
    }
}
// per x: nodes and weights by rys_roots, then by rys_one (order N; 2 x 2N numbers)
template <int N>
__global__ void rys_kernel(const double *lm, const double *rows, const double *x, int n, double *out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double *o = out + (size_t)i * 4 * N;
        rys_roots<N>(lm, x[i], o, o + N);
        for (int q = 0; q < 2 * N; q++) o[2 * N + q] = rys_one<N>(rows, x[i], q);
    }
}
extern "C" int t_roots(const double *x, int n, double *out) {
    roots_kernel<<<64, 256>>>(x, n, out);
    return cudaDeviceSynchronize();
}
extern "C" int t_rys(int order, const double *x, int n, double *out) {
    const double *lm = bqc_rys_table_lm(), *rows = bqc_rys_table();
    switch (order) {
#define C(N) case N: rys_kernel<N><<<8, 128>>>(lm, rows, x, n, out); break;
        C(1) C(2) C(3) C(4) C(5) C(6) C(7)
    default: return -1;
    }
    return cudaDeviceSynchronize();
}
'''


@pytest.fixture(scope='module')
def lib(cuda, tmp_path_factory):
    from byteqc_b200 import build
    d = tmp_path_factory.mktemp('rys')
    src, so = d / 't.cu', d / 't.so'
    src.write_text(SOURCE)
    subprocess.run([build.NVCC] + build.ARCH + build.FLAGS + ['-shared', str(src), os.path.join(CSRC, 'rys_table.cu'),
                                                              '-o', str(so)], check=True)
    return ctypes.CDLL(str(so))


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def test_reciprocal_square_root(cuda, lib):
    """1/sqrt(x), and 1/x as its square, over exponent sums (1e-3 .. 1e7) and Rys
    arguments (20 .. 1e12), against 64-bit mantissas.  The last Newton step y +
    y e / 2 has a rounding of 2^-53, and half the 2^-53 of x y in e: 1.67e-16;
    the square twice that and a rounding more: 4.45e-16 (second-order terms are
    below 1e-18)."""
    import torch
    rng = np.random.default_rng(5)
    x = np.concatenate([np.exp(rng.uniform(np.log(1e-3), np.log(1e7), 200000)),
                        np.exp(rng.uniform(np.log(20.), np.log(1e12), 200000)), 4. ** np.arange(-5, 20)])
    t = torch.as_tensor(x, device=cuda)
    out = torch.zeros((len(x), 2), dtype=torch.float64, device=cuda)
    torch.cuda.synchronize()
    assert lib.t_roots(_ptr(t), len(x), _ptr(out)) == 0
    got, w = out.cpu().numpy().astype(np.longdouble), x.astype(np.longdouble)
    e_rs = float(np.abs(got[:, 0] * np.sqrt(w) - 1).max())
    e_rec = float(np.abs(got[:, 1] * w - 1).max())
    print('relative error: rsqrt %.3e, reciprocal %.3e' % (e_rs, e_rec))
    assert np.finfo(np.longdouble).nmant >= 63
    assert e_rs < 1.68e-16 and e_rec < 4.46e-16


def test_rys_functions_match_golden(cuda, lib):
    """rys_roots and rys_one on every golden record, on both sides of XMAX;
    bound as for the tables (test_rys_table.py)."""
    import torch
    golden = json.load(open(os.path.join(ROOT, 'tests', 'golden', 'rys_mpmath.json')))
    worst = 0.
    for n in sorted({g['n'] for g in golden}):
        rec = [g for g in golden if g['n'] == n]
        x = torch.tensor([float(g['x']) for g in rec], dtype=torch.float64, device=cuda)
        out = torch.zeros((len(rec), 2, 2 * n), dtype=torch.float64, device=cuda)
        torch.cuda.synchronize()
        assert lib.t_rys(n, _ptr(x), len(rec), _ptr(out)) == 0
        ref = np.array([[float(v) for v in g['r'] + g['w']] for g in rec])
        err = np.abs(out.cpu().numpy() / ref[:, None] - 1).max()
        worst = max(worst, err)
        assert err < 2e-15, (n, err)
    print('worst relative error %.2e' % worst)
