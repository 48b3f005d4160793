"""The FP64 path's integer-pipe quotient, root, halving and comparisons
(csrc/swgpu_soft64.cuh) against IEEE arithmetic, bit for bit: random
significands and exponents, significands at the ends of their range and next
to one another, exact quotients and squares, zeros, subnormals, infinities,
NaN, and quotients at both ends of the range; and h^(7/3) against numpy's pow
within the sum of the two's error bounds."""
import ctypes as C
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HARNESS = r"""
#include "swgpu_soft64.cuh"
using namespace swgpu;
__global__ void apply(const double *a, const double *b, long n, double *q, double *r, double *h,
                      double *p, int *lt) {
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    q[i] = fdiv64(a[i], b[i]);
    const Two t = div2(a[i], b[i], b[i], a[i]);
    const Three u = div3(b[i], a[i], a[i], b[i], a[i], b[i]);
    if (bits64(t.a) != bits64(q[i]) || bits64(u.b) != bits64(q[i]) ||
        bits64(u.c) != bits64(q[i]) || bits64(t.b) != bits64(u.a))
        q[i] = 12345.0;  // the three forms disagree
    r[i] = fsqrt64(a[i]);
    const Two s = sqrt2(a[i], b[i]);
    if (bits64(s.a) != bits64(r[i])) r[i] = 12345.0;
    h[i] = half_of(a[i]);
    p[i] = pow_seven_thirds(fabs(a[i]));
    lt[i] = (lt64(a[i], b[i]) ? 1 : 0) | (mag_lt(a[i], b[i]) ? 2 : 0) |
            (lt_zero(a[i]) ? 4 : 0) | (gt_zero(a[i]) ? 8 : 0) |
            (lt_pos(a[i], 1.0e-3) ? 16 : 0) | (lt64_nan(a[i], b[i]) ? 32 : 0);
}
extern "C" int run(const double *a, const double *b, long n, double *q, double *r, double *h,
                   double *p, int *lt) {
    double *d[6];
    int *dl;
    for (int i = 0; i < 6; i++)
        if (cudaMalloc(&d[i], n * 8)) return 1;
    if (cudaMalloc(&dl, n * 4)) return 1;
    cudaMemcpy(d[0], a, n * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(d[1], b, n * 8, cudaMemcpyHostToDevice);
    apply<<<(unsigned)((n + 255) / 256), 256>>>(d[0], d[1], n, d[2], d[3], d[4], d[5], dl);
    cudaMemcpy(q, d[2], n * 8, cudaMemcpyDeviceToHost);
    cudaMemcpy(r, d[3], n * 8, cudaMemcpyDeviceToHost);
    cudaMemcpy(h, d[4], n * 8, cudaMemcpyDeviceToHost);
    cudaMemcpy(p, d[5], n * 8, cudaMemcpyDeviceToHost);
    cudaMemcpy(lt, dl, n * 4, cudaMemcpyDeviceToHost);
    const int bad = cudaDeviceSynchronize() != cudaSuccess;
    for (int i = 0; i < 6; i++) cudaFree(d[i]);
    cudaFree(dl);
    return bad;
}
"""


@pytest.fixture(scope="module")
def soft64(tmp_path_factory):
    from anuga_cuda import _build as B
    d = tmp_path_factory.mktemp("soft64")
    src = d / "soft64.cu"
    src.write_text(HARNESS)
    so = str(d / "libsoft64.so")
    subprocess.run([B._nvcc()] + B.COMMON + B.UNITS["swgpu_fp64.cu"] +
                   ["-I" + B.CSRC, "-shared", str(src), "-o", so], check=True)
    lib = C.CDLL(so)
    p, ip = C.POINTER(C.c_double), C.POINTER(C.c_int)
    lib.run.argtypes = [p, p, C.c_long, p, p, p, p, ip]
    return lib


def _operands(kind, rng, n=1 << 20):
    man = lambda: rng.integers(0, 1 << 52, n, dtype=np.uint64)  # noqa: E731
    top = np.uint64((1 << 52) - 1)
    a, b = man(), man()
    exp = lambda lo, hi: rng.integers(lo, hi, n).astype(np.uint64) << np.uint64(52)  # noqa: E731
    ea, eb = exp(900, 1150), exp(900, 1150)
    if kind == "ends":
        a = np.where(rng.random(n) < 0.5, top - a % np.uint64(5), a % np.uint64(5))
        b = np.where(rng.random(n) < 0.5, top - b % np.uint64(5), b % np.uint64(5))
    elif kind == "near":
        a = (b + rng.integers(0, 7, n).astype(np.uint64)) & top
    elif kind == "exact":
        x = rng.integers(1, 1 << 26, n).astype(np.float64)
        y = rng.integers(1, 1 << 26, n).astype(np.float64)
        return np.where(rng.random(n) < 0.5, x * y, x * x), x
    elif kind == "wide":
        ea, eb = exp(0, 2048), exp(0, 2048)
        few = rng.random(n) < 0.05
        a = np.where(few, np.uint64(0), a)
        b = np.where(rng.random(n) < 0.05, np.uint64(0), b)
    sign = lambda: rng.integers(0, 2, n).astype(np.uint64) << np.uint64(63)  # noqa: E731
    return (a | ea | sign()).view(np.float64), (b | eb | sign()).view(np.float64)


@pytest.mark.parametrize("kind", ["random", "ends", "near", "exact", "wide"])
def test_soft64_is_ieee(kind, soft64):
    rng = np.random.default_rng(["random", "ends", "near", "exact", "wide"].index(kind))
    a, b = _operands(kind, rng)
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    n = len(a)
    q, r, h, p = (np.empty(n) for _ in range(4))
    lt = np.empty(n, np.int32)
    f = lambda x: x.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731
    assert soft64.run(f(a), f(b), n, f(q), f(r), f(h), f(p),
                      lt.ctypes.data_as(C.POINTER(C.c_int))) == 0
    with np.errstate(all="ignore"):
        for got, want in ((q, a / b), (r, np.sqrt(a)), (h, 0.5 * a)):
            same = (got.view(np.int64) == want.view(np.int64)) | (np.isnan(got) & np.isnan(want))
            assert same.all(), (a[~same][:3], b[~same][:3], got[~same][:3], want[~same][:3])
        # h^(7/3) within 0.52 ulp, numpy's pow within one: two units apart at most
        want = np.abs(a) ** (7.0 / 3)
        ok = (np.abs(p.view(np.int64) - want.view(np.int64)) <= 2) | (np.isnan(p) & np.isnan(want))
        assert ok.all(), (a[~ok][:3], p[~ok][:3], want[~ok][:3])
        num = ~(np.isnan(a) | np.isnan(b))
        want = ((a < b) * 1 + (np.abs(a) < np.abs(b)) * 2 + (a < 0) * 4 + (a > 0) * 8
                + (a < 1.0e-3) * 16 + (a < b) * 32)
        assert np.array_equal(lt[num], want[num])
        assert not (lt[np.isnan(a)] & 32).any()
