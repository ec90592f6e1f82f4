"""Arithmetic of the kernels' headers, compiled from them: exact division by multiplication, packed FP32
operations, the fast reciprocal and the pair counter."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "etherparallelparticles.jl_b200", "csrc")

SOURCE = r"""
#include "epp_pair.cuh"
using namespace epp;

__global__ void div_kernel(FastDiv f, const int* v, int* q, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) q[i] = f.div(v[i]);
}
__global__ void packed_kernel(const float* a, const float* b, unsigned* bad, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (2 * i + 1 >= n) return;
    float s0, s1, m0, m1;
    const f32x2 x = f2_pack(a[2 * i], a[2 * i + 1]), y = f2_pack(b[2 * i], b[2 * i + 1]);
    f2_unpack(f2_sub(x, y), s0, s1);
    f2_unpack(f2_mul(x, y), m0, m1);
    auto differs = [](float p, float q) { return __float_as_uint(p) != __float_as_uint(q); };
    if (differs(s0, __fsub_rn(a[2 * i], b[2 * i])) || differs(s1, __fsub_rn(a[2 * i + 1], b[2 * i + 1])) ||
        differs(m0, __fmul_rn(a[2 * i], b[2 * i])) || differs(m1, __fmul_rn(a[2 * i + 1], b[2 * i + 1])))
        atomicAdd(bad, 1u);
}
__global__ void rcp_kernel(const float* x, float* r, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) r[i] = rcp_fast(x[i]);
}
__global__ void count_kernel(const int* cnt, unsigned long long* total) { count_pairs(total, cnt[threadIdx.x]); }

static int grid(int n) { return (n + 127) / 128; }
extern "C" {
void div_host(int d, const int* v, int* q, int n) {
    FastDiv f;
    f.set(d);
    for (int i = 0; i < n; ++i) q[i] = f.div(v[i]);
}
int div_device(int d, const int* v, int* q, int n) {
    FastDiv f;
    f.set(d);
    div_kernel<<<grid(n), 128>>>(f, v, q, n);
    return (int)cudaDeviceSynchronize();
}
int packed(const float* a, const float* b, unsigned* bad, int n) {
    packed_kernel<<<grid(n / 2), 128>>>(a, b, bad, n);
    return (int)cudaDeviceSynchronize();
}
int reciprocal(const float* x, float* r, int n) {
    rcp_kernel<<<grid(n), 128>>>(x, r, n);
    return (int)cudaDeviceSynchronize();
}
int count(const int* cnt, unsigned long long* total) {
    count_kernel<<<1, 32>>>(cnt, total);
    return (int)cudaDeviceSynchronize();
}
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    d = tmp_path_factory.mktemp("arith")
    src, so = str(d / "a.cu"), str(d / "a.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.check_call([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "-Xcompiler", "-fPIC",
                           "-shared", "-I", CSRC, "-o", so, src])
    return C.CDLL(so)


def ptr(t):
    return C.c_void_p(t.ctypes.data if isinstance(t, np.ndarray) else t.data_ptr())


DIVISORS = [1, 2, 3, 7, 64, 1000, 1367, 65535, 65537, (1 << 22) + 1, (1 << 30) - 1, 1 << 30, (1 << 31) - 1]


def dividends(d):
    rng = np.random.default_rng(d)
    k = np.arange(2000, dtype=np.int64) * d
    v = np.concatenate([rng.integers(0, 1 << 31, 20000), k, k + d - 1, [0, (1 << 31) - 1]])
    return v[(v >= 0) & (v < 1 << 31)].astype(np.int32)


@pytest.mark.parametrize("d", DIVISORS)
def test_division_on_the_host(lib, d):
    v = dividends(d)
    q = np.empty_like(v)
    lib.div_host(d, ptr(v), ptr(q), len(v))
    assert np.array_equal(q, v // d)


@pytest.mark.gpu
@pytest.mark.parametrize("d", DIVISORS)
def test_division_on_the_device(lib, d):
    import torch
    v = dividends(d)
    dv = torch.from_numpy(v).cuda()
    q = torch.empty_like(dv)
    assert lib.div_device(d, ptr(dv), ptr(q), len(v)) == 0
    assert np.array_equal(q.cpu().numpy(), v // d)


# The cell lists and neighbour sets are exact because a packed operation rounds each half as the scalar one.
@pytest.mark.gpu
def test_packed_sub_and_mul_round_as_the_scalar_ones(lib):
    import torch
    rng = np.random.default_rng(9)
    n = 1 << 22
    bits = rng.integers(0, 1 << 32, (2, n), dtype=np.uint64).astype(np.uint32)
    near = np.float32(rng.uniform(-4, 4, (2, n)))
    for a, b in ((bits[0].view(np.float32), bits[1].view(np.float32)), (near[0], near[1]),
                 (near[0], near[0] * np.float32(1 + 1e-6))):
        ok = np.isfinite(a) & np.isfinite(b)   # (a NaN's bits are the hardware's own)
        a, b = (np.ascontiguousarray(np.where(ok, x, np.float32(1))) for x in (a, b))
        da, db, bad = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), torch.zeros(1, dtype=torch.int32, device="cuda")
        assert lib.packed(ptr(da), ptr(db), ptr(bad), n) == 0
        assert int(bad.item()) == 0


# rcp.approx.ftz.f32: at most 1 ulp where argument and result are normal
@pytest.mark.gpu
def test_fast_reciprocal_is_within_one_ulp(lib):
    import torch
    mant = np.arange(1 << 23, dtype=np.uint32)
    for e in (1, 60, 126, 127, 128, 200, 252):
        x = (mant | np.uint32(e << 23)).view(np.float32)
        dx = torch.from_numpy(x).cuda()
        r = torch.empty_like(dx)
        assert lib.reciprocal(ptr(dx), ptr(r), len(x)) == 0
        want = 1.0 / x.astype(np.float64)
        ulp = 2.0 ** (np.floor(np.log2(want)) - 23)
        assert np.all(np.abs(r.cpu().numpy().astype(np.float64) - want) <= ulp), e


# 32 lanes of 2^27 neighbours and more (contexts hold 2^28 particles): beyond 32 bits
@pytest.mark.gpu
@pytest.mark.parametrize("cnt", [0, 1, 65535, 65536, (1 << 27) + 3, (1 << 28) - 1])
def test_pair_counter_of_a_warp(lib, cnt):
    import torch
    c = torch.arange(32, dtype=torch.int32, device="cuda") * (1 if cnt else 0) + max(cnt - 31, 0)
    total = torch.full((1,), 5, dtype=torch.int64, device="cuda")
    assert lib.count(ptr(c), ptr(total)) == 0
    assert int(total.item()) == 5 + int(c.to(torch.int64).sum().item())
