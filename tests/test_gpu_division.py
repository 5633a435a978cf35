"""recip() and quot() (csrc/wq3d_models.cuh) give the bits of "/" over the
whole of their stated ranges, and what is built on them (the Rayleigh loss,
the ray derivatives) the bits of the plain form.  A test kernel compiled here
compares both on the device.  Nothing is rounded differently on either side,
so no tolerance is needed."""
import ctypes as C
import subprocess

import pytest

from underseamodelinglibrary_b200 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cuda_runtime.h>
#include "wq3d_models.cuh"
using namespace wq3d;
typedef unsigned long long u64;

/* splitmix64 (S. Vigna) */
__device__ u64 mix(u64 x) {
    x += 0x9e3779b97f4a7c15ull;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    return x ^ (x >> 31);
}
__device__ double unit(u64 h) { return (double)(h >> 11) * 0x1p-53; }
__device__ double bits(u64 m, int e, int sign) { /* +-1.m x 2^e */
    return __longlong_as_double((m & 0xfffffffffffffull) | ((u64)(e + 1023) << 52) | ((u64)sign << 63));
}
__device__ bool differ(double x, double y) { return __double_as_longlong(x) != __double_as_longlong(y); }
/* significands beside the ends and with long runs of ones and zeros */
__device__ u64 edge(int k) {
    switch (k & 15) {
        case 0: return 0;
        case 1: return 1;
        case 2: return 2;
        case 3: return 0xfffffffffffffull;
        case 4: return 0xffffffffffffeull;
        case 5: return 0xffffffffffffdull;
        case 6: return 0xfffff00000000ull;
        case 7: return 0xfffff00000001ull;
        case 8: return 0x00000ffffffffull;
        case 9: return 0x00000fffffffeull;
        case 10: return 0x8000000000000ull;
        case 11: return 0x7ffffffffffffull;
        case 12: return 0xfffffefffffffull;
        case 13: return 0x5555555555555ull;
        case 14: return 0xaaaaaaaaaaaaaull;
        default: return 0x0000100000000ull;
    }
}

__device__ void tally(u64* out, bool tried, bool wrong) {
    if (tried) atomicAdd(out, 1ull);
    if (tried && wrong) atomicAdd(out + 1, 1ull);
}

/* random operands over the whole ranges; out: compared, different, refused */
__global__ void k_random(u64 n, u64* out) {
    u64 tried = 0, wrong = 0, refused = 0;
    for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
        const u64 h = mix(i), g = mix(h);
        const double b = bits(g, (int)(mix(g) % 1000) - 500, (int)(h & 1));
        const double a = bits(h >> 8, (int)(mix(h + 1) % 799) - 399, (int)(h >> 1 & 1));
        if (!divisor_ok(b) || !dividend_ok(a)) {
            ++refused;
            continue;
        }
        ++tried;
        wrong += differ(quot(a, recip(b)), a / b) || differ(recip(b).y, 1.0 / b);
    }
    atomicAdd(out, tried);
    atomicAdd(out + 1, wrong);
    atomicAdd(out + 2, refused);
}

/* The hardest quotients: b = B and a = A x 2^54 with A, B whole, so that
 * M B = A 2^54 + r with an odd M of 54 bits, half way between two quotients,
 * and a small r: a / b misses the midpoint M by r / B. */
__global__ void k_midpoint(u64 n, u64* out) {
    u64 tried = 0, wrong = 0;
    for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
        const u64 h = mix(i ^ 0x5bd1e995ull);
        const u64 B = (h & 0xfffffffffffffull) | 0x10000000000000ull | 1;
        u64 inv = B; /* of B modulo 2^64, five bits of which are right at first */
        for (int k = 0; k < 6; ++k) inv *= 2 - B * inv;
        const long long r = 2 * (long long)(mix(h) % 16) - 15;
        const u64 M = ((u64)r * inv) & 0x3fffffffffffffull;
        if (!(M >> 53)) continue;
        /* A = (M B - r) / 2^54 */
        u64 lo = M * B, hi = __umul64hi(M, B);
        const u64 l2 = lo - (u64)r;
        hi -= r >= 0 ? (lo < (u64)r) : -(long long)(l2 < lo);
        lo = l2;
        const u64 A = (hi << 10) | (lo >> 54);
        if (lo << 10 || A >> 53 || !A) continue;
        const int e = (int)(mix(h + 2) % 601) - 300;
        const double b = ldexp((double)B, e), a = (double)A;
        if (!divisor_ok(b)) continue;
        ++tried;
        wrong += differ(quot(a, recip(b)), a / b) || differ(recip(b).y, 1.0 / b);
    }
    atomicAdd(out, tried);
    atomicAdd(out + 1, wrong);
}

/* every pair of edge significands with exponents at the ends of the ranges,
 * either sign, and dividends of either zero */
__global__ void k_edges(u64* out) {
    const int eb[] = {-501, -500, -1, 0, 1, 498, 499, 500}, ea[] = {-401, -400, -399, 0, 398, 399, 400};
    const int i = threadIdx.x; /* 16 x 16 significands */
    for (int p = 0; p < 8; ++p)
        for (int q = 0; q < 9; ++q)
            for (int s = 0; s < 4; ++s) {
                const double b = bits(edge(i >> 4), eb[p], s & 1);
                const double a = q < 7 ? bits(edge(i), ea[q], s >> 1) : (s >> 1) ? -0.0 : 0.0;
                const bool ok = divisor_ok(b) && dividend_ok(a);
                tally(out, ok, ok && (differ(quot(a, recip(b)), a / b) || differ(recip(b).y, 1.0 / b)));
                /* what must be refused: exponents beyond the ends, a low word of ones, zero,
                 * infinities, NaN, and dividends beyond theirs */
                const bool in_b = eb[p] >= -500 && eb[p] < 500 && (unsigned)(edge(i >> 4)) != 0xffffffffu;
                const bool in_a = q >= 7 || (ea[q] >= -400 && ea[q] < 400) || (ea[q] == 400 && edge(i) == 0);
                tally(out + 2, true, divisor_ok(b) != in_b || dividend_ok(a) != in_a);
            }
    const double none[] = {0.0, -0.0, INFINITY, -INFINITY, NAN, 5e-324, -1e-310, 1.7976931348623157e308};
    tally(out + 2, i < 8, divisor_ok(none[i & 7]));
    tally(out + 2, i < 8, dividend_ok(none[i & 7]) != ((i & 7) < 2));
    tally(out + 2, true, divisor_ok_positive(bits(edge(i), 0, 1)) ||
                             divisor_ok_positive(bits(edge(i), 0, 0)) != divisor_ok(bits(edge(i), 0, 0)));
}

/* largest relative error of the seed, in units of 2^-40 */
__global__ void k_seed(u64 n, u64* out) {
    u64 worst = 0;
    for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
        const double b = bits(mix(i), (int)(i % 1000) - 500, (int)(i & 1));
        double y;
        asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
        worst = max(worst, (u64)(fabs(fma(-b, y, 1.0)) * 0x1p40));
    }
    atomicMax(out, worst);
}

/* the Rayleigh loss at n grazing angles over -pi/2 .. pi/2, ends and zero included */
__global__ void k_rayleigh(LossDev L, u64 n, u64* out) {
    LossDev P = L;
    P.rl_fast = 0;
    for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
        double x = M_PI * ((double)i / (double)(n - 1) - 0.5);
        if (i & 1) x += (unit(mix(i)) - 0.5) * 1e-6;
        double a0, p0, a1, p1, a2, p2;
        reflect_loss_scalar(P, x, &a0, &p0);
        reflect_loss_scalar(L, x, &a1, &p1);
        tally(out, true, differ(a0, a1) || differ(p0, p1));
        tally(out + 2, reflect_loss_rayleigh_fast(L, x, &a2, &p2), differ(a0, a2) || differ(p0, p2));
    }
}

/* ray derivatives; odd i: at the edges of the fast form's ranges and beyond */
template <bool RADIAL>
__global__ void k_derivs(u64 n, u64* out) {
    for (u64 i = blockIdx.x * (u64)blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
        u64 h = mix(i);
        auto next = [&] { return unit(h = mix(h)); };
        double c = 1400.0 + 200.0 * next(), pos[3] = {6.37e6 - 6000.0 * next(), 3.1 * next(), 6.28 * next()};
        double sg[3] = {0.4 * (next() - 0.5), 4e2 * (next() - 0.5), 4e2 * (next() - 0.5)}, nd[3];
        for (int k = 0; k < 3; ++k) nd[k] = (next() - 0.5) / 700.0;
        if (i & 1) {
            const int which = (int)(mix(h) % 8);
            const u64 m = edge((int)(mix(h + 1) & 15));
            const int e = (int)(mix(h + 2) % 3) - 1;
            if (which == 0) c = bits(m, 10 + e, 0);
            if (which == 1) pos[0] = bits(m, 22 + e, 0);
            if (which == 2) pos[1] = bits(m, -30 * (e + 2), 0);
            if (which == 3) pos[1] = e ? M_PI : 0.0;
            if (which == 4) sg[0] = e ? -0.0 : bits(m, -420, 0);
            if (which == 5) sg[1] = e ? 0.0 : bits(m, -300, 1);
            if (which == 6) nd[2] = e ? -0.0 : bits(m, -60, 1);
            if (which == 7) c = -c;
        }
        if (RADIAL) sg[1] = sg[2] = 0.0;
        double pg[3], ng[3], st, o[7];
        ray_derivs<RADIAL>(c, sg[0], sg[1], sg[2], pos, nd, pg, ng, &st);
        ray_derivs_plain(c, sg[0], sg[1], sg[2], pos, nd, o);
        bool wrong = differ(st, o[6]);
        for (int k = 0; k < 3; ++k)
            wrong = wrong || (differ(pg[k], o[k]) && !(isnan(pg[k]) && isnan(o[k]))) ||
                    (differ(ng[k], o[3 + k]) && !(isnan(ng[k]) && isnan(o[3 + k])));
        tally(out, true, wrong);
    }
}

extern "C" int run(int what, u64 n, const double* m, u64* out) {
    u64* d = nullptr;
    if (cudaMalloc(&d, 4 * sizeof(u64)) != cudaSuccess) return 1;
    cudaMemset(d, 0, 4 * sizeof(u64));
    LossDev L{};
    if (what == 4) { /* the constants as setup_boundary forms them */
        L.kind = WQ3D_LOSS_RAYLEIGH;
        const double conv = 1.0 / (20.0 * M_LOG10E * (2.0 * M_PI));
        L.rl_den = 1000.0 * m[0];
        L.rl_spd = 1500.0 * m[1];
        L.rl_att = m[2] * conv;
        L.rl_shr = 1500.0 * m[3];
        L.rl_satt = m[4] * conv;
        L.rl_fast = 1;
        L.rl_shear_const = L.rl_shr == 0.0;
        if (L.rl_shear_const) {
            cplx cos2, add;
            rl_shear(L, 1.0, &cos2, &add);
            L.rl_cos2[0] = cos2.re;
            L.rl_cos2[1] = cos2.im;
            L.rl_add[0] = add.re;
            L.rl_add[1] = add.im;
        }
    }
    if (what == 0) k_random<<<1184, 256>>>(n, d);
    if (what == 1) k_midpoint<<<1184, 256>>>(n, d);
    if (what == 2) k_edges<<<1, 256>>>(d);
    if (what == 3) k_seed<<<1184, 256>>>(n, d);
    if (what == 4) k_rayleigh<<<592, 128>>>(L, n, d);
    if (what == 5) k_derivs<false><<<592, 128>>>(n, d);
    if (what == 6) k_derivs<true><<<592, 128>>>(n, d);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(out, d, 4 * sizeof(u64), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? 0 : 2;
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("division")
    (d / "t.cu").write_text(SOURCE)
    subprocess.check_call([build.nvcc()] + build.NVCC_FLAGS + ["-I", build.CSRC, "-shared", str(d / "t.cu"),
                                                               "-o", str(d / "t.so")])
    lib = C.CDLL(str(d / "t.so"))

    def call(what, n=0, material=(0.0,) * 5):
        out = (C.c_ulonglong * 4)()
        assert lib.run(what, C.c_ulonglong(n), (C.c_double * 5)(*material), out) == 0
        return list(out)

    return call


def test_random_operands(run):
    tried, wrong, refused, _ = run(0, 1 << 30)
    assert wrong == 0 and tried + refused == 1 << 30 and refused < 1 << 20


def test_quotients_beside_a_midpoint(run):
    tried, wrong = run(1, 1 << 30)[:2]
    assert wrong == 0 and tried > 1 << 28


def test_ends_of_the_ranges(run):
    tried, wrong, checked, misjudged = run(2)
    assert wrong == 0 and misjudged == 0 and tried == 35_256 and checked > 70_000


def test_seed_is_within_the_bound_that_the_cubic_step_needs(run):
    assert run(3, 1 << 28)[0] < 1 << 21  # 2^-19


@pytest.mark.parametrize("material", [
    (1.9, 1.10, 0.8, 0.00, 2.5),    # sand: no shear speed, a shear attenuation
    (2.5, 2.50, 0.01, 1.30, 0.02),  # limestone: shear
    (1.5, 0.98, 0.2, 0.00, 0.00),   # slower than water, no shear at all
    (1.0, 1.00, 0.0, 0.00, 0.00),   # as water: total transmission
    (2.0, 1.80, 0.0, 0.45, 0.00),   # no attenuation: total reflection below the critical angle
])
def test_rayleigh_loss(run, material):
    tried, wrong, fast, fast_wrong = run(4, 1_000_001, material)
    # half of the angles are below the horizon, where a bottom like water
    # has a denominator of zero and leaves the fast form
    assert tried == 1_000_001 and wrong == 0 and fast_wrong == 0 and fast > 490_000


@pytest.mark.parametrize("what", [5, 6])
def test_ray_derivatives(run, what):
    tried, wrong = run(what, 20_000_000)[:2]
    assert tried == 20_000_000 and wrong == 0
