// The branch-free quotients and roots of csrc/dem_law.cuh against CUDA's
// correctly rounded ones, and contact_law_fast against contact_law, bit for
// bit.  Prints one line per check: name, cases, mismatches (and, for the law,
// the cases the fast form took).
#include <cstdio>
#include <cstring>
#include "dem_law.cuh"
using namespace dem;
__device__ unsigned long long g_bad[8], g_took[8];

__global__ void k_f32(int ex) {   // every significand at one exponent (roots: two)
    const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m < (1u << 23)) {
        const float b = __uint_as_float(((unsigned)(127 + ex) << 23) | m);
        if (x_rcp(b) != __frcp_rn(b)) atomicAdd(&g_bad[0], 1ull);
    }
    if (m < (1u << 24)) {
        const float x = __uint_as_float(((unsigned)(127 + ex) << 23) + m);
        if (x_sqrt(x) != __fsqrt_rn(x)) atomicAdd(&g_bad[1], 1ull);
    }
}
__device__ unsigned long long mix(unsigned long long& z) {
    z += 0x9E3779B97F4A7C15ull;
    unsigned long long x = z;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}
__device__ double unit(unsigned long long& z) { return (double)(mix(z) >> 11) * 0x1p-53; }
__global__ void k_div(int reps) {   // random and nearly halfway quotients
    unsigned long long z = blockIdx.x * 65536ull + threadIdx.x + 1;
    for (int i = 0; i < reps; i++) {
        const unsigned long long w = mix(z), v = mix(z);
        const float b = __uint_as_float(((107u + (unsigned)((w >> 50) % 40)) << 23) | (unsigned)(w & 0x7fffff));
        const float q = __uint_as_float((127u << 23) | (unsigned)(v & 0x7fffff));
        float a = __uint_as_float(((107u + (unsigned)((v >> 50) % 40)) << 23) | (unsigned)((w >> 23) & 0x7fffff));
        if (i & 1) a = (float)((double)b * ((double)q + 0x1p-24));
        if (x_div(a, b) != __fdiv_rn(a, b)) atomicAdd(&g_bad[2], 1ull);
        const double bd = __longlong_as_double(((1003ull + (w >> 58) % 40) << 52) | (w & 0xfffffffffffffull));
        double ad = __longlong_as_double(((1003ull + (v >> 58) % 40) << 52) | (v & 0xfffffffffffffull));
        if (i & 1) ad = bd * __longlong_as_double((1023ull << 52) | (v & 0xfffffffffffffull));
        if (x_div(ad, bd) != __ddiv_rn(ad, bd)) atomicAdd(&g_bad[3], 1ull);
        if (x_sqrt(bd) != __dsqrt_rn(bd)) atomicAdd(&g_bad[4], 1ull);
    }
}
template <typename F> __device__ bool same(V3<F> a, V3<F> b) { return a.x == b.x && a.y == b.y && a.z == b.z; }
// contacts over the whole range of overlaps, radii, motions and histories,
// with exact zeros and values far outside the fast form's range among them
template <typename F> __global__ void k_law(int reps, LawParams<F> p, int slot) {
    unsigned long long z = (blockIdx.x * 65536ull + threadIdx.x) * 977 + 5;
    for (int i = 0; i < reps; i++) {
        auto scale = [&](double lo, double hi) { return exp2(lo + (hi - lo) * unit(z)); };
        auto vec = [&](double s) { return mk(s * (unit(z) - 0.5), s * (unit(z) - 0.5), s * (unit(z) - 0.5)); };
        const int kind = (int)(mix(z) % 16);
        const double wide = kind == 0 ? 1.0 : 0.0;
        const F delta = (F)scale(wide ? -80 : -18, wide ? 40 : -4), rs = (F)scale(-6, 2), ms = (F)scale(-6, 4);
        V3<double> n = vec(2.0);
        const double l = sqrt(dot(n, n));
        const V3<F> nn = mk((F)(n.x / l), (F)(n.y / l), (F)(n.z / l));
        const V3<F> U = cvt<F>(vec(kind == 1 ? 0.0 : scale(-40, -8))), W = cvt<F>(vec(kind == 2 ? 0.0 : scale(-40, -8)));
        V3<double> h = vec(kind == 3 ? 0.0 : scale(kind == 4 ? -120 : -40, -4)), h2 = h;
        V3<F> F1, T1, M1, F2, T2, M2;
        contact_law<F>(delta, nn, rs, ms, U, W, h, (F)20000, p, F1, T1, M1);
        if (!contact_law_fast<F>(delta, nn, rs, ms, U, W, h2, (F)20000, p, F2, T2, M2)) continue;
        atomicAdd(&g_took[slot], 1ull);
        if (!same(F1, F2) || !same(T1, T2) || !same(M1, M2) || !same(h, h2)) atomicAdd(&g_bad[slot], 1ull);
    }
}
int main() {
    for (int ex = -60; ex <= 60; ex += 15) k_f32<<<(1 << 24) / 256, 256>>>(ex);
    k_div<<<592, 256>>>(400);
    dem_contact c{566830.28, 0.3, 0.29, 0.225, 0.225, 0.0, 0.002};
    k_law<float><<<592, 256>>>(100, make_law<float>(c), 5);
    k_law<double><<<592, 256>>>(100, make_law<double>(c), 6);
    if (cudaDeviceSynchronize() != cudaSuccess) return 1;
    unsigned long long bad[8], took[8];
    cudaMemcpyFromSymbol(bad, g_bad, sizeof(bad));
    cudaMemcpyFromSymbol(took, g_took, sizeof(took));
    const char* name[7] = {"rcp32", "sqrt32", "div32", "div64", "sqrt64", "law32", "law64"};
    for (int k = 0; k < 7; k++) printf("%s %llu %llu\n", name[k], bad[k], took[k]);
    return 0;
}
