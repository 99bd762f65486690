// The branch-free FP64 quotients and roots of csrc/dem_law.cuh where rounding
// is hardest, and contact_law_fast over all constants that LawParams::fast
// admits.  The hard operands are built in integers: quotients A / B and roots
// of X whose distance from the middle of two numbers is a few parts in 2^106,
// reciprocals of divisors just below a power of two.  Prints one line per
// check: name, cases, mismatches.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>
#include "dem_law.cuh"
using namespace dem;
typedef unsigned long long u64;
__device__ u64 g_n[8], g_bad[8];

__device__ u64 mix(u64& z) {
    z += 0x9E3779B97F4A7C15ull;
    u64 x = z;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}
__device__ double unit(u64& z) { return (double)(mix(z) >> 11) * 0x1p-53; }
__device__ bool bits(double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); }
__device__ bool bits(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }
template <typename F> __device__ bool bits(V3<F> a, V3<F> b) { return bits(a.x, b.x) && bits(a.y, b.y) && bits(a.z, b.z); }
__device__ void count(int slot, bool same) {
    atomicAdd(&g_n[slot], 1ull);
    if (!same) atomicAdd(&g_bad[slot], 1ull);
}

// reciprocals of all but the last significand: the 2^24 below it, and every
// second divisor near the next power of two
__global__ void k_rcp_last() {
    const u64 k = blockIdx.x * 256ull + threadIdx.x + 1;
    const double b = __longlong_as_double((long long)(0x3fffffffffffffffull - k));
    count(0, bits(x_rcp(b), __drcp_rn(b)));
}
__global__ void k_rcp(int reps) {
    u64 z = blockIdx.x * 65536ull + threadIdx.x + 7;
    for (int i = 0; i < reps; i++) {
        const u64 w = mix(z), e = 1023ull - 30 + mix(z) % 61;
        const u64 m = (i & 1) ? 0xfffffffffffffull - (w >> (11 + mix(z) % 52)) : w >> 12;
        const double b = __longlong_as_double((long long)((e << 52) | (m & 0xfffffffffffffull)));
        if ((m & 0xfffffffffffffull) != 0xfffffffffffffull) count(0, bits(x_rcp(b), __drcp_rn(b)));
    }
}
// n operands from the host: quotients a / b (with b != 0) or roots of a
__global__ void k_given(int n, const double* a, const double* b) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (b[i] == 0.0) count(2, bits(x_sqrt(a[i]), __dsqrt_rn(a[i])));
    else count(1, bits(x_div(a[i], b[i]), __ddiv_rn(a[i], b[i])));
}
// contacts over the range of overlaps, radii, masses, motions and histories,
// a block per set of constants
template <typename F> __global__ void k_law(int reps, const LawParams<F>* ps, int slot) {
    const LawParams<F> p = ps[blockIdx.x];
    u64 z = (blockIdx.x * 65536ull + threadIdx.x) * 977 + 11;
    for (int i = 0; i < reps; i++) {
        auto scale = [&](double lo, double hi) { return exp2(lo + (hi - lo) * unit(z)); };
        auto vec = [&](double s) { return mk(s * (unit(z) - 0.5), s * (unit(z) - 0.5), s * (unit(z) - 0.5)); };
        const bool wide = i & 1;
        const F delta = (F)(wide ? scale(-31, 31) : scale(-18, -4)), rs = (F)(wide ? scale(-31, 31) : scale(-6, 2)),
                ms = (F)(wide ? scale(-31, 31) : scale(-6, 4));
        const V3<double> n = vec(2.0);
        const double l = sqrt(dot(n, n));
        const V3<F> nn = mk((F)(n.x / l), (F)(n.y / l), (F)(n.z / l));
        const V3<F> U = cvt<F>(vec(scale(-40, wide ? 20 : -8))), W = cvt<F>(vec(scale(-40, wide ? 20 : -8)));
        V3<double> h = vec(scale(-45, wide ? 30 : -4)), h2 = h;
        V3<F> F1, T1, M1, F2, T2, M2;
        contact_law<F>(delta, nn, rs, ms, U, W, h, (F)20000, p, F1, T1, M1);
        if (!contact_law_fast<F>(delta, nn, rs, ms, U, W, h2, (F)20000, p, F2, T2, M2)) continue;
        count(slot, bits(F1, F2) && bits(T1, T2) && bits(M1, M2) && bits(h, h2));
    }
}
template <typename F> std::vector<LawParams<F>> constants(int n) {
    std::mt19937_64 r(3);
    std::vector<LawParams<F>> v;
    auto pick = [&](double lo, double hi) {   // log-uniform, the ends among them
        const int e = (int)(r() % 8);
        return e == 0 ? lo : e == 1 ? hi : lo * std::pow(hi / lo, (double)(r() >> 11) * 0x1p-53);
    };
    auto zero = [&](double lo, double hi) { return r() % 4 ? pick(lo, hi) : 0.0; };
    while ((int)v.size() < n) {
        const double nu[6] = {0.0, 0.29, 0.5, -1.0, 0.99, 0.9999};
        const dem_contact c{pick(1e-3, 1e15), pick(1e-3, 1e3), nu[r() % 6], zero(1e-6, 1e6), zero(1e-6, 1e6),
                            zero(1e-9, 1e3), zero(1e-9, 1e3)};
        const LawParams<F> p = make_law<F>(c);
        if (p.fast) v.push_back(p);
    }
    return v;
}
template <typename F> void law(int slot) {
    const std::vector<LawParams<F>> v = constants<F>(4096);
    LawParams<F>* d;
    cudaMalloc(&d, v.size() * sizeof(v[0]));
    cudaMemcpy(d, v.data(), v.size() * sizeof(v[0]), cudaMemcpyHostToDevice);
    k_law<F><<<4096, 128>>>(64, d, slot);
}
int main() {
    k_rcp_last<<<65536, 256>>>();
    k_rcp<<<592, 256>>>(400);
    std::vector<double> a, b;
    std::mt19937_64 r(1);
    const u64 one54 = (1ull << 54) - 1;
    // A = (B M + d) / 2^54 exactly, M odd of 54 bits: A / B is d / (B M) away
    // from the middle M / 2^54; every second B near the next power of two
    for (int i = 0; i < 4000000; i++) {
        u64 B = (r() >> 12) | (1ull << 52) | 1;
        if (i & 1) B = (1ull << 53) - 3 - 2 * (r() % (1ull << (i % 44)));   // all but the last one
        u64 inv = B;
        for (int t = 0; t < 6; t++) inv *= 2 - B * inv;   // B^-1 modulo 2^64
        const long long d = (long long)(r() % 16) * 2 - 15;
        const u64 M = ((u64)(-d) * inv) & one54;
        if (!(M >> 53)) continue;
        const u64 A = (u64)(((__int128)B * (__int128)M + d) >> 54);
        if (A >> 53) continue;
        const int e = (int)(r() % 41) - 20;
        a.push_back(std::ldexp((double)A, e - 52));
        b.push_back(std::ldexp((double)B, -52));
    }
    // X = M^2 - c of at most 53 bits, M of 54 bits: M^2 = c modulo 2^55, c = 1 modulo 8
    for (long long c = -65535; c < 65536; c += 8) {
        u64 m = 1;
        for (int k = 3; k < 58; k++)
            if (((m * m - (u64)c) >> k) & 1) m += 1ull << (k - 1);
        for (int v = 0; v < 8; v++) {
            const u64 M = ((v & 1 ? (u64)-m : m) + ((u64)(v >> 1) << 54)) & one54;
            if (!(M >> 53)) continue;
            __int128 X = (__int128)M * M - c;
            int e = 0;
            while (!(X & 1)) { X >>= 1; e++; }
            if (X >> 53) continue;
            a.push_back(std::ldexp((double)(u64)X, e - 106 + 2 * (int)((c & 0xff) >> 3) - 32));
            b.push_back(0.0);
        }
    }
    double *da, *db;
    if (cudaMalloc(&da, a.size() * 8) || cudaMalloc(&db, b.size() * 8)) return 1;
    cudaMemcpy(da, a.data(), a.size() * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(db, b.data(), b.size() * 8, cudaMemcpyHostToDevice);
    k_given<<<((int)a.size() + 255) / 256, 256>>>((int)a.size(), da, db);
    law<float>(3);
    law<double>(4);
    if (cudaDeviceSynchronize() != cudaSuccess) return 1;
    u64 n[8], bad[8];
    cudaMemcpyFromSymbol(n, g_n, sizeof(n));
    cudaMemcpyFromSymbol(bad, g_bad, sizeof(bad));
    const char* name[5] = {"rcp64", "div64", "sqrt64", "law32", "law64"};
    for (int k = 0; k < 5; k++) printf("%s %llu %llu\n", name[k], n[k], bad[k]);
    return 0;
}
