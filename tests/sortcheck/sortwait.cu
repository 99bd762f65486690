// A pass of the radix sort whose first tile is never stepped: the ticket
// counter starts at one, so the tiles behind wait for a count that no block
// publishes, until their limit.  They must still place their records where the
// whole input's stable order has them.  Prints the records checked and those
// out of place (records of the first tile that were written among them).
#include <cstdio>
#include <cstdarg>
#include <cstdlib>
#include "dem_sort.cu"
// what dem_sort.cu takes from the library's other files, unused here
namespace dem {
int fail(int code, const char*, ...) { return code; }
int cuda_fail(cudaError_t, const char*, const char*, int) { return 2; }
int compat_device(CompatDevice**) { return 1; }
int compat_scratch(CompatDevice*, size_t, uint**) { return 1; }
cudaStream_t compat_stream() { return 0; }
}  // namespace dem
using namespace dem;

template <int NT> int run(uint n, int pass) {
    const unsigned tile = NT * kRsItems, nt = (n + tile - 1) / tile;
    std::vector<uint2> in(n), out(n, make_uint2(0u, kEmpty));
    unsigned long long z = n;
    for (uint i = 0; i < n; i++) {
        z = z * 6364136223846793005ull + 1442695040888963407ull;
        in[i] = make_uint2((uint)(z >> 32), i);
    }
    uint2 *d0, *d1;
    uint* sc;
    const size_t words = kRsHead + 2 * (size_t)nt * 256;
    if (cudaMalloc(&d0, n * sizeof(uint2)) || cudaMalloc(&d1, n * sizeof(uint2)) || cudaMalloc(&sc, words * 4)) return 1;
    cudaMemcpy(d0, in.data(), n * sizeof(uint2), cudaMemcpyHostToDevice);
    cudaMemcpy(d1, out.data(), n * sizeof(uint2), cudaMemcpyHostToDevice);
    cudaMemset(sc, 0, words * 4);
    k_radix_hist<<<64, kHistThreads>>>(d0, n, 4, sc);
    const uint one = 1;
    uint* ticket = sc + 4 * 256;
    cudaMemcpy(ticket, &one, 4, cudaMemcpyHostToDevice);
    constexpr int smem = NT * kRsItems * 8 + (NT / 32) * 256 * 4;
    cudaFuncSetAttribute(k_radix_pass<uint, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    uint* look = sc + kRsHead;
    k_radix_pass<uint, NT><<<nt, NT, smem>>>(d0, d1, n, pass, sc, ticket, look, look + (size_t)nt * 256);
    if (cudaMemcpy(out.data(), d1, n * sizeof(uint2), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    std::vector<uint> place(257, 0u);
    for (uint i = 0; i < n; i++) place[((in[i].x >> (8 * pass)) & 255u) + 1]++;
    for (int d = 0; d < 256; d++) place[d + 1] += place[d];
    uint checked = 0, bad = 0;
    for (uint i = 0; i < n; i++) {
        const uint2 v = out[place[(in[i].x >> (8 * pass)) & 255u]++];
        const bool first = i < tile;   // not stepped: its places stay as they were
        checked += !first;
        bad += first ? v.y != kEmpty : (v.x != in[i].x || v.y != i);
    }
    printf("%u %u\n", checked, bad);
    cudaFree(d0);
    cudaFree(d1);
    cudaFree(sc);
    return 0;
}
int main() {
    // two tiles; more than a look-back round's, with a last one of one record
    return run<256>(4096 + 4096, 0) || run<256>(21 * 4096 + 1, 1) || run<512>(40 * 8192 + 5, 3);
}
