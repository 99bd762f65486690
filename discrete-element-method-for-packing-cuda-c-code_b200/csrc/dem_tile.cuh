// dem_tile.cuh -- the window of a bed whose components do not fit a block
// (included by dem_engine.cu: it uses that file's step functions).
//
// The bound particles are cut into tiles, runs of a Hilbert curve through the
// box, and one persistent launch steps every tile through the window.  A tile
// evaluates the pairs of its own particles -- a pair across two tiles by both
// of them, with the same arguments and so the same bits -- so that a step
// exchanges particle states only: pair results stay in shared memory, and the
// tiles that share pairs wait for one another by step counters instead of a
// grid barrier.  States are double-buffered in tile order (ts): a tile
// reads step s from one buffer and writes step s + 1 to the other; a tile
// whose neighbours have all finished step s - 1 may overwrite what they read
// in it (the neighbour relation is symmetric: both tiles hold the pair).
// The arithmetic and the order of every sum are pair_item's, wall_item's and
// bound_item's, so the states are those of k_window bit for bit.
//
// Why: k_window on a settled bed of 500,000 spheres (1.83 M pairs) took 150 us
// a step, half of it DRAM traffic -- each pair's force and torque written at
// both ends' slots and gathered back, a working set above L2 -- and on a bed
// of 20,000 14 us a step, two grid barriers and two chains of dependent
// loads.  The tiles: 101 us and 6.6 us (mixed); what is left is the shared-
// memory pipe (two 64-byte states and 40 bytes of results per pair, ~50 %
// busy) and the instructions of the law (~45 % of the issue slots).

// A particle in shared memory: its record and its displacement since the
// list.  The stride is an odd number of 16-byte words, so that random
// partners spread over the banks.
template <typename Real> struct TileRec;
template <> struct alignas(16) TileRec<float> { char rec[64]; float4 q; };
template <> struct alignas(16) TileRec<double> { char rec[80]; float4 q; char pad[16]; };
static_assert(sizeof(TileRec<float>) == 80 && sizeof(TileRec<double>) == 112, "tile record layout");

// Threads of a block (a particle each in the particle phase, so also the
// particles of a tile at most); a tile's pairs and wall items at most (the
// arrays' stride) when every tile is resident (Q1) and when blocks stream
// several (Q2: two stages leave less room for results); particles per tile
// the arrays are allocated for at least; shared memory of a block: two blocks
// per SM, so that one block's barriers and loads overlap another's
// arithmetic; registers.  Measured on a 500,000-sphere bed, mixed, per
// 20-step window: 256 threads of 128 registers 2,020 us, 320 of 96 2,190, 256
// of 80 (three blocks) 2,290 -- the spilled words miss the L1 that the shared
// memory leaves -- , one block of 512 of 128 2,080; 100,003 spheres, FP64: 192
// threads of 168 694 us, 256 of 128 762.
template <typename Real> struct TileCap;
template <> struct TileCap<float> {
    static constexpr uint P = 256, Q1 = 1920, Q2 = 1536, floor = 128, smem = 113664;
    static constexpr int regs = 128;
};
template <> struct TileCap<double> {
    static constexpr uint P = 192, Q1 = 1024, Q2 = 832, floor = 80, smem = 113664;
    static constexpr int regs = 168;
};
constexpr uint kTileMin = 32;        // particles per tile at least (small systems)
constexpr uint kTileNbr = 128;       // tiles that share pairs with one tile, at most
constexpr uint kTileHash = 512;      // their hash set while they are collected
constexpr uint kTileRow = 8;         // row entries that k_tile_lists holds in registers
constexpr uint kFlagStride = 32;     // words between step counters: a 128-byte line each (in 14 shared lines the
                                     // polls of 436 tiles queued at a few L2 slices: ~4,800 cycles a wait)
constexpr uint kTileRetry = 64;      // windows after which larger tiles are tried again (a window that does not fit
                                     // costs its lists and the grid-barrier kernel's time: ~1 % if it fails again)
constexpr uint kCurveEvery = 256;    // windows between two computations of the curve: at 0.1 m/s a sphere of the
                                     // 1 mm configurations moves 0.26 d in that time, so tiles stay compact

__host__ __device__ constexpr uint al16(uint b) { return (b + 15u) & ~15u; }

// A tile's tables, packed (byte offsets in its blob and in shared memory):
// te, an entry per pair -- first the pairs inside the tile, lo | hi << 9 |
// result << 18 (particles and result by their index in the tile), then those
// across tiles, own particle | (1 << 9: it is hi) | result << 18 -- ; tx, the
// partner's slot of each pair across tiles; tn, those tiles; tr, the reverse
// rows as results; tp, per particle its row (first result | count << 16), its
// reverse row (first in tr | count << 16), the result of its wall item
// (kEmpty: none) and its id.
struct TileTables {
    uint ox, on, orr, op, bytes;
    __host__ __device__ TileTables(uint m, uint nin, uint tot, uint nrev, uint nnbr) {
        ox = al16(4u * tot);
        on = ox + al16(4u * (tot - nin));
        orr = on + al16(4u * nnbr);
        op = orr + al16(2u * nrev);
        bytes = op + 16u * m;
    }
};
__host__ __device__ constexpr uint tile_blob(uint q, uint p) { return q * 10u + kTileNbr * 4u + 64u + p * 16u; }

template <typename Real> struct TileArgs {
    uint* tw;
    uint G, Q, BB;           // resident blocks; the per-tile arrays' stride; bytes of a blob
    uint* curve;             // every particle's id along the curve
    uint* inv;               // a bound particle's slot: its place among the bound ones along the curve
    uint* flag;              // per tile (kFlagStride apart): steps finished in this window
    uint4* head;             // per tile, two: pairs inside, all pairs, wall items; reverse entries,
                             // neighbour tiles
    unsigned char* blob;     // per tile: its tables
    uint* tk;                // per tile Q: a pair's slot in the list (top bit: the other tile owns its history)
    unsigned short* twl;     // per tile P: its wall items' particles
    PRec<Real>* ts[2];       // states by slot, step parity
    float4* tq;              // displacements since the list by slot
    PRec<Real>* So;          // the states after the window
    Planes3<double> Ho;      // the pair histories after the window
    Planes3<double> th;      // per tile Q: its pairs' histories between the first and the last step
};

// The window's tiles of its n bound particles: particles per tile and shared
// memory of one stage (states and tables).  f pairs per particle; a fraction c ~ 1.45 /
// P^(1/3) of a tile's pairs crosses its surface (a cube of P particles
// loses 1.5 / P^(1/3)); 15 % of the pairs' bytes for uneven density, and
// `shrink` sixteenths less after a window in which a tile did not fit.  A
// stage that is the average tile's with the spare room shared out refuses a
// dense core under a loose cloud at any size (rows of 6 among a mean of 1.2):
// such windows stay with the grid-barrier kernel, which is the faster one
// there in PCCP (stages as the largest tile needs let them run as tiles: 69,408
// spheres FP64 414 -> 522 us a window, 246,080 mixed 716 -> 747; PP 988 -> 523
// and 991 -> 744).  One tile per block when the system fits the resident blocks (its states then stay in
// shared memory), else two stages per block (the next tile's loads run beside
// the current one's steps), evened out over whole rounds of the G blocks.
struct TilePlan { uint p, stage; };
__host__ __device__ inline TilePlan tile_plan(long long n, long long pairs, uint G, uint P, uint smem,
                                              uint rec, uint res, uint shrink) {
    TilePlan t{0u, 0u};
    if (n <= 0 || shrink > 12u) return t;
    const double f = 1.15 * (double)pairs / (double)n;
    auto stage1 = [&](double p) {
        const double c = fmin(0.6, 1.45 / cbrt(p));
        return rec + 17.0 + 4.0 * f * (1.0 + c) + 8.0 * c * f + 2.0 * f;
    };
    auto result1 = [&](double p) { return res * (f * (1.0 + fmin(0.6, 1.45 / cbrt(p))) + 0.3); };
    const double room = (double)smem - 256.0, cut = (16.0 - (double)shrink) / 16.0;
    double p = (double)((n + G - 1) / G);
    if (p < (double)kTileMin) p = (double)kTileMin;
    if (p <= (double)P * cut && p * (stage1(p) + result1(p)) <= room * cut) {
        t.p = (uint)p;
        t.stage = al16((uint)(p * stage1(p)));
        const double rest = room - p * (stage1(p) + result1(p));   // the spare room, shared out
        if (rest > 0.0) t.stage += al16((uint)(rest * stage1(p) / (stage1(p) + result1(p)))) & ~15u;
        return t;
    }
    double p0 = (double)P;
    for (int k = 0; k < 4; k++) p0 = fmin((double)P, room / (2.0 * stage1(p0) + result1(p0)));
    p0 = floor(p0 * cut);
    if (p0 < (double)kTileMin) return t;
    const long long rounds = (n + (long long)(G * p0) - 1) / (long long)(G * p0);
    p = (double)((n + (long long)G * rounds - 1) / ((long long)G * rounds));
    t.p = (uint)p;
    const double rest = room - p * (2.0 * stage1(p) + result1(p));
    t.stage = al16((uint)(p * stage1(p)));
    if (rest > 0.0) t.stage += (uint)(rest * stage1(p) / (2.0 * stage1(p) + result1(p))) & ~15u;
    return t;
}

// Tiles a context of n particles may need.
inline long long tile_max(long long n, uint G, uint floor) {
    const long long small = (n + kTileMin - 1) / kTileMin, large = (n + floor - 1) / floor + 1;
    return std::min<long long>(small, std::max<long long>(G, large));
}

// Position of a lattice point on the Hilbert curve of `b` bits per axis
// (Skilling, "Programming the Hilbert curve", 2004: the inverse undo, then
// Gray decoding on the transposed index).
__host__ __device__ inline uint hilbert3(uint x, uint y, uint z, int b) {
    uint X[3] = {x, y, z};
    const uint top = 1u << (b - 1);
    for (uint q = top; q > 1; q >>= 1) {
        const uint m = q - 1;
        for (int i = 0; i < 3; i++) {
            if (X[i] & q) {
                X[0] ^= m;
            } else {
                const uint t = (X[0] ^ X[i]) & m;
                X[0] ^= t;
                X[i] ^= t;
            }
        }
    }
    X[1] ^= X[0];
    X[2] ^= X[1];
    uint t = 0;
    for (uint q = top; q > 1; q >>= 1)
        if (X[2] & q) t ^= q - 1;
    X[0] ^= t; X[1] ^= t; X[2] ^= t;
    uint k = 0;
    for (int i = b - 1; i >= 0; i--)
        k = (k << 3) | (((X[0] >> i) & 1u) << 2) | (((X[1] >> i) & 1u) << 1) | ((X[2] >> i) & 1u);
    return k;
}

// The curve's bins: the box in cubes of 2^bits cells of edge cs, the cubes in
// raster order, a Hilbert curve through each (a box far from cubic wastes no
// bins on a cube around it).
constexpr uint kCurveBins = 1u << 21;   // at most
struct CurveGrid { double cs; int bits, cx, cy, cz; uint nbins; };
inline CurveGrid curve_grid(const double world[3], double cell) {
    CurveGrid g{cell, 1, 1, 1, 1, 8u};
    const double least = std::min(world[0], std::min(world[1], world[2]));
    for (;; g.cs *= 1.26) {
        g.bits = 1;
        while (g.bits < 7 && g.cs * 1.5 * (double)(1 << g.bits) < least) g.bits++;
        const double cube = g.cs * (double)(1 << g.bits);
        const double x = std::ceil(world[0] / cube), y = std::ceil(world[1] / cube), z = std::ceil(world[2] / cube);
        if (x * y * z * std::pow(8.0, g.bits) > (double)kCurveBins) continue;
        g.cx = std::max(1, (int)x); g.cy = std::max(1, (int)y); g.cz = std::max(1, (int)z);
        g.nbins = ((uint)g.cx * (uint)g.cy * (uint)g.cz) << (3 * g.bits);
        return g;
    }
}
__device__ __forceinline__ uint curve_bin(const V3<double>& p, const GridC& g, const CurveGrid& c) {
    auto cell = [&](double v, int cubes) -> uint {   // clamped (not a number: 0)
        const double f = v / c.cs, top = (double)((cubes << c.bits) - 1);
        return f >= top ? (uint)((cubes << c.bits) - 1) : (f > 0.0 ? (uint)f : 0u);
    };
    const uint x = cell(p.x - g.ox, c.cx), y = cell(p.y - g.oy, c.cy), z = cell(p.z - g.oz, c.cz);
    const uint m = (1u << c.bits) - 1u;
    const uint cube = ((z >> c.bits) * (uint)c.cy + (y >> c.bits)) * (uint)c.cx + (x >> c.bits);
    return (cube << (3 * c.bits)) | hilbert3(x & m, y & m, z & m, c.bits);
}

// The window's tiles in one cooperative launch: their size, the step
// counters; when the curve is missing or old, the particles' order along it (a
// counting sort by bin, any order inside one); the bound ones in that order,
// numbered; then each tile's lists, by one
// block: its pairs (the rows of its particles, and the reverse-row pairs
// whose lower particle is in another tile), the tables above, the wall items,
// and its particles' states in tile order.  One launch: as separate kernels
// the window graph took 24 more nodes, 90 us longer to instantiate.  Bound by
// the latency of its gathers; with the partners' slots held in registers and
// three blocks per SM (80 registers), and the plan made by every block instead of
// behind a barrier: 44 -> 28 us for a bed of 20,000 spheres, 88 -> 62 us of
// 100,000 in FP64, 187 -> 155 us of 500,000.
template <typename Real, bool PP>
__global__ void __launch_bounds__(TileCap<Real>::P, 3)
    k_tile_lists(StepArgs<Real> a, TileArgs<Real> T, const uint* __restrict__ bflag, GridC g, CurveGrid cg, uint ntmax,
                 uint* key, uint* __restrict__ arrival, uint* __restrict__ count, uint* __restrict__ start,
                 uint* __restrict__ bsum, uint* bar) {
    if (a.ccw && !a.ccw[1]) return;   // the cluster batches step this window
    const uint Q = T.Q;
    constexpr uint PC = TileCap<Real>::P;
    constexpr uint kTileThreads = PC;
    constexpr uint RB = 10 * sizeof(Real);   // bytes of a result
    __shared__ uint s_own[kTileThreads], s_ob[kTileThreads], s_cb[kTileThreads], s_ib[kTileThreads], s_hb[kTileThreads],
        s_rb[kTileThreads], s_wb[kTileThreads];
    __shared__ uint s_tmp[34], s_hash[kTileHash], s_nbr[kTileNbr], s_nn;
    const uint p = threadIdx.x, nthr = gridDim.x * kTileThreads, gid = blockIdx.x * kTileThreads + p;
    const long long n = a.n;
    const uint nbound = a.bpos[n];
    uint nbar = 0;
    for (uint t = gid; t < ntmax; t += nthr) T.flag[(size_t)t * kFlagStride] = 0u;
    // the plan: every block makes it from the same words, the first writes it
    // once all have read them (after the next barrier)
    __shared__ uint s_plan[8];
    if (p == 0) {
        const long long pairs = a.off[n];
        // how much smaller: a sixteenth more after a window whose tiles did not
        // fit, one less after kTileRetry windows; smaller tiles do not help one
        // that has too many neighbours: no tiles for as many windows
        const uint over = T.tw[kTwOver];
        uint shrink = T.tw[kTwShrink], since = T.tw[kTwSince] + 1u, rest = T.tw[kTwRest];
        if (over == 2u) {
            ++shrink;
            since = 0u;
        } else if (shrink && since >= kTileRetry) {
            --shrink;
            since = 0u;
        }
        rest = over == 3u ? kTileRetry : rest ? rest - 1u : 0u;
        TilePlan pl{0u, 0u};
        if (pairs <= a.cap && !rest)
            pl = tile_plan((long long)nbound, pairs, T.G, PC, TileCap<Real>::smem, (uint)sizeof(TileRec<Real>), RB, shrink);
        const uint nt = pl.p ? (nbound + pl.p - 1) / pl.p : 0u;
        const bool fits = nbound == 0u || (pl.p && nt <= ntmax);
        const uint age = T.tw[kTwAge];
        const bool need = (!T.tw[kTwValid] || age >= kCurveEvery) && fits && nt;
        s_plan[0] = pl.p; s_plan[1] = nt; s_plan[2] = pl.stage; s_plan[3] = fits ? 0u : 1u;
        s_plan[4] = need ? 1u : 0u;
        s_plan[5] = shrink; s_plan[6] = since; s_plan[7] = rest;
    }
    __syncthreads();
    const uint PT = s_plan[0], nt = s_plan[1], stage = s_plan[2];
    const bool go = PT != 0u && nt != 0u && nt <= ntmax;
    auto barrier = [&]() { grid_barrier(bar, nbar++, gridDim.x, a.words); };
    auto publish = [&]() {
        if (gid != 0) return;
        T.tw[kTwP] = PT;
        T.tw[kTwTiles] = nt;
        T.tw[kTwStage] = stage;
        T.tw[kTwOver] = s_plan[3];
        T.tw[kTwShrink] = s_plan[5];
        T.tw[kTwSince] = s_plan[6];
        T.tw[kTwRest] = s_plan[7];
        if (go) {
            T.tw[kTwAge] = s_plan[4] ? 1u : T.tw[kTwAge] + 1u;
            T.tw[kTwValid] = 1u;
        }
    };
    if (!go) {
        barrier();
        publish();
        return;
    }
    if (s_plan[4]) {
        for (long long i = gid; i < n; i += nthr) {
            const uint c = curve_bin(ld_pos<false>(a.S + i), g, cg);
            key[i] = c;
            arrival[i] = atomicAdd(count + c, 1u);
        }
        grid_barrier(bar, nbar++, gridDim.x, a.words);
        // exclusive scan of the counts: a contiguous run of bins per block
        const uint per = (cg.nbins + gridDim.x - 1) / gridDim.x;
        const uint b0 = min(cg.nbins, blockIdx.x * per), b1 = min(cg.nbins, b0 + per);
        uint v = 0;
        for (uint k = b0 + p; k < b1; k += kTileThreads) v += __ldcg(count + k);
        s_own[p] = v;
        const uint mine = block_exscan(s_own, s_ob, kTileThreads, s_tmp);
        if (p == 0) bsum[blockIdx.x] = mine;
        grid_barrier(bar, nbar++, gridDim.x, a.words);
        v = 0;
        for (uint k = p; k < blockIdx.x; k += kTileThreads) v += __ldcg(bsum + k);
        s_own[p] = v;
        uint run = block_exscan(s_own, s_ob, kTileThreads, s_tmp);
        for (uint k0 = b0; k0 < b1; k0 += kTileThreads) {
            const uint k = k0 + p;
            s_own[p] = k < b1 ? __ldcg(count + k) : 0u;
            const uint sum = block_exscan(s_own, s_ob, kTileThreads, s_tmp);
            if (k < b1) {
                start[k] = run + s_ob[p];
                count[k] = 0u;   // for the next time
            }
            run += sum;
        }
        grid_barrier(bar, nbar++, gridDim.x, a.words);
        for (long long i = gid; i < n; i += nthr) {
            const uint t = __ldcg(start + key[i]) + arrival[i];
            if ((long long)t >= n) continue;   // cannot happen (counts left over from a wait that gave up)
            T.curve[t] = (uint)i;
        }
        grid_barrier(bar, nbar++, gridDim.x, a.words);
    }
    // the bound particles along the curve: their ids (bl) and their slots
    uint* bl = key;
    {
        const uint per = (uint)((n + gridDim.x - 1) / gridDim.x);
        const uint b0 = (uint)min(n, (long long)blockIdx.x * per), b1 = (uint)min(n, (long long)b0 + per);
        uint v = 0;
        for (uint k = b0 + p; k < b1; k += kTileThreads) v += bflag[__ldcg(T.curve + k)];
        s_own[p] = v;
        const uint mine = block_exscan(s_own, s_ob, kTileThreads, s_tmp);
        uint* bs = bsum + gridDim.x;   // the curve's sums may still be read
        if (p == 0) bs[blockIdx.x] = mine;
        grid_barrier(bar, nbar++, gridDim.x, a.words);
        publish();
        v = 0;
        for (uint k = p; k < blockIdx.x; k += kTileThreads) v += __ldcg(bs + k);
        s_own[p] = v;
        uint run = block_exscan(s_own, s_ob, kTileThreads, s_tmp);
        for (uint k0 = b0; k0 < b1; k0 += kTileThreads) {
            const uint k = k0 + p, i = k < b1 ? __ldcg(T.curve + k) : 0u;
            const uint on = k < b1 ? bflag[i] : 0u;
            s_own[p] = on;
            const uint sum = block_exscan(s_own, s_ob, kTileThreads, s_tmp);
            if (on && run + s_ob[p] < nbound) {
                bl[run + s_ob[p]] = i;
                T.inv[i] = run + s_ob[p];
            }
            run += sum;
        }
        grid_barrier(bar, nbar++, gridDim.x, a.words);
    }
    if (ld_acquire(bar + kBarGiveUp)) {   // the orders may be incomplete: the grid-barrier kernel has the window
        if (p == 0) { T.tw[kTwOver] = 1u; T.tw[kTwValid] = 0u; }
        return;
    }
    for (uint t = blockIdx.x; t < nt; t += gridDim.x) {
        const uint first = t * PT, slot = first + p;
        const uint m = min(PT, nbound - first);
        uint id = kEmpty, o0 = 0, no = 0, r0 = 0, nr = 0, nc = 0, ni = 0, ws = kEmpty;
        if (p < m) {
            id = __ldcg(bl + slot);
            o0 = a.off[id]; no = a.off[id + 1] - o0;
            r0 = a.roff[id]; nr = a.roff[id + 1] - r0;
            if (!PP) ws = a.wslot[id];   // PP: a particle steps its walls itself
        }
        // the partners' slots of the first kTileRow entries, loaded side by side
        // and kept: one after the other, a row's entries are a chain of loads
        // (three for a reverse entry), and each of the three walks below had it
        uint so[kTileRow], rr[kTileRow], rl[kTileRow], sr[kTileRow];
#pragma unroll
        for (uint e = 0; e < kTileRow; e++) {
            so[e] = e < no ? a.ln[o0 + e] : kEmpty;
            rr[e] = e < nr ? a.rk[r0 + e] : kEmpty;
        }
#pragma unroll
        for (uint e = 0; e < kTileRow; e++) {
            if (e < no) so[e] = __ldcg(T.inv + so[e]);
            rl[e] = e < nr ? a.lp[rr[e]] : kEmpty;
        }
#pragma unroll
        for (uint e = 0; e < kTileRow; e++) sr[e] = e < nr ? __ldcg(T.inv + rl[e]) : kEmpty;
        // f(place in the row, slot) over the row; g(place, pair, lo, slot) over the reverse row
        auto own = [&](auto&& f) {
#pragma unroll
            for (uint e = 0; e < kTileRow; e++)
                if (e < no) f(e, so[e]);
            for (uint e = kTileRow; e < no; e++) f(e, __ldcg(T.inv + a.ln[o0 + e]));
        };
        auto rev = [&](auto&& f) {
#pragma unroll
            for (uint e = 0; e < kTileRow; e++)
                if (e < nr) f(e, rr[e], rl[e], sr[e]);
            for (uint e = kTileRow; e < nr; e++) {
                const uint k = a.rk[r0 + e], lo = a.lp[k];
                f(e, k, lo, __ldcg(T.inv + lo));
            }
        };
        own([&](uint, uint s) { ni += s - first < m ? 1u : 0u; });   // unsigned: inside the tile
        rev([&](uint, uint, uint, uint s) { nc += s - first < m ? 0u : 1u; });
        for (uint k = p; k < kTileHash; k += kTileThreads) s_hash[k] = kEmpty;
        if (p == 0) s_nn = 0u;
        s_own[p] = no;
        s_cb[p] = nc;
        s_ib[p] = ni;
        s_hb[p] = no - ni + nc;
        s_rb[p] = nr;
        s_wb[p] = ws != kEmpty ? 1u : 0u;
        __syncthreads();
        const uint town = block_exscan(s_own, s_ob, kTileThreads, s_tmp);
        const uint tcross = block_exscan(s_cb, s_cb, kTileThreads, s_tmp);
        const uint tin = block_exscan(s_ib, s_ib, kTileThreads, s_tmp);
        block_exscan(s_hb, s_hb, kTileThreads, s_tmp);
        const uint trev = block_exscan(s_rb, s_rb, kTileThreads, s_tmp);
        const uint twall = block_exscan(s_wb, s_wb, kTileThreads, s_tmp);
        const uint tot = town + tcross;
        // the tiles of the partners outside
        auto meet = [&](uint s) {
            if (s - first < m) return;
            const uint nb = s / PT;
            uint h = (nb * 2654435761u) >> 23;   // 9 bits: kTileHash
            for (uint tries = 0; tries < kTileHash; tries++) {
                const uint old = atomicCAS(&s_hash[h], kEmpty, nb);
                if (old == nb) return;
                if (old == kEmpty) {
                    const uint k = atomicAdd(&s_nn, 1u);
                    if (k < kTileNbr) s_nbr[k] = nb;
                    return;
                }
                h = (h + 1u) & (kTileHash - 1u);
            }
            atomicAdd(&s_nn, kTileNbr);   // the set is full: too many
        };
        own([&](uint, uint s) { meet(s); });
        rev([&](uint, uint, uint, uint s) { meet(s); });
        __syncthreads();
        const uint nnbr = s_nn;
        // whether it fits (the same for every thread): the arrays' strides, a
        // stage, and the results beside one stage or two
        const uint nstage = nt <= T.G ? 1u : 2u;
        bool fits = tot + twall <= Q && trev <= Q && nnbr <= kTileNbr;
        if (fits) {
            const TileTables L(m, tin, tot, trev, nnbr);
            fits = m * (uint)sizeof(TileRec<Real>) + L.bytes <= stage &&
                   nstage * stage + (tot + twall) * RB <= TileCap<Real>::smem;
        }
        if (!fits) {
            if (p == 0) atomicMax(T.tw + kTwOver, nnbr > kTileNbr ? 3u : 2u);
            __syncthreads();   // s_nn is the next tile's
            continue;
        }
        const TileTables L(m, tin, tot, trev, nnbr);
        unsigned char* B = T.blob + (size_t)t * T.BB;
        uint* te = reinterpret_cast<uint*>(B);
        uint* tx = reinterpret_cast<uint*>(B + L.ox);
        if (p < nnbr) reinterpret_cast<uint*>(B + L.on)[p] = s_nbr[p];
        unsigned short* tr = reinterpret_cast<unsigned short*>(B + L.orr);
        uint4* tp = reinterpret_cast<uint4*>(B + L.op);
        uint* tk = T.tk + (size_t)t * Q;
        uint ii = s_ib[p], hh = s_hb[p];
        own([&](uint e, uint s) {
            const uint k = o0 + e, res = s_ob[p] + e;
            if (s - first < m) {
                te[ii] = p | ((s - first) << 9) | (res << 18);
                tk[ii++] = k;
            } else {
                tx[hh] = s;
                te[tin + hh] = p | (res << 18);
                tk[tin + hh++] = k;
            }
        });
        uint c = 0;
        rev([&](uint u, uint k, uint lo, uint s) {
            uint res;
            if (s - first < m) {
                res = s_ob[s - first] + (k - a.off[lo]);
            } else {
                res = town + s_cb[p] + c++;
                tx[hh] = s;
                te[tin + hh] = p | 512u | (res << 18);
                tk[tin + hh++] = k | 0x80000000u;
            }
            tr[s_rb[p] + u] = (unsigned short)res;
        });
        if (ws != kEmpty) T.twl[(size_t)t * PC + s_wb[p]] = (unsigned short)p;
        if (p < m) {
            tp[p] = make_uint4(s_ob[p] | (no << 16), s_rb[p] | (nr << 16), ws != kEmpty ? tot + s_wb[p] : kEmpty, id);
            V3<double> x, d;
            V3<Real> av;
            Real r;
            ld_rec<false>(a.S + id, x, d, av, r);
            st_rec(T.ts[0] + slot, x, d, av, r);
            T.tq[slot] = a.Q[id];
        }
        if (p == 0) {
            T.head[2 * (size_t)t] = make_uint4(tin, tot, twall, 0u);
            T.head[2 * (size_t)t + 1] = make_uint4(trev, nnbr, 0u, 0u);
        }
        __syncthreads();   // the shared arrays are the next tile's
    }
}

// A pair's results in shared memory: F (3), the torque on lo (3), on hi (3),
// 1 when touching: 5 two-vectors (40 or 80 bytes, no two of 16 consecutive
// ones in the same banks).
template <typename Real> struct Two;
template <> struct Two<float> { typedef float2 T; };
template <> struct Two<double> { typedef double2 T; };
__device__ __forceinline__ float2 mk2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ double2 mk2(double a, double b) { return make_double2(a, b); }

// Waits until tile flag *f reaches `target` (bounded as grid_wait: after the
// limit kStBarrier is recorded and the launch's give-up word raised, and no
// wait of the launch waits any more).
__device__ __forceinline__ void tile_wait(const uint* f, uint target, uint* giveup, EngineWords* words) {
    if (ld_acquire(f) >= target) return;
    unsigned long long t0 = global_ns();
    uint polls = 0;
    while (ld_acquire(f) < target) {
        ++polls;
        if ((polls & 63u) == 1u) {
            if (ld_acquire(giveup)) return;
            const unsigned long long now = global_ns();
            if (now < t0) t0 = now;
            if ((now - t0 > kBarrierNs && polls > kBarrierMinPolls) || polls > kBarrierMaxPolls) {
                atomicOr(&words->status, kStBarrier);
                atomicExch(giveup, 1u);
                return;
            }
        }
    }
}

// The block's "neighbours are ready" signal: an mbarrier of one arrival, one
// phase per tile-step.  The waiting warps are suspended (a spin on a shared
// word took a quarter of the SM's issue slots); the wait ends with the
// bounded wait of the warp that arrives, and is bounded itself.
__device__ __forceinline__ void ready_init(unsigned long long* b) {
    asm volatile("mbarrier.init.shared.b64 [%0], 1;" ::"r"((uint)__cvta_generic_to_shared(b)) : "memory");
}
__device__ __forceinline__ void ready_arrive(unsigned long long* b) {
    asm volatile("{ .reg .b64 s; mbarrier.arrive.release.cta.shared.b64 s, [%0]; }" ::"r"(
                     (uint)__cvta_generic_to_shared(b))
                 : "memory");
}
__device__ __forceinline__ void ready_wait(unsigned long long* b, uint parity, EngineWords* words) {
    const uint a = (uint)__cvta_generic_to_shared(b);
    for (uint k = 0; k < kBarrierMaxPolls; k++) {
        uint ok;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.acquire.cta.shared.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(ok)
            : "r"(a), "r"(parity)
            : "memory");
        if (ok) return;
    }
    atomicOr(&words->status, kStBarrier);
}

__device__ __forceinline__ void cp16(void* dst, const void* src) {
    const uint d = (uint)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Starts the copies of tile t's states (step parity buffer cur) and tables
// into the stage at dst.
template <typename Real>
__device__ __forceinline__ void tile_stage(const TileArgs<Real>& T, uint t, uint4 h0, uint4 h1, uint first, uint m,
                                           const PRec<Real>* cur, unsigned char* dst) {
    constexpr uint NT = TileCap<Real>::P;
    constexpr uint C = sizeof(Real) == 4 ? 4 : 5;   // 16-byte words of a record
    const unsigned char* src = reinterpret_cast<const unsigned char*>(cur + first);
    for (uint c = threadIdx.x; c < m * C; c += NT) {
        const uint p = c / C, w = c % C;
        cp16(dst + p * (uint)sizeof(TileRec<Real>) + 16u * w, src + (size_t)p * sizeof(PRec<Real>) + 16u * w);
    }
    for (uint p = threadIdx.x; p < m; p += NT)
        cp16(dst + p * (uint)sizeof(TileRec<Real>) + 16u * C, T.tq + first + p);
    const TileTables L(m, h0.x, h0.y, h1.x, h1.y);
    const unsigned char* B = T.blob + (size_t)t * T.BB;
    unsigned char* d2 = dst + m * (uint)sizeof(TileRec<Real>);
    for (uint c = threadIdx.x; c < L.bytes / 16u; c += NT) cp16(d2 + 16u * c, B + 16u * c);
}

// MODE: the PCCP window, the same writing the adjoint's tape, or the PP window
// (k_window_pp, one thread through all of a sphere's pairs twice over, took 771
// us per 20-step window of a 60,001-sphere bed, this 226 and 50 for the lists)
// (a pair's force subtracted on hi; each particle's walls evaluated after its
// pairs and gravity, added to its force wall by wall, as pp_item and
// particle_finish do).
enum : int { kTilePccp = 0, kTileTape = 1, kTilePp = 2 };
template <typename Real, int MODE>
__global__ void __maxnreg__(TileCap<Real>::regs)
    k_tile(StepArgs<Real> a, TileArgs<Real> T, int K, StepPartials part, size_t clr1, uint* bar) {
    constexpr bool TAPE = MODE == kTileTape, PP = MODE == kTilePp;
    if ((a.ccw && !a.ccw[1]) || T.tw[kTwOver]) return;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ __align__(8) unsigned long long s_ready;
    const uint Q = T.Q;
    constexpr uint PC = TileCap<Real>::P;
    constexpr uint kTileThreads = PC;
    constexpr uint RS = sizeof(TileRec<Real>);
    typedef typename Two<Real>::T R2;
    const uint PT = T.tw[kTwP], nt = T.tw[kTwTiles], stage = T.tw[kTwStage], tid = threadIdx.x;
    R2* res = reinterpret_cast<R2*>(smem + (nt <= gridDim.x ? 1u : 2u) * stage);
    // this block's tiles: a block with one keeps its states in shared memory
    const uint nbound = a.bpos[a.n];
    uint t = blockIdx.x;
    const uint mine = t < nt ? (nt - t + gridDim.x - 1) / gridDim.x : 0u;
    double mz = 0.0;
    uint cnt = 0, flags = 0;
    if (mine) {
        ParticleCommon pc = a.pc;
        uint sb = 0;
        uint4 hd = T.head[2 * (size_t)t];
        uint4 hx = T.head[2 * (size_t)t + 1];
        uint seq = 0;   // tile-steps of this block
        uint tp0 = t;   // the tile stepped last, and the steps it has finished
        int sdone = 0;
        if (tid == 0) ready_init(&s_ready);
        tile_stage<Real>(T, t, hd, hx, t * PT, min(PT, nbound - t * PT), T.ts[0], smem);
        for (int s = 0; s < K;) {
            const bool last = s == K - 1;
            pc.first = s == 0 ? 1 : 0;
            const long long ts = TAPE ? (long long)a.tstep0 + s : -1ll;
            const PRec<Real>* cur = (s & 1) ? T.ts[1] : T.ts[0];
            PRec<Real>* nxt = (s & 1) ? T.ts[0] : T.ts[1];
            const uint first = t * PT;
            const uint m = min(PT, nbound - first);
            const uint nin = hd.x, tot = hd.y, nitem = hd.y + hd.z;
            unsigned char* S = smem + sb * stage;
            const TileTables L(m, nin, tot, hx.x, hx.y);
            const unsigned char* B = S + m * RS;
            const uint* te = reinterpret_cast<const uint*>(B);
            const uint* tx = reinterpret_cast<const uint*>(B + L.ox);
            const unsigned short* tr = reinterpret_cast<const unsigned short*>(B + L.orr);
            const uint4* tps = reinterpret_cast<const uint4*>(B + L.op);
            const size_t q0 = (size_t)t * Q;
            double *hx0 = T.th.x + q0, *hy0 = T.th.y + q0, *hz0 = T.th.z + q0;
            cp_wait_all();
            __syncthreads();   // the tile's stage is filled, its states written; the other stage and the results are free
            // the next tile of this block (the next step's first one after the last)
            uint tn = t;
            int sn = s + 1;
            uint4 hn = hd;
            uint4 hxn = hx;
            if (mine > 1) {
                tn += gridDim.x;
                if (tn >= nt) tn = blockIdx.x;
                hn = T.head[2 * (size_t)tn];
                sn = tn > t ? s : s + 1;
                hxn = T.head[2 * (size_t)tn + 1];
                if (sn < K) {
                    sb ^= 1u;
                    tile_stage<Real>(T, tn, hn, hxn, tn * PT, min(PT, nbound - tn * PT),
                                     (sn & 1) ? T.ts[1] : T.ts[0], smem + sb * stage);
                }
            }
            // the last warp (the one with the fewest items) publishes the
            // states the block wrote last, then waits until the neighbour
            // tiles have written theirs of this step, and tells the block
            if (tid >= kTileThreads - 32) {
                if (tid == kTileThreads - 32 && seq > 0 && sdone < K)
                    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(T.flag + (size_t)tp0 * kFlagStride),
                                 "r"((uint)sdone)
                                 : "memory");
                __syncwarp();
                if (s > 0) {
                    const uint* tnb = reinterpret_cast<const uint*>(B + L.on);
                    for (uint j = tid & 31u; j < hx.y; j += 32u)
                        tile_wait(T.flag + (size_t)tnb[j] * kFlagStride, (uint)s, bar + kBarGiveUp, a.words);
                }
                __syncwarp();
                if (tid == kTileThreads - 32) ready_arrive(&s_ready);
            }
            // histories of this thread's first pair; the next one's are loaded
            // while a pair is evaluated
            V3<double> h = zero3<double>();
            if (s > 0 && tid < tot) h = mk(hx0[tid], hy0[tid], hz0[tid]);
            for (uint u = tid; u < nitem; u += kTileThreads) {
                if (u < tot) {
                    const uint ent = te[u];
                    uint k = 0;
                    if (TAPE || s == 0 || last) k = T.tk[q0 + u];
                    V3<double> hn = zero3<double>();
                    if (s == 0) {
                        const uint kk = k & 0x7fffffffu;
                        h = mk(ldx<true>(a.H.x + kk), ldx<true>(a.H.y + kk), ldx<true>(a.H.z + kk));
                    } else if (u + kTileThreads < tot) {
                        const uint un = u + kTileThreads;
                        hn = mk(hx0[un], hy0[un], hz0[un]);
                    }
                    const bool own = !(k >> 31);
                    if (TAPE && own) {
                        double* th = a.th + 3 * a.cap * ts;
                        th[k] = h.x; th[a.cap + k] = h.y; th[2 * a.cap + k] = h.z;
                    }
                    V3<double> xi, di, xj, dj;
                    V3<Real> ai, aj;
                    Real ri, rj;
                    lds_rec(reinterpret_cast<const PRec<Real>*>(S + (ent & 511u) * RS), xi, di, ai, ri);
                    // a pair across tiles is evaluated from the own particle's
                    // side; when that is hi, the history (lo's) and the
                    // results change sign, which changes no other bit
                    bool hi = false;
                    if (u < nin) {
                        lds_rec(reinterpret_cast<const PRec<Real>*>(S + ((ent >> 9) & 511u) * RS), xj, dj, aj, rj);
                    } else {
                        const PRec<Real>* o = cur + tx[u - nin];
                        hi = (ent & 512u) != 0u;
                        if (hi) h = -h;
                        ready_wait(&s_ready, seq & 1u, a.words);
                        ld_rec<true>(o, xj, dj, aj, rj);
                    }
                    V3<Real> Fi = zero3<Real>(), Ti = zero3<Real>(), Tj = zero3<Real>();
                    const int c = pair_eval<Real>(xi, xj, di, dj, ai, aj, ri, rj, h, a.pp, a.inv_dt, a.density, Fi, Ti,
                                                  Tj);
                    if (hi) {
                        h = -h;
                        Fi = -Fi;
                        Tj = Ti;
                    }
                    if (last) {
                        if (own) { T.Ho.x[k] = h.x; T.Ho.y[k] = h.y; T.Ho.z[k] = h.z; }
                    } else {
                        hx0[u] = h.x; hy0[u] = h.y; hz0[u] = h.z;
                    }
                    // without contact zeros: adding them to a sum that started
                    // from +0 changes no bit
                    R2* o = res + 5 * (ent >> 18);
                    if (!c) Fi = Ti = Tj = zero3<Real>();
                    o[0] = mk2(Fi.x, Fi.y);
                    o[1] = mk2(Fi.z, Ti.x);
                    o[2] = mk2(Ti.y, Ti.z);
                    o[3] = mk2(Tj.x, Tj.y);
                    o[4] = mk2(Tj.z, c ? (Real)1 : (Real)0);
                    h = hn;
                } else {
                    const uint p = T.twl[(size_t)t * PC + (u - tot)];
                    const uint i = tps[p].w;
                    V3<double> x, d;
                    V3<Real> av;
                    Real r;
                    lds_rec(reinterpret_cast<const PRec<Real>*>(S + p * RS), x, d, av, r);
                    const Real mass = a.density * (Real)8 * r * r * r;
                    V3<double> hw = ld3p<true>(a.W, i);
                    if (TAPE) {
                        double* w = a.twh + 3 * a.tnp * ts;
                        w[i] = hw.x; w[a.tnp + i] = hw.y; w[2 * a.tnp + i] = hw.z;
                    }
                    V3<Real> Fw = zero3<Real>(), Tw = zero3<Real>();
                    wall_contacts<Real>(a.pc.hx, a.pc.hy, x, cvt<Real>(d), av, r, mass, hw, a.inv_dt, a.pw, Fw, Tw,
                                        (Real*)nullptr);
                    a.W.x[i] = hw.x; a.W.y[i] = hw.y; a.W.z[i] = hw.z;
                    R2* o = res + 5 * u;
                    o[0] = mk2(Fw.x, Fw.y);
                    o[1] = mk2(Fw.z, Tw.x);
                    o[2] = mk2(Tw.y, Tw.z);
                }
            }
            __syncthreads();
            uint4 tp = make_uint4(0u, 0u, kEmpty, kEmpty);
            if (tid < m) tp = tps[tid];
            if (tp.w != kEmpty) {
                const uint i = tp.w;
                V3<double> x, d;
                V3<Real> av;
                Real r;
                TileRec<Real>* sp = reinterpret_cast<TileRec<Real>*>(S + tid * RS);
                lds_rec(reinterpret_cast<const PRec<Real>*>(sp), x, d, av, r);
                float4 q = sp->q;
                if (TAPE) {   // state before the step
                    const long long np = a.tnp, o = 3 * np * ts;
                    a.tx[o + i] = x.x; a.tx[o + np + i] = x.y; a.tx[o + 2 * np + i] = x.z;
                    a.td[o + i] = d.x; a.td[o + np + i] = d.y; a.td[o + 2 * np + i] = d.z;
                    a.ta[o + i] = av.x; a.ta[o + np + i] = av.y; a.ta[o + 2 * np + i] = av.z;
                }
                V3<Real> F = zero3<Real>(), M = zero3<Real>();
                uint ci = 0;
                const bool count = TAPE || last;
                for (uint e = tp.x & 0xffffu, e1 = e + (tp.x >> 16); e < e1; e++) {
                    const R2* o = res + 5 * e;
                    const R2 v0 = o[0], v1 = o[1], v2 = o[2];
                    F.x += v0.x; F.y += v0.y; F.z += v1.x;
                    M.x += v1.y; M.y += v2.x; M.z += v2.y;
                    if (count) ci += o[4].y != (Real)0 ? 1u : 0u;
                }
                for (uint v = tp.y & 0xffffu, v1e = v + (tp.y >> 16); v < v1e; v++) {
                    const R2* o = res + 5 * (uint)tr[v];
                    const R2 v0 = o[0], v1 = o[1], v3 = o[3], v4 = o[4];
                    F.x += -v0.x; F.y += -v0.y; F.z += -v1.x;
                    M.x += v3.x; M.y += v3.y; M.z += v4.x;
                    if (count) ci += v4.y != (Real)0 ? 1u : 0u;
                }
                F.z += -sphere_mass(a.density, r);
                const Real mass = sphere_mass(a.density, r);
                uint wflag = __float_as_uint(q.w);
                if (PP) {
                    const double rd = (double)r;
                    const bool touch = (x.z < rd) || (x.x + pc.hx < rd) || (pc.hx - x.x < rd) || (x.y + pc.hy < rd) ||
                                       (pc.hy - x.y < rd);
                    if (touch || wflag) {
                        V3<double> hw = wflag ? ld3p<true>(a.W, i) : zero3<double>();
                        const int hit = wall_contacts<Real>(pc.hx, pc.hy, x, cvt<Real>(d), av, r, mass, hw, a.inv_dt, a.pw,
                                                            F, M, (Real*)nullptr);
                        a.W.x[i] = hw.x; a.W.y[i] = hw.y; a.W.z[i] = hw.z;
                        wflag = hit ? 1u : 0u;
                    }
                } else if (tp.z != kEmpty) {
                    const R2* o = res + 5 * tp.z;
                    const R2 v0 = o[0], v1 = o[1], v2 = o[2];
                    F.x += v0.x; F.y += v0.y; F.z += v1.x;
                    M.x += v1.y; M.y += v2.x; M.z += v2.y;
                }
                if (TAPE) {
                    double* f = a.tF + 3 * a.tnp * ts;
                    double* g = a.tT + 3 * a.tnp * ts;
                    f[3 * i] = F.x; f[3 * i + 1] = F.y; f[3 * i + 2] = F.z;
                    g[3 * i] = M.x; g[3 * i + 1] = M.y; g[3 * i + 2] = M.z;
                    a.tc[a.tnp * ts + i] = ci;
                }
                const Real I = (Real)0.4 * mass * (r * r);
                if (pc.first) { q.x = 0.f; q.y = 0.f; q.z = 0.f; }
                double mzi;
                integrate<Real>(F, M, mass, I, pc.dt, a.dtr, pc.half_skin2, x, d, av, q, flags, mzi);
                q.w = __uint_as_float(wflag);
                if (last) {
                    st_rec(T.So + i, x, d, av, r);
                    a.Q[i] = q;
                    mz = fmax(mz, mzi);
                    cnt += ci;
                } else {
                    sts_rec(reinterpret_cast<PRec<Real>*>(sp), x, d, av, r);
                    sp->q = q;
                }
            }
            // a warp writes its particles' new states out together (whole
            // lines; a store per lane and field touched a line per lane)
            const uint w0 = tid & ~31u;
            if (!last && w0 < m) {
                constexpr uint C = sizeof(Real) == 4 ? 4 : 5;
                const uint nrow = min(32u, m - w0), lane = tid & 31u;
                __syncwarp();
                unsigned char* dst = reinterpret_cast<unsigned char*>(nxt + first + w0);
                for (uint c = lane; c < nrow * C; c += 32u) {
                    const uint p = c / C, w = c % C;
                    *reinterpret_cast<uint4*>(dst + (size_t)p * sizeof(PRec<Real>) + 16u * w) =
                        *reinterpret_cast<const uint4*>(S + (w0 + p) * RS + 16u * w);
                }
                if (mine > 1 && lane < nrow)
                    T.tq[first + tid] = reinterpret_cast<const TileRec<Real>*>(S + tid * RS)->q;
            }
            tp0 = t;
            sdone = s + 1;
            t = tn;
            s = sn;
            hd = hn;
            hx = hxn;
            seq++;
        }
    }
    block_observables(mz, cnt, flags, 1, part, a.words);
    clear_partials(part, gridDim.x, clr1);
}
