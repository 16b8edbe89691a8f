// SPH: fixed-radius neighbour search and variable smoothing length (the pair
// sums over the neighbour lists are in sph_pairs.cu).
//
// Neighbour search: the reference walks the tree once per particle with a
// per-thread stack (SPH::fixedRadiusNN, src/sph/sph.cu:93-281).  Here a warp
// walks once for 32 consecutive SFC-sorted particles, lane-parallel over a
// shared-memory stack, stages the particles of overlapping leaves and small
// cells as candidates, keeps those that can reach one of the warp's four
// 8-particle sub-groups, and tests each sub-group's particles only against
// its own candidates with the reference's pair rule d^2 < h_i^2 && d^2 < h_j^2
// (j != i), d^2 formed without FMA contraction like the reference build.  All
// pruning is conservative, so the neighbour set equals the brute-force set.
#include <algorithm>

#include "sph.cuh"
#include "walk.cuh"

namespace {

constexpr int kBlock = 128;
constexpr int kWarps = kBlock / 32;
// cells with at most this many particles are staged whole (8: 4 % slower, 4: 20 %)
constexpr int kSmall = 16;
// Gap between consecutive particles, in h, at which a group is cut.  Variable h
// of a 2^20 cloud in us, uncut / 2 / 1.5 / 1 / 0.7: 3870 / 3600 / 3440 / 3390 /
// 3400; list walk of a 35,937 lattice 95 / 95 / 107 / 115 / 212, of larger lattices
// the same from 1 on.  Where h is no longer than the spacing every gap is longer
// than that: a cut must also be kCutMean times the mean of the group's other gaps,
// and while there are more than kMaxCuts the gap asked for is doubled.  List walk
// in us, uncut / 1.5 h alone / now: lattice of 262,144 at h = 0.4 and 1 spacings 48 /
// 633 / 59 and 71 / 96 / 89, of 1,000,000 at 0.4 1814 / 2543 / 243, uniform ball of
// 1,000,000 at 0.4 and 2 neighbours 10600 / 1846 / 440 and 10300 / 815 / 634.  (Means
// times 2.5: 66 us at 262,144, 0.4; times 4: a Plummer sphere of 20,000 in groups of
// 8 stays uncut, 316 against 48.  2 cuts: 100,000 at 60 neighbours 176 against 167.)
constexpr double kCut = 1.5, kCutMean = 3.0;
constexpr int kMaxCuts = 3;

// ------------------------------------------------------------ FRNN walk
// One warp per 32 consecutive (sorted or listed) particles, lane = particle,
// four sub-groups of 8 lanes.
//
// Traversal: lane-parallel over a per-warp stack in shared memory.  Every
// step pops up to 32 nodes, one per lane; a node whose particle box is farther
// from the box of the group's particles than the group's largest h, or than
// the largest h below the node, is dropped; leaves, cells of
// at most kSmall particles and shared-key buckets become candidate ranges;
// other cells push their children.  Stack bound as in the gravity list walk:
// a pop of k nodes pushes at most 8k, and k is limited so that a depth-first
// descent (7 per level, 22 levels) always fits on top of the stack.
//
// Candidates: the ranges are expanded 32 at a time; each candidate particle
// is tested against the four sub-groups: its distance from the sub-group's box
// must be below h_j and the sub-group's largest h, both with the rounding of
// the FP32 offsets on top, so no pair that passes the exact test is dropped.
// (Distances, not boxes grown by h: a box of side s grown by r on all sides
// holds (s + 2 r)^3, the points within r of it a quarter less at s = 0.75 r,
// and the pairs to test are proportional to that.)
// Candidates reaching some sub-group go to a shared-memory pool (x, y, z
// relative to the group's centre and h_j^2, in FP32, and j) and to that
// sub-group's list.  A full pool is flushed: for each sub-group, lane (8q + p)
// tests particle p of the sub-group against list entry 4c + q, so the warp
// tests 32 pairs per step, and hits are written in list order (ballot prefix
// over the 4 lanes of a particle).
//
// The pair rule is the reference's, d^2 < h_i^2 && d^2 < h_j^2 (j != i), d^2
// formed without FMA contraction in FP64.  The flush forms d^2 in FP32 and
// settles the pairs whose d^2 is farther from min(h_i^2, h_j^2) than the FP32
// error; the few others are tested exactly.  With H the group's largest h and
// R its half edge plus H (the reach of every candidate), offsets
// are off by 2^-24 R each, so d^2 for d <= 2 H by less than 8.3e-7 R H +
// 1.3e-6 H^2, and a pair farther apart cannot come within that of H^2 while
// R < 1e5 H.  The walk and the box tests are conservative too, so each
// neighbour set equals the brute-force set.
// Bound: issue (64 to 72 % of the slots, ALU pipe 52 to 58 %) and fixed latency, 23
// warps active of the 28 resident per SM.  List walk in us with FP64 tests and grown boxes / now: Sedov lattice of
// 262,144 particles 258 / 203, of 2,097,152 1693 / 1303; all walks of a cloud step,
// 2^20 particles 2229 / 1500, 2^23 16600 / 10500.  Of the 1303: the tree walk 334,
// staging the candidates 180, pair tests and list writes 790.
//
// mode 0: write lists (h_i = h[i], h_j = h[j]) for all particles; mode 1:
// count only, with h_i = h[i], h_j = h[j] (the variable-h sweep passes the
// sweep's snapshot as h), for the particles of `list` (list_count entries, in
// sorted order, so 32 consecutive entries are still spatially close); mode 2:
// mode 0 for the variable-h iteration on lists: runs only when *gate is
// nonzero, and a count above maxnb (the list keeps its first maxnb entries,
// noi the full count) sets *trunc instead of an error; no statistics.
constexpr int kStack = 512;
constexpr int kReserve = 7 * 22 + 8;
constexpr int kPool = 128;

struct FrnnSmem {
    int stk[kStack];
    float4 cp[kPool];                                     // candidate: offset from the centre, h_j^2
    int cj[kPool];                                        // candidate particle
    unsigned char lst[4][kPool];                          // pool slots per sub-group
    int rf[32];                                           // staged ranges: first particle less begin
    float4 slo[4], shi[4];                                // sub-group boxes about the centre; largest h (.w)
};

#ifndef MHPC_FRNN_MIN_BLOCKS
#define MHPC_FRNN_MIN_BLOCKS 7
#endif
template <int MODE>
// 7 blocks per SM: the list walk of 2,097,152 particles in us with 5 / 6 / 7: 1632 /
// 1496 / 1432 (the extra warps hide more of the walk's latency)
__global__ void __launch_bounds__(kBlock, MHPC_FRNN_MIN_BLOCKS) k_frnn(TreeDev T, int n, int ppw, int maxnb, const double* __restrict__ sx,
                                                 const double* __restrict__ sy, const double* __restrict__ sz,
                                                 const double* __restrict__ sh, const int* __restrict__ list,
                                                 const int* __restrict__ list_count,
                                                 const float* __restrict__ node_hmax, int* __restrict__ nbr,
                                                 int* __restrict__ noi, DevStatus* st,
                                                 const int* __restrict__ gate = nullptr, int* trunc = nullptr) {
    __shared__ FrnnSmem smem[kWarps];
    if (st->code) return;
    if (MODE == 2 && *gate == 0) return;
    const int M = *T.nodes;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    FrnnSmem& S = smem[w];
    const long total = MODE == 1 ? (long)*list_count : (long)n;
    // one group per warp (a gated re-walk that mostly returns at once has a
    // smaller grid and takes several)
    for (long g = ((long)blockIdx.x * kBlock + threadIdx.x) >> 5; g * ppw < total; g += (long)gridDim.x * kWarps) {
    long s = g * ppw + lane;
    const bool valid = lane < ppw && s < total;
    if (MODE == 1) s = valid ? list[s] : 0;
    int k = 0;     // neighbours found for this lane's particle
    // The curve jumps between cells of the tree: a group across such a place would
    // walk the whole box between its two ends.  It is cut where two consecutive
    // particles are far apart, and its parts walk one after the other.
    unsigned rest = __ballot_sync(MHPC_FULL, valid);
    unsigned cuts;
    {
        double px = 0, py = 0, pz = 0, hm = 0;
        if (valid) { px = sx[s]; py = sy[s]; pz = sz[s]; hm = sh[s]; }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) hm = fmax(hm, __shfl_xor_sync(MHPC_FULL, hm, o));
        const double nx = __shfl_down_sync(MHPC_FULL, px, 1), ny = __shfl_down_sync(MHPC_FULL, py, 1);
        const double nz = __shfl_down_sync(MHPC_FULL, pz, 1);
        const bool next = lane < 31 && ((rest >> (lane + 1)) & 1u);
        const double gap = fmax(fmax(fabs(nx - px), fabs(ny - py)), fabs(nz - pz));
        double far = kCut * hm;
        cuts = __ballot_sync(MHPC_FULL, next && gap > far);
        if (cuts) {
            float sum = next ? (float)gap : 0.f, top = sum;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                sum += __shfl_xor_sync(MHPC_FULL, sum, o);
                top = fmaxf(top, __shfl_xor_sync(MHPC_FULL, top, o));
            }
            far = fmax(far, kCutMean * (double)((sum - top) / (float)max(__popc(rest) - 2, 1)));
            cuts = __ballot_sync(MHPC_FULL, next && gap > far);
            for (int k = 0; __popc(cuts) > kMaxCuts; ++k) {
                far *= 2.0;
                cuts = k < 10 ? __ballot_sync(MHPC_FULL, next && gap > far) : 0u;
            }
        }
    }
    while (rest) {
    const unsigned after = cuts & ~((1u << (__ffs(rest) - 1)) - 1u);
    const unsigned part = after ? rest & (2u * (after & (0u - after)) - 1u) : rest;
    rest &= ~part;
    cuts &= ~part;
    const bool active = (part >> lane) & 1u;
    double px = 0, py = 0, pz = 0, hi = 0;
    if (active) { px = sx[s]; py = sy[s]; pz = sz[s]; hi = sh[s]; }
    // points box and largest h over the sub-group (8 lanes), then over the warp
    double hm = active ? hi : 0.0, shm = 0.0;
    double sl[3] = {}, su[3] = {};  // the sub-group's box
    double plx = active ? px : 1e300, ply = active ? py : 1e300, plz = active ? pz : 1e300;
    double pux = active ? px : -1e300, puy = active ? py : -1e300, puz = active ? pz : -1e300;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        plx = fmin(plx, __shfl_xor_sync(MHPC_FULL, plx, o));
        ply = fmin(ply, __shfl_xor_sync(MHPC_FULL, ply, o));
        plz = fmin(plz, __shfl_xor_sync(MHPC_FULL, plz, o));
        pux = fmax(pux, __shfl_xor_sync(MHPC_FULL, pux, o));
        puy = fmax(puy, __shfl_xor_sync(MHPC_FULL, puy, o));
        puz = fmax(puz, __shfl_xor_sync(MHPC_FULL, puz, o));
        hm = fmax(hm, __shfl_xor_sync(MHPC_FULL, hm, o));
        if (o == 4) {
            sl[0] = plx; sl[1] = ply; sl[2] = plz; su[0] = pux; su[1] = puy; su[2] = puz;
            shm = hm;
        }
    }
    const float3 g0 = make_float3(__double2float_rd(plx), __double2float_rd(ply), __double2float_rd(plz));
    const float3 g1 = make_float3(__double2float_ru(pux), __double2float_ru(puy), __double2float_ru(puz));
    const double cx = 0.5 * (plx + pux), cy = 0.5 * (ply + puy), cz = 0.5 * (plz + puz);
    const float fx = (float)(px - cx), fy = (float)(py - cy), fz = (float)(pz - cz), fh2 = (float)(hi * hi);
    const float H = __double2float_ru(hm);
    const float R = 1.00001f * ((float)fmax(fmax(pux - cx, puy - cy), puz - cz) + H);
    // |d^2(FP32) - min(h_i^2, h_j^2)| up to which the exact test decides, and what
    // the rounding of the offsets adds to a distance; at scales where the bounds
    // do not hold, every candidate goes to every sub-group's exact test
    const bool scaled = H > 1e-15f && R < 1e15f && R < 1e5f * H;
    const float band = scaled ? 1e-6f * R * H + 1.6e-6f * H * H : INFINITY;
    const float slack = scaled ? 3e-7f * R : INFINITY;
    // a sub-group's box about the centre, and its largest h
    if ((lane & 7) == 0) {
        const int q = lane >> 3;
        const float ax = __double2float_rd(sl[0] - cx), ay = __double2float_rd(sl[1] - cy), az = __double2float_rd(sl[2] - cz);
        const float bx = __double2float_ru(su[0] - cx), by = __double2float_ru(su[1] - cy), bz = __double2float_ru(su[2] - cz);
        const bool any = shm > 0.0;
        S.slo[q] = make_float4(ax, ay, az, any ? 1.000001f * __double2float_ru(shm) + slack : -1.f);
        S.shi[q] = make_float4(bx, by, bz, 0.f);
    }
    int pool = 0;  // pool entries (warp-uniform)
    int cnt0 = 0, cnt1 = 0, cnt2 = 0, cnt3 = 0;  // list entries per sub-group (warp-uniform)
    auto flush = [&]() {
        __syncwarp();
        const int q = lane >> 3, p = lane & 7;
#pragma unroll 1
        for (int sg = 0; sg < 4; ++sg) {
            const int cntg = sg == 0 ? cnt0 : sg == 1 ? cnt1 : sg == 2 ? cnt2 : cnt3;
            const int src = 8 * sg + p;
            const float ix = __shfl_sync(MHPC_FULL, fx, src), iy = __shfl_sync(MHPC_FULL, fy, src);
            const float iz = __shfl_sync(MHPC_FULL, fz, src), ih2 = __shfl_sync(MHPC_FULL, fh2, src);
            const int is = __shfl_sync(MHPC_FULL, (int)s, src);
            const int mine = __shfl_sync(MHPC_FULL, (int)active, src) ? cntg : 0;  // entries to test
            int kb = __shfl_sync(MHPC_FULL, k, src);
            const unsigned pmask = 0x01010101u << p;
            int* const row = nbr + nb_index(is, 0, maxnb);
            // two entries per lane and step: their loads and sums overlap
            for (int c0 = 0; c0 < cntg; c0 += 8) {
                bool hit[2], near[2];
                int j[2];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int c = c0 + 4 * u + q;
                    hit[u] = near[u] = false;
                    j[u] = is;
                    if (c < mine) {
                        const int slot = S.lst[sg][c];
                        j[u] = S.cj[slot];
                        const float4 q4 = S.cp[slot];
                        const float dx = ix - q4.x, dy = iy - q4.y, dz = iz - q4.z;
                        const float over = fmaf(dx, dx, fmaf(dy, dy, dz * dz)) - fminf(ih2, q4.w);
                        hit[u] = over < -band;
                        near[u] = !(fabsf(over) > band);
                    }
                }
                if (near[0] || near[1]) {
                    const double hs = sh[is], xs = sx[is], ys = sy[is], zs = sz[is];
#pragma unroll
                    for (int u = 0; u < 2; ++u)
                        if (near[u]) {
                            const double hj = sh[j[u]];
                            const double d = d2_exact(xs - sx[j[u]], ys - sy[j[u]], zs - sz[j[u]]);
                            hit[u] = d < hs * hs && d < hj * hj;
                        }
                }
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    hit[u] = hit[u] && j[u] != is;
                    const unsigned b = __ballot_sync(MHPC_FULL, hit[u]) & pmask;
                    if (MODE != 1 && hit[u]) {
                        const int pos = kb + __popc(b & lt);
                        if (pos < maxnb) row[32 * pos] = j[u];
                    }
                    kb += __popc(b);
                }
            }
            // lane p (q = 0) holds particle 8 sg + p's count: its owner takes it
            const int knew = __shfl_sync(MHPC_FULL, kb, p);
            if (q == sg) k = knew;
        }
        __syncwarp();
        pool = 0;
        cnt0 = cnt1 = cnt2 = cnt3 = 0;
    };
    // the root's children: node 0 and its skip chain
    int top = 0;
    if (lane == 0) {
        int c = 0;
        while (c < M && top < 8) { S.stk[top++] = c; c = __ldg(&T.link[c].x); }
        if (c < M) set_status(st, MHPC_ERR_DEPTH, 3);
    }
    top = __shfl_sync(MHPC_FULL, top, 0);
    __syncwarp();
    while (top > 0) {
        const int room = (kStack - kReserve - top) / 7;
        int kk = top < 32 ? top : 32;
        if (kk > room) kk = room > 1 ? room : 1;
        const bool act = lane < kk;
        const int nd = act ? S.stk[top - 1 - lane] : 0;
        __syncwarp();
        top -= kk;
        int rf = 0, rlen = 0, kmask = 0;
        if (act) {
            const int2 lk = __ldg(T.link + nd);
            const float4 bl = __ldg(T.bmin + nd), bh = __ldg(T.bmax + nd);
            // a pair needs d < h_i and d < h_j: the boxes must come within both
            const float lim = node_hmax ? fminf(H, __ldg(node_hmax + nd)) : H;
            if (box_gap2(g0, g1, bl, bh) <= __fmul_ru(lim, lim)) {
                rf = __ldg(T.first + nd);
                if (lk.y & ND_LEAF) {
                    rlen = 1;
                } else {
                    const int l = __ldg(T.last + nd);
                    const int km = __ldg(T.kmask + nd);
                    // small cells and shared-key buckets (all particles share
                    // one key) are staged whole; other cells open
                    if (l - rf + 1 <= kSmall || (km & 0x100)) rlen = l - rf + 1;
                    else kmask = km & 0xff;
                }
            }
        }
        // push the children of opened cells
        // (one scan for the children, at most 256, and for the staged ranges;
        // ranges above 65,536 particles, a shared-key bucket's, by a second one)
        const int nkid = __popc(kmask);
        const bool wide = __any_sync(MHPC_FULL, rlen > 65536);
        const int both = warp_scan(nkid | (wide ? 0 : rlen << 9), lane);
        const int incl = both & 511;
        const int rincl = wide ? warp_scan(rlen, lane) : both >> 9;
        const int total = __shfl_sync(MHPC_FULL, incl, 31);
        if (top + total > kStack) {
            // unreachable by the bound on kk; stop instead of overrunning
            if (lane == 0) set_status(st, MHPC_ERR_DEPTH, 4);
            return;
        }
        if (nkid) {
            const int4 k0 = __ldg(reinterpret_cast<const int4*>(T.kids + 8 * (size_t)nd));
            const int4 k1 = __ldg(reinterpret_cast<const int4*>(T.kids + 8 * (size_t)nd) + 1);
            const int all[8] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w};
            int wpos = top + incl - nkid;
#pragma unroll
            for (int d = 0; d < 8; ++d)
                if ((kmask >> d) & 1) S.stk[wpos++] = all[d];
        }
        top += total;
        // staged ranges: compact, each with its first particle less its begin
        const int begin = rincl - rlen;
        const int ncand = __shfl_sync(MHPC_FULL, rincl, 31);
        const unsigned br = __ballot_sync(MHPC_FULL, rlen > 0);
        if (rlen > 0) S.rf[__popc(br & lt)] = rf - begin;
        __syncwarp();
        int begun = 0;  // ranges that begin before this batch
        for (int c0 = 0; c0 < ncand; c0 += 32) {
            if (pool + 32 > kPool) flush();
            const int c = c0 + lane;
            int mask = 0, j = 0;
            float rx = 0.f, ry = 0.f, rz = 0.f;
            double hj = 0;
            // a lane's range is the last that begins at or before it
            const unsigned at = (unsigned)(begin - c0);
            const unsigned bits = __reduce_or_sync(MHPC_FULL, rlen > 0 && at < 32u ? 1u << at : 0u);
            if (c < ncand) {
                j = S.rf[begun + __popc(bits & (2u * lt + 1u)) - 1] + c;
                const double qx = __ldg(sx + j), qy = __ldg(sy + j), qz = __ldg(sz + j);
                hj = __ldg(sh + j);
                rx = (float)(qx - cx); ry = (float)(qy - cy); rz = (float)(qz - cz);
                const float hf = 1.000001f * (float)hj + slack;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float4 a = S.slo[q], b = S.shi[q];
                    const float gx = fmaxf(fmaxf(a.x - rx, rx - b.x), 0.f), gy = fmaxf(fmaxf(a.y - ry, ry - b.y), 0.f),
                                gz = fmaxf(fmaxf(a.z - rz, rz - b.z), 0.f);
                    const float lim = fminf(a.w, hf);
                    mask |= (int)(lim > 0.f && fmaf(gx, gx, fmaf(gy, gy, gz * gz)) <= lim * lim) << q;
                }
            }
            const unsigned b0 = __ballot_sync(MHPC_FULL, mask & 1), b1 = __ballot_sync(MHPC_FULL, mask & 2);
            const unsigned b2 = __ballot_sync(MHPC_FULL, mask & 4), b3 = __ballot_sync(MHPC_FULL, mask & 8);
            const unsigned bp = b0 | b1 | b2 | b3;
            if (mask) {
                const int slot = pool + __popc(bp & lt);
                S.cp[slot] = make_float4(rx, ry, rz, (float)(hj * hj));
                S.cj[slot] = j;
                if (mask & 1) S.lst[0][cnt0 + __popc(b0 & lt)] = (unsigned char)slot;
                if (mask & 2) S.lst[1][cnt1 + __popc(b1 & lt)] = (unsigned char)slot;
                if (mask & 4) S.lst[2][cnt2 + __popc(b2 & lt)] = (unsigned char)slot;
                if (mask & 8) S.lst[3][cnt3 + __popc(b3 & lt)] = (unsigned char)slot;
            }
            begun += __popc(bits);
            cnt0 += __popc(b0); cnt1 += __popc(b1); cnt2 += __popc(b2); cnt3 += __popc(b3);
            pool += __popc(bp);
        }
        __syncwarp();
    }
    flush();
    }
    if (valid) {
        noi[s] = k;
        if (MODE == 0 && k > maxnb) set_status(st, MHPC_ERR_NEIGHBOURS, (int)s);
        if (MODE == 2 && k > maxnb) *trunc = 1;
        if (MODE == 0) atomicMax(&st->max_noi, k);
    }
    if (MODE == 0) {
        unsigned long long tot = valid ? (unsigned long long)k : 0ULL;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(MHPC_FULL, tot, o);
        if (lane == 0) atomicAdd(&st->noi_sum, tot);
    }
    }
}

// Count walk for sparse lists (later variable-h sweeps, where the particles
// still iterating are scattered, so a shared group box would be large): one
// warp per particle (warp_walk), its lanes testing 32 candidates at a time
// with the reference's pair rule.  The longest walks (particles with a large
// h) set a sweep's time, so each particle gets a whole warp.
struct CountVisit {
    const double *sx, *sy, *sz, *sh;
    double px, py, pz, hi2;
    long s;
    int* k;
    __device__ void operator()(int j) const {
        if (j == s) return;
        const double d = d2_exact(px - __ldg(sx + j), py - __ldg(sy + j), pz - __ldg(sz + j));
        const double hj = __ldg(sh + j);
        *k += (d < hi2 && d < hj * hj);
    }
};

__global__ void __launch_bounds__(kBlock) k_count_warp(TreeDev T, const double* __restrict__ sx,
                                                       const double* __restrict__ sy, const double* __restrict__ sz,
                                                       const double* __restrict__ sh, const int* __restrict__ list,
                                                       const int* __restrict__ list_count,
                                                       const float* __restrict__ node_hmax, int* __restrict__ count,
                                                       DevStatus* st) {
    __shared__ int stk[kWarps][kWalkStack];
    __shared__ int rfs[kWarps][32];
    if (st->code) return;
    const int M = *T.nodes;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long cnt = *list_count;
    const long nwarps = (long)gridDim.x * kWarps;
    for (long q = ((long)blockIdx.x * kBlock + threadIdx.x) >> 5; q < cnt; q += nwarps) {
        const int s = list[q];
        const double px = sx[s], py = sy[s], pz = sz[s], hi = sh[s];
        int k = 0;
        CountVisit v{sx, sy, sz, sh, px, py, pz, hi * hi, (long)s, &k};
        warp_walk(T, M, true, px, py, pz, hi, node_hmax, stk[w], rfs[w], st, v);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) k += __shfl_xor_sync(MHPC_FULL, k, o);
        if (lane == 0) count[s] = k;
        __syncwarp();
    }
}

// ------------------------------------------------------- variable h update
// Convergence rule and update of fixedRadiusNN_variableSML
// (src/sph/sph.cu:911-933): stop when nit > max_iter or |n - target| < tol,
// provided n < maxnb; otherwise h *= 0.5 (1 + (target / max(n,1))^(1/3)).
//
// The sweep's counts are complete when this runs, so the new h goes straight
// into the snapshot too (hold), and a larger h raises the largest-h bound of
// the particle's leaf and ancestors (grow-only, stopping at the first ancestor
// already as large; a bound left larger than the subtree's h only prunes less).
// *next_count (when given) is zeroed; at sweep 1 of the list form the particles
// still iterating are recorded (the fallback count when the first sweep started
// from predicted smoothing lengths).
__global__ void k_vh_update(const int* __restrict__ list, const int* __restrict__ list_count, int* next_count,
                            DevStatus* record, int n, const int* __restrict__ count, double* h, double* hold, int* done, int* nit, int target,
                            int tol, int max_iter, int maxnb, float* node_hmax, const int* __restrict__ leaf_node,
                            const int* __restrict__ parent, const long long* __restrict__ ord) {
    const int m = *list_count;
    // h never grows past the edge of the (cubic) bounding box: a particle whose
    // neighbours' h do not reach it (an isolated or ejected particle) would
    // otherwise multiply its h by up to 2.46 per sweep, without bound across
    // steps (the reference has no such bound); at the box edge its search
    // already covers every particle.
    const double hcap = ord_to_dbl(ord[1]) - ord_to_dbl(ord[0]);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (next_count) *next_count = 0;
        if (record) { record->predictor_fallback = m; record->predictor_used = n - m; }
    }
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < m; q += gridDim.x * blockDim.x) {
        const int i = list[q];
        const int it = ++nit[i];
        const int c = count[i];
        if ((it > max_iter || abs(c - target) < tol) && c < maxnb) {
            done[i] = 1;
        } else {
            const int cc = c < 1 ? 1 : c;
            const double h0 = h[i];
            const double hn = fmin(h0 * (0.5 * (1.0 + pow((double)target / (double)cc, 1. / 3.))), fmax(hcap, h0));
            h[i] = hn;
            hold[i] = hn;
            if (hn > h0) {
                // positive floats order like their bit patterns
                const int v = __float_as_int(__double2float_ru(hn));
                for (int nd = leaf_node[i]; nd >= 0; nd = parent[nd])
                    if (atomicMax(reinterpret_cast<int*>(node_hmax + nd), v) >= v) break;
            }
        }
    }
}

__global__ void k_flags(int n, const int* __restrict__ done, int* flags) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) flags[i] = done[i] ? 0 : 1;
}

__global__ void k_compact(int n, const int* __restrict__ flags, const int* __restrict__ off, int* list) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        if (flags[i]) list[off[i]] = i;
}

__global__ void k_record_unconverged(const int* __restrict__ list_count, DevStatus* st) {
    st->sml_unconverged = *list_count;
}

__global__ void k_copy(int n, const double* __restrict__ a, double* b) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) b[i] = a[i];
}

// Start of the iteration: every state array and counter, and the list of all
// particles.
__global__ void k_vh_init(int n, const double* __restrict__ h, double* hnew, int* done, int* nit, int* dirty, int* list,
                          int* list_count, int* ctr) {
    if (blockIdx.x == 0 && threadIdx.x < kBandCtr) ctr[threadIdx.x] = threadIdx.x == 3 ? 1 : 0;  // the first walk runs
    if (blockIdx.x == 0 && threadIdx.x == 0) *list_count = n;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        hnew[i] = h[i];
        done[i] = 0;
        nit[i] = -1;
        dirty[i] = 0;
        list[i] = i;
    }
}

// End of a sweep on lists: every iterating particle takes its new h, and the
// particles that have not stopped form the next list (in any order: every
// particle's update and pair edits depend on it alone, and the appended lists
// are sorted at the end); the lists are re-walked once a count was above maxnb
// (ctr[2] stays set: every sweep from then on) or when the sweep's pair changes
// overflowed the event buffer (nothing was edited).
__global__ void k_vh_commit(const int* __restrict__ list, const int* __restrict__ list_count,
                            const double* __restrict__ hnew, double* h, const int* __restrict__ done, int* next,
                            int* next_count, int* ctr) {
    const int m = *list_count;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        ctr[3] = (ctr[1] || ctr[2]) ? 1 : 0;
        ctr[0] = ctr[1] = 0;
    }
    const int step = gridDim.x * blockDim.x;
    for (int q0 = blockIdx.x * blockDim.x; q0 < m; q0 += step) {
        const int q = q0 + threadIdx.x;
        const int i = q < m ? list[q] : 0;
        if (q < m) h[i] = hnew[i];
        warp_append(q < m && !done[i], i, next, next_count);
    }
}

// Statistics and the capacity check of the list walk, for lists that the
// variable-h iteration kept current instead of a final walk.
__global__ void k_noi_stats(int n, int maxnb, const int* __restrict__ noi, const int* __restrict__ unconverged,
                            DevStatus* st) {
    if (blockIdx.x == 0 && threadIdx.x == 0) st->sml_unconverged = *unconverged;
    int mx = 0;
    unsigned long long tot = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int k = noi[i];
        if (k > maxnb) set_status(st, MHPC_ERR_NEIGHBOURS, i);
        mx = max(mx, k);
        tot += (unsigned long long)k;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mx = max(mx, __shfl_xor_sync(MHPC_FULL, mx, o));
        tot += __shfl_xor_sync(MHPC_FULL, tot, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&st->max_noi, mx);
        atomicAdd(&st->noi_sum, tot);
    }
}

__global__ void k_export_nnl(int n, int maxnb, const int* __restrict__ nbr, const int* __restrict__ noi,
                             const int* __restrict__ perm, int* nnl, int* noi_out) {
    for (long s = blockIdx.x * (long)blockDim.x + threadIdx.x; s < n; s += (long)gridDim.x * blockDim.x) {
        const int o = perm[s];
        const int k = noi[s];
        if (noi_out) noi_out[o] = k;
        if (nnl) {
            const int kk = min(k, maxnb);
            for (int q = 0; q < maxnb; ++q)
                nnl[(size_t)o * maxnb + q] = q < kk ? perm[nbr[nb_index(s, q, maxnb)]] : -1;
        }
    }
}

}  // namespace

namespace {
// Particles per warp of the neighbour walk.  With 32 a small n has one warp per
// scheduler or fewer, and a walk is a chain of round trips and list tests; with
// one sub-group of 8 there are four times the warps, with less to test each.
// List walk in us with 8 / 16 / 32: Sedov lattice of 8,000 particles 56 / 74 / 109,
// 35,937 127 / 115 / 156, 110,592 213 / 168 / 138; variable h of a cloud of 20,011
// 493 / 527 / 556, 50,000 628 / 626 / 695, 100,000 841 / 798 / 773.
int frnn_group(int n) { return n <= 25000 ? 8 : n <= 65000 ? 16 : 32; }
long frnn_blocks(int n, int ppw) { return (((long)n + ppw - 1) / ppw + kWarps - 1) / kWarps; }
}  // namespace

int sph_frnn(const TreeDev& T, const SphParams& P, const SphSorted& S, int* nbr, int* noi, DevStatus* st,
             cudaStream_t s) {
    if (P.n <= 0) return MHPC_OK;
    const int ppw = frnn_group(P.n);
    const long blocks = frnn_blocks(P.n, ppw);
    const float* hmax = nullptr;
    if (P.avg_h) {  // smoothing lengths differ: prune nodes by their largest h
        int rc = tree_node_hmax(T, S.h, st, s);
        if (rc) return rc;
        hmax = T.hmax;
    }
    k_frnn<0><<<(int)blocks, kBlock, 0, s>>>(T, P.n, ppw, P.maxnb, S.x, S.y, S.z, S.h, nullptr, nullptr, hmax, nbr, noi,
                                              st);
    CUDA_TRY(cudaGetLastError());
    return MHPC_OK;
}

int sph_variable_h(const TreeDev& T, const SphParams& P, const double* x, const double* y, const double* z,
                   double* h, const VhBuffers& B, int target, int tol, int max_iter, int sweeps, DevStatus* st,
                   cudaStream_t s) {
    if (P.n <= 0) return MHPC_OK;
    const int ppw = frnn_group(P.n);
    const long blocks = frnn_blocks(P.n, ppw);
    const int g = grid_for(P.n, 256, 148 * 16);
    const int* list_count = B.off + P.n;
    // Jacobi snapshot of h and the largest-h bounds; k_vh_update keeps both
    // current from then on
    CUDA_TRY(cudaMemsetAsync(B.done, 0, sizeof(int) * P.n, s));
    CUDA_TRY(cudaMemsetAsync(B.nit, 0xff, sizeof(int) * P.n, s));  // nit starts at -1
    k_copy<<<g, 256, 0, s>>>(P.n, h, B.hold);
    int rc0 = tree_node_hmax(T, B.hold, st, s);
    if (rc0) return rc0;
    for (int it = 0; it < sweeps; ++it) {
        // the list of particles still iterating
        k_flags<<<g, 256, 0, s>>>(P.n, B.done, B.flags);
        int rc = scan_exclusive_i32(B.flags, B.off, P.n, B.scan_scratch, s);
        if (rc) return rc;
        k_compact<<<g, 256, 0, s>>>(P.n, B.flags, B.off, B.list);
        if (it == 0) {
            // first sweep: (nearly) every particle, group walks
            k_frnn<1><<<(int)blocks, kBlock, 0, s>>>(T, P.n, ppw, P.maxnb, x, y, z, B.hold, B.list, list_count, T.hmax,
                                                      nullptr, B.count, st);
        } else {
            // later sweeps: the few particles still iterating, a warp each
            k_count_warp<<<148 * 8, kBlock, 0, s>>>(T, x, y, z, B.hold, B.list, list_count, T.hmax, B.count, st);
        }
        k_vh_update<<<g, 256, 0, s>>>(B.list, list_count, nullptr, it == 1 ? st : nullptr, P.n, B.count, h, B.hold, B.done, B.nit, target, tol, max_iter,
                                      P.maxnb, T.hmax, T.leaf_node, T.parent, P.ord);
    }
    k_flags<<<g, 256, 0, s>>>(P.n, B.done, B.flags);
    int rc = scan_exclusive_i32(B.flags, B.off, P.n, B.scan_scratch, s);
    if (rc) return rc;
    k_record_unconverged<<<1, 1, 0, s>>>(list_count, st);
    CUDA_TRY(cudaGetLastError());
    return MHPC_OK;
}

int sph_variable_h_lists(const TreeDev& T, const SphParams& P, const double* x, const double* y, const double* z,
                         double* h, int* nbr, int* noi, const VhBuffers& V, const BandBuffers& B, int target,
                         int tol, int max_iter, int sweeps, bool sort_lists, DevStatus* st, cudaStream_t s) {
    if (P.n <= 0) return MHPC_OK;
    const int ppw = frnn_group(P.n);
    const long blocks = frnn_blocks(P.n, ppw);
    const int g = grid_for(P.n, 256, 148 * 16);
    int* trunc = B.ctr + 2;   // some list holds fewer entries than its count
    int* rewalk = B.ctr + 3;  // the lists are re-walked after this sweep
    double* hnew = B.hnew;
    k_vh_init<<<g, 256, 0, s>>>(P.n, h, hnew, V.done, V.nit, B.dirty, V.list, V.cnt, B.ctr);
    int rc = tree_node_hmax(T, h, st, s);
    if (rc) return rc;
    // the lists and counts of the starting h: the counts of the first sweep
    k_frnn<2><<<(int)blocks, kBlock, 0, s>>>(T, P.n, ppw, P.maxnb, x, y, z, h, nullptr, nullptr, T.hmax, nbr, noi, st,
                                              rewalk, trunc);
    // gated re-walks: several groups per warp, so that the launch that finds
    // nothing to do has few blocks to retire
    const long gated = std::min(blocks, std::max(148L * MHPC_FRNN_MIN_BLOCKS, blocks / 8));
    for (int it = 0; it < sweeps; ++it) {
        // the first sweep lists every particle, a later one those that have not stopped
        const int* cur = (it & 1) ? V.list2 : V.list;
        int* next = (it & 1) ? V.list : V.list2;
        const int* cur_count = V.cnt + (it & 1);
        int* next_count = V.cnt + ((it + 1) & 1);
        // the reference's update from the exact counts of the current h (Jacobi:
        // every new h goes to hnew first)
        k_vh_update<<<g, 256, 0, s>>>(cur, cur_count, next_count, it == 1 ? st : nullptr, P.n, noi, hnew, hnew, V.done,
                                      V.nit, target, tol, max_iter, P.maxnb, T.hmax, T.leaf_node, T.parent, P.ord);
        rc = sph_apply_h_changes(T, P, x, y, z, h, hnew, nbr, noi, cur, cur_count, B, trunc, st, s);
        if (rc) return rc;
        k_vh_commit<<<g, 256, 0, s>>>(cur, cur_count, hnew, h, V.done, next, next_count, B.ctr);
        k_frnn<2><<<(int)gated, kBlock, 0, s>>>(T, P.n, ppw, P.maxnb, x, y, z, h, nullptr, nullptr, T.hmax, nbr, noi, st,
                                                 rewalk, trunc);
    }
    if (sort_lists) {
        rc = sph_sort_appended(P, nbr, noi, B.appended, s);
        if (rc) return rc;
    }
    k_noi_stats<<<grid_for(P.n, 256, 148 * 4), 256, 0, s>>>(P.n, P.maxnb, noi, V.cnt + (sweeps & 1), st);
    CUDA_TRY(cudaGetLastError());
    return MHPC_OK;
}

namespace {
__global__ void k_band(int n, const int* __restrict__ noi, int target, int tol, DevStatus* st) {
    int bad = 0;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        bad += abs(noi[i] - target) >= tol;
    for (int o = 16; o > 0; o >>= 1) bad += __shfl_xor_sync(MHPC_FULL, bad, o);
    if ((threadIdx.x & 31) == 0 && bad) atomicAdd(&st->sml_out_of_band, bad);
}
}  // namespace

int sph_band_stats(const SphParams& P, const int* noi, int target, int tol, DevStatus* st, cudaStream_t s) {
    if (P.n <= 0) return MHPC_OK;
    k_band<<<grid_for(P.n, 256, 148 * 4), 256, 0, s>>>(P.n, noi, target, tol, st);
    CUDA_TRY(cudaGetLastError());
    return MHPC_OK;
}

int sph_export_nnl(const SphParams& P, const int* nbr, const int* noi, const int* perm, int* nnl, int* noi_out,
                   cudaStream_t s) {
    if (P.n <= 0) return MHPC_OK;
    k_export_nnl<<<grid_for(P.n, 256, 148 * 16), 256, 0, s>>>(P.n, P.maxnb, nbr, noi, perm, nnl, noi_out);
    CUDA_TRY(cudaGetLastError());
    return MHPC_OK;
}
