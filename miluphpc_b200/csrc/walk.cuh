// One-particle-per-warp neighbour walk shared by the sparse neighbour counts
// of the variable-h iteration and the neighbour-band repair.
#pragma once
#include "sph.cuh"

// Lower bound (every step rounded down) of the squared distance between the
// boxes [al, ah] and [bl, bh].
__device__ __forceinline__ float box_gap2(const float3& al, const float3& ah, const float4& bl, const float4& bh) {
    const float gx = fmaxf(fmaxf(__fsub_rd(bl.x, ah.x), __fsub_rd(al.x, bh.x)), 0.f);
    const float gy = fmaxf(fmaxf(__fsub_rd(bl.y, ah.y), __fsub_rd(al.y, bh.y)), 0.f);
    const float gz = fmaxf(fmaxf(__fsub_rd(bl.z, ah.z), __fsub_rd(al.z, bh.z)), 0.f);
    return __fmaf_rd(gx, gx, __fmaf_rd(gy, gy, __fmul_rd(gz, gz)));
}

// v appended to list by the lanes that want it, one atomic per warp.  All
// lanes of the warp call it.
__device__ __forceinline__ void warp_append(bool want, int v, int* list, int* count) {
    const unsigned b = __ballot_sync(MHPC_FULL, want);
    if (b == 0) return;
    const int lane = threadIdx.x & 31, leader = __ffs(b) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(count, __popc(b));
    base = __shfl_sync(MHPC_FULL, base, leader);
    if (want) list[base + __popc(b & ((1u << lane) - 1u))] = v;
}

// inclusive sum over the lanes
__device__ __forceinline__ int warp_scan(int v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(MHPC_FULL, v, o);
        if (lane >= o) v += u;
    }
    return v;
}

constexpr int kWalkStack = 512;
constexpr int kWalkReserve = 7 * 22 + 8;
constexpr int kWalkSmall = 16;   // cells with at most this many particles are tested whole

// One particle per warp (all 32 lanes call this; a lane that is not `valid`
// walks nothing but takes part in the warp's votes).  Visits every particle
// j of the leaves, small cells and shared-key buckets whose box comes within
// `rad` of the particle and whose largest h below the node reaches it:
// visit(j) is called on one lane per candidate (j may be the particle itself).
// Pruning is conservative (FP32 boxes rounded outward), so every j with
// d < rad and d < h_j is visited.  The walks here serve few, often far-reaching
// particles, so a whole warp pops up to 32 nodes per step; stack bound as in
// the other walks: a pop of k nodes pushes at most 8k, and k is limited so
// that a depth-first descent (7 per level, 22 levels) always fits on top.
template <class Visit>
__device__ __forceinline__ void warp_walk(const TreeDev& T, int M, bool valid, double px, double py, double pz,
                                          double rad, const float* __restrict__ node_hmax, int* S, int* RF,
                                          DevStatus* st, Visit& visit) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    if (!__any_sync(MHPC_FULL, valid)) return;
    const float3 p0 = make_float3(__double2float_rd(px), __double2float_rd(py), __double2float_rd(pz));
    const float3 p1 = make_float3(__double2float_ru(px), __double2float_ru(py), __double2float_ru(pz));
    const float fr = __double2float_ru(rad);
    int top = 0;
    if (lane == 0) {
        int c = 0;
        while (c < M && top < 8) { S[top++] = c; c = __ldg(&T.link[c].x); }
        if (c < M) set_status(st, MHPC_ERR_DEPTH, 7);
    }
    top = __shfl_sync(MHPC_FULL, top, 0);
    __syncwarp();
    while (top > 0) {
        const int room = (kWalkStack - kWalkReserve - top) / 7;
        int kk = top < 32 ? top : 32;
        if (kk > room) kk = room > 1 ? room : 1;
        const bool act = lane < kk;
        const int nd = act ? S[top - 1 - lane] : 0;
        __syncwarp();
        top -= kk;
        int rf = 0, rlen = 0, kmask = 0;
        int4 k0 = make_int4(0, 0, 0, 0), k1 = k0;
        if (act) {
            // the child slots come with the box: a walk of one particle waits for
            // each round trip
            k0 = __ldg(reinterpret_cast<const int4*>(T.kids + 8 * (size_t)nd));
            k1 = __ldg(reinterpret_cast<const int4*>(T.kids + 8 * (size_t)nd) + 1);
            const int2 lk = __ldg(T.link + nd);
            const float4 bl = __ldg(T.bmin + nd), bh = __ldg(T.bmax + nd);
            const float hn = __ldg(node_hmax + nd);
            const int fs = __ldg(T.first + nd), l = __ldg(T.last + nd), km = __ldg(T.kmask + nd);
            // a pair needs d < rad and d < h_j: the box must come within both
            const float lim = fminf(fr, hn);
            if (box_gap2(p0, p1, bl, bh) <= __fmul_ru(lim, lim)) {
                rf = fs;
                if (lk.y & ND_LEAF) {
                    rlen = 1;
                } else {
                    if (l - rf + 1 <= kWalkSmall || (km & 0x100)) rlen = l - rf + 1;
                    else kmask = km & 0xff;
                }
            }
        }
        // (one scan for the children, at most 256, and for the candidate ranges;
        // ranges above 65,536 particles, a shared-key bucket's, by a second one)
        const int nkid = __popc(kmask);
        const bool wide = __any_sync(MHPC_FULL, rlen > 65536);
        const int both = warp_scan(nkid | (wide ? 0 : rlen << 9), lane);
        const int incl = both & 511;
        const int rincl = wide ? warp_scan(rlen, lane) : both >> 9;
        const int total = __shfl_sync(MHPC_FULL, incl, 31);
        if (top + total > kWalkStack) {  // unreachable by the bound on kk
            if (lane == 0) set_status(st, MHPC_ERR_DEPTH, 8);
            return;
        }
        if (nkid) {
            const int all[8] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w};
            int wpos = top + incl - nkid;
#pragma unroll
            for (int d = 0; d < 8; ++d)
                if ((kmask >> d) & 1) S[wpos++] = all[d];
        }
        top += total;
        // candidate ranges of this step: compact, each with its first particle less
        // its begin; a lane's range is the last that begins at or before it
        const int begin = rincl - rlen;
        const int ncand = __shfl_sync(MHPC_FULL, rincl, 31);
        const unsigned br = __ballot_sync(MHPC_FULL, rlen > 0);
        if (rlen > 0) RF[__popc(br & lt)] = rf - begin;
        __syncwarp();
        int begun = 0;  // ranges that begin before this batch
        for (int c0 = 0; c0 < ncand; c0 += 32) {
            const unsigned at = (unsigned)(begin - c0);
            const unsigned bits = __reduce_or_sync(MHPC_FULL, rlen > 0 && at < 32u ? 1u << at : 0u);
            if (c0 + lane < ncand) visit(RF[begun + __popc(bits & (2u * lt + 1u)) - 1] + c0 + lane);
            begun += __popc(bits);
        }
        __syncwarp();
    }
}

