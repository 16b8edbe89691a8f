// Stable LSD radix sort of (64-bit key, 32-bit value) pairs and a device-wide
// exclusive scan.
//
// The reference sorts with cub::DeviceRadixSort::SortPairs and a cudaMalloc /
// cudaFree of temporary storage on every call (src/helper.cu:150-166).  This
// sort is the library's own, eight passes of 8-bit digits in one of three
// forms by size:
//  - up to kBlockSortN keys: all passes in one block, in shared memory;
//  - up to kLookN: one read of the keys builds all eight digit histograms,
//    then each pass is a single "onesweep" kernel (tile ranking with warp
//    ballots, decoupled look-back across tiles, shared-memory staging so that
//    the scatter writes runs of equal digits contiguously);
//  - above: each pass counts its tiles' digits, scans the counts, and ranks
//    and scatters without any wait between tiles.
// Scratch is caller-provided; nothing is allocated per call.  Sorting is
// stable, so equal keys keep ascending input position, which is the contract
// of the CUB call it replaces.
#include <mutex>

#include "common.cuh"

namespace {

constexpr int kRadixBits = 8;
constexpr int kRadix = 256;
constexpr int kPasses = 8;
constexpr int kBlock = 256;
constexpr int kWarps = kBlock / 32;
// Where the lines lie, sort of n keys in us (before: look-back over single
// predecessors with tiles of 4096 for every n, and two more launches):
//   n              1,000  4,000  17,000  131,072  262,144  600,000  2^20  2^21  2^24
//   before            79     79      91      116      126             187   302  1559
//   one block         16     38     (8,000: 65, 16,000: 138)
//   look-back, 1024   42     58      64       83      112      175
//   look-back, 4096   75     75      91       95      114      116   179   300  1678
//   counted, 2048                                              150   167   233  1361
//   counted, 3072                                                    181   247  1301
// The look-back's cost grows with the number of tiles (50-80 ns each: the prefix
// travels from tile to tile), the counted form's with its 24 launches.
constexpr long kBlockSortN = 4096;
constexpr long kLookN = 600000;
// keys per thread of a pass
constexpr int pass_items(long n) { return n <= 200000 ? 4 : n <= kLookN ? 16 : n <= 6000000 ? 8 : 12; }
constexpr int kLook = 8;        // predecessors that the look-back reads at once
constexpr long tiles_of(long n, int items) { return (n + kBlock * items - 1) / (kBlock * items); }
constexpr unsigned long long kFlagAgg = 1ULL << 62;
constexpr unsigned long long kFlagInc = 2ULL << 62;
constexpr long kSpinLimit = 1L << 22;

__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

struct SortScratch {
    uint64_t* keys_tmp;
    int* vals_tmp;
    unsigned* hist;                 // [kPasses][kRadix] digit counts of the whole input
    unsigned* tile_counter;         // [kPasses]
    unsigned long long* look;       // look-back: [kPasses][ntiles][kRadix]; counts: unsigned [kRadix][ntiles]
};

static size_t align256(size_t b) { return (b + 255) & ~size_t(255); }

static SortScratch carve(void* base, int n) {
    char* p = (char*)base;
    SortScratch s;
    s.keys_tmp = (uint64_t*)p; p += align256(sizeof(uint64_t) * (size_t)n);
    s.vals_tmp = (int*)p; p += align256(sizeof(int) * (size_t)n);
    s.hist = (unsigned*)p; p += align256(sizeof(unsigned) * kPasses * kRadix);
    s.tile_counter = (unsigned*)p; p += align256(sizeof(unsigned) * kPasses);
    s.look = (unsigned long long*)p;
    return s;
}

// Lanes of the warp holding the same 8-bit digit d: eight ballots, one per
// digit bit (on B200 cheaper than a match instruction unless most lanes share
// the digit).  Every lane of the warp must call it.
__device__ __forceinline__ unsigned digit_peers(unsigned d) {
    unsigned peers = MHPC_FULL;
#pragma unroll
    for (int b = 0; b < kRadixBits; ++b) {
        const unsigned bb = __ballot_sync(MHPC_FULL, (d >> b) & 1u);
        peers &= ((d >> b) & 1u) ? bb : ~bb;
    }
    return peers;
}

// All eight digit histograms in one read of the keys: plain shared-memory
// atomics per key and digit (same-address conflicts within a warp are
// resolved by the hardware faster than aggregating them first), then one
// global atomic per bin per block.
__global__ void __launch_bounds__(kBlock) k_hist(const uint64_t* __restrict__ keys, int n, unsigned* hist) {
    __shared__ unsigned sh[kPasses * kRadix];
    for (int i = threadIdx.x; i < kPasses * kRadix; i += kBlock) sh[i] = 0;
    __syncthreads();
    long stride = (long)gridDim.x * kBlock;
    for (long i = (long)blockIdx.x * kBlock + threadIdx.x; i < n; i += stride) {
        const uint64_t k = __ldg(keys + i);
#pragma unroll
        for (int p = 0; p < kPasses; ++p)
            atomicAdd(&sh[p * kRadix + ((unsigned)(k >> (p * kRadixBits)) & (kRadix - 1))], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kPasses * kRadix; i += kBlock)
        if (sh[i]) atomicAdd(&hist[i], sh[i]);
}

// Digit counts of every tile of one pass (counts[digit][tile]).
template <int ITEMS>
__global__ void __launch_bounds__(kBlock) k_tile_count(const uint64_t* __restrict__ keys, int n, int pass,
                                                       long ntiles, unsigned* __restrict__ counts) {
    __shared__ unsigned sh[kRadix];
    sh[threadIdx.x] = 0;
    __syncthreads();
    const long base = (long)blockIdx.x * (kBlock * ITEMS) + threadIdx.x;
    uint64_t k[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) k[i] = base + i * kBlock < n ? __ldg(keys + base + i * kBlock) : 0;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
        if (base + i * kBlock < n) atomicAdd(&sh[(unsigned)(k[i] >> (pass * kRadixBits)) & (kRadix - 1)], 1u);
    __syncthreads();
    counts[threadIdx.x * ntiles + blockIdx.x] = sh[threadIdx.x];
}

__device__ __forceinline__ unsigned warp_incl(unsigned v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(MHPC_FULL, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Block d: exclusive scan of digit d's counts over the tiles, in place, and
// the digit's total.
__global__ void __launch_bounds__(kBlock) k_tile_scan(unsigned* counts, long ntiles, unsigned* totals) {
    __shared__ unsigned ws[kWarps];
    unsigned* c = counts + blockIdx.x * ntiles;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int kPer = 8;
    unsigned carry = 0;
    for (long b = 0; b < ntiles; b += kBlock * kPer) {
        const long i0 = b + (long)threadIdx.x * kPer;
        unsigned v[kPer], sum = 0;
#pragma unroll
        for (int q = 0; q < kPer; ++q) { v[q] = i0 + q < ntiles ? c[i0 + q] : 0; sum += v[q]; }
        const unsigned incl = warp_incl(sum);
        if (lane == 31) ws[warp] = incl;
        __syncthreads();
        unsigned before = carry + incl - sum, all = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            if (w < warp) before += ws[w];
            all += ws[w];
        }
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            if (i0 + q < ntiles) c[i0 + q] = before;
            before += v[q];
        }
        carry += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

template <int ITEMS>
struct PassSmem {
    unsigned whist[kWarps][kRadix];
    unsigned tile_off[kRadix];
    unsigned gbase[kRadix];
    unsigned wsum[2][kWarps];
    unsigned tile_id;
    uint64_t keys[kBlock * ITEMS];
    int vals[kBlock * ITEMS];
};

// One pass: rank the tile's keys by digit, and scatter.  `hist` holds the digit
// counts of the whole input.  LOOK: the tile's place among the keys of each
// digit by look-back over `look`, kLook predecessors at once; otherwise from
// the scanned counts (`counts`).
template <int ITEMS, bool LOOK>
__global__ void __launch_bounds__(kBlock, ITEMS > 12 ? 2 : ITEMS > 8 ? 3 : 4)
k_pass(const uint64_t* __restrict__ kin, const int* __restrict__ vin, uint64_t* __restrict__ kout,
       int* __restrict__ vout, int n, int pass, long ntiles, const unsigned* __restrict__ hist,
       const unsigned* __restrict__ counts, unsigned* tile_counter, unsigned long long* look, DevStatus* st) {
    constexpr int kTile = kBlock * ITEMS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    PassSmem<ITEMS>& S = *reinterpret_cast<PassSmem<ITEMS>*>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int shift = pass * kRadixBits;
    if (LOOK && tid == 0) S.tile_id = atomicAdd(tile_counter, 1u);
    const unsigned total = __ldg(hist + tid);
    for (int i = tid; i < kWarps * kRadix; i += kBlock) (&S.whist[0][0])[i] = 0;
    __syncthreads();
    const long tile = LOOK ? S.tile_id : blockIdx.x;
    const long base = tile * kTile + (long)warp * (32 * ITEMS);

    uint64_t key[ITEMS];
    int val[ITEMS];
    unsigned rank[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        long idx = base + i * 32 + lane;
        if (idx < n) {
            key[i] = __ldg(kin + idx);
            val[i] = vin ? __ldg(vin + idx) : (int)idx;
        } else {
            key[i] = 0;
            val[i] = 0;
        }
    }
    const unsigned before = LOOK ? 0 : __ldg(counts + tid * ntiles + tile);
    const unsigned lt = lanemask_lt();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        long idx = base + i * 32 + lane;
        bool valid = idx < n;
        unsigned vm = __ballot_sync(MHPC_FULL, valid);
        unsigned d = (unsigned)(key[i] >> shift) & (kRadix - 1);
        unsigned peers = digit_peers(d) & vm;
        if (!valid) peers = 1u << lane;
        int leader = __ffs(peers) - 1;
        unsigned b = 0;
        if (valid && lane == leader) b = S.whist[warp][d];
        b = __shfl_sync(MHPC_FULL, b, leader);
        rank[i] = b + __popc(peers & lt);
        __syncwarp();
        if (valid && lane == leader) S.whist[warp][d] = b + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    // per digit (one per thread): prefix over the warps, and the tile's total
    unsigned run = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
        unsigned c = S.whist[w][tid];
        S.whist[w][tid] = run;
        run += c;
    }
    unsigned long long* mine = look + ((long)pass * ntiles + tile) * kRadix + tid;
    if (LOOK) st_relaxed(mine, (tile == 0 ? kFlagInc : kFlagAgg) | (unsigned long long)run);
    // smaller digits, in the whole input and in the tile
    const unsigned gi = warp_incl(total), ti = warp_incl(run);
    if (lane == 31) { S.wsum[0][warp] = gi; S.wsum[1][warp] = ti; }
    unsigned long long excl = before;
    if (LOOK && tile > 0) {
        long j = tile - 1, spins = 0;
        bool done = false;
        while (!done) {
            unsigned long long v[kLook];
#pragma unroll
            for (int q = 0; q < kLook; ++q)
                v[q] = j - q >= 0 ? ld_relaxed(look + ((long)pass * ntiles + j - q) * kRadix + tid) : kFlagInc;
            bool wait = false;
#pragma unroll
            for (int q = 0; q < kLook; ++q) {
                const unsigned long long f = v[q] & (3ULL << 62);
                wait = wait || f == 0;  // not there yet: read again from here
                if (!done && !wait) {
                    excl += v[q] & 0xffffffffULL;
                    done = f == kFlagInc;
                    --j;
                }
            }
            if (wait && !done && ++spins > kSpinLimit) {
                set_status(st, MHPC_ERR_TIMEOUT, 100 + pass);
                done = true;
            }
        }
        st_relaxed(mine, kFlagInc | (excl + run));
    }
    __syncthreads();
    {
        unsigned g = gi - total, t = ti - run;
#pragma unroll
        for (int w = 0; w < kWarps; ++w)
            if (w < warp) { g += S.wsum[0][w]; t += S.wsum[1][w]; }
        S.gbase[tid] = g + (unsigned)excl;
        S.tile_off[tid] = t;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        long idx = base + i * 32 + lane;
        if (idx < n) {
            unsigned d = (unsigned)(key[i] >> shift) & (kRadix - 1);
            unsigned pos = S.tile_off[d] + S.whist[warp][d] + rank[i];
            S.keys[pos] = key[i];
            S.vals[pos] = val[i];
        }
    }
    __syncthreads();
    long tile_count = (long)n - tile * kTile;
    if (tile_count > kTile) tile_count = kTile;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const int q = i * kBlock + tid;
        if (q < tile_count) {
            uint64_t k = S.keys[q];
            unsigned d = (unsigned)(k >> shift) & (kRadix - 1);
            unsigned dest = S.gbase[d] + (q - S.tile_off[d]);
            kout[dest] = k;
            vout[dest] = S.vals[q];
        }
    }
}

// All passes in one block, for at most THREADS x ITEMS keys.  Keys
// and their input positions stay in shared memory; a pass ranks like k_pass.
// Slots from n on hold the largest key and come last: they follow every input
// position, and the sort is stable.  The outputs may be the inputs' arrays (the
// other forms go through scratch), so none of the four is __restrict__.
template <int THREADS, int ITEMS>
struct BlockSortSmem {
    uint64_t key[THREADS * ITEMS];
    unsigned short pos[THREADS * ITEMS];
    unsigned short whist[(THREADS / 32)][kRadix];
    unsigned off[kRadix];
    unsigned wsum[kRadix / 32];
};

template <int THREADS, int ITEMS>
__global__ void __launch_bounds__(THREADS) k_block_sort(const uint64_t* kin, const int* vin, uint64_t* kout,
                                                        int* vout, int n) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    BlockSortSmem<THREADS, ITEMS>& S = *reinterpret_cast<BlockSortSmem<THREADS, ITEMS>*>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int base = warp * (32 * ITEMS) + lane;
    uint64_t key[ITEMS];
    unsigned short pos[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const int idx = base + i * 32;
        key[i] = idx < n ? kin[idx] : ~0ULL;
        pos[i] = (unsigned short)idx;
    }
    const unsigned lt = lanemask_lt();
    for (int shift = 0; shift < 64; shift += kRadixBits) {
        for (int i = tid; i < (THREADS / 32) * kRadix / 2; i += THREADS)
            reinterpret_cast<unsigned*>(&S.whist[0][0])[i] = 0;
        __syncthreads();
        unsigned short rank[ITEMS];
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const unsigned d = (unsigned)(key[i] >> shift) & (kRadix - 1);
            const unsigned peers = digit_peers(d);
            const int leader = __ffs(peers) - 1;
            unsigned b = S.whist[warp][d];  // (every peer reads the same count)
            rank[i] = (unsigned short)(b + __popc(peers & lt));
            __syncwarp();
            if (lane == leader) S.whist[warp][d] = (unsigned short)(b + __popc(peers));
            __syncwarp();
        }
        __syncthreads();
        unsigned run = 0, incl = 0;
        if (tid < kRadix) {
#pragma unroll
            for (int w = 0; w < (THREADS / 32); ++w) {
                const unsigned c = S.whist[w][tid];
                S.whist[w][tid] = (unsigned short)run;
                run += c;
            }
            incl = warp_incl(run);
            if (lane == 31) S.wsum[warp] = incl;
        }
        __syncthreads();
        if (tid < kRadix) {
            unsigned b = incl - run;
#pragma unroll
            for (int w = 0; w < kRadix / 32; ++w)
                if (w < warp) b += S.wsum[w];
            S.off[tid] = b;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const unsigned d = (unsigned)(key[i] >> shift) & (kRadix - 1);
            const unsigned to = S.off[d] + S.whist[warp][d] + rank[i];
            S.key[to] = key[i];
            S.pos[to] = pos[i];
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            key[i] = S.key[base + i * 32];
            pos[i] = S.pos[base + i * 32];
        }
    }
    // every value is read before the first is written
    int val[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        val[i] = pos[i];
        if (vin && base + i * 32 < n) val[i] = vin[pos[i]];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const int idx = base + i * 32;
        if (idx < n) {
            kout[idx] = key[i];
            vout[idx] = val[i];
        }
    }
}

// a pass without look-back
template <int ITEMS>
void count_pass(const uint64_t* kin, const int* vin, uint64_t* kout, int* vout, int n, int pass, long ntiles,
                unsigned* hist, unsigned* counts, DevStatus* st, cudaStream_t s) {
    k_tile_count<ITEMS><<<(int)ntiles, kBlock, 0, s>>>(kin, n, pass, ntiles, counts);
    k_tile_scan<<<kRadix, kBlock, 0, s>>>(counts, ntiles, hist);
    k_pass<ITEMS, false><<<(int)ntiles, kBlock, sizeof(PassSmem<ITEMS>), s>>>(kin, vin, kout, vout, n, pass, ntiles, hist,
                                                                            counts, nullptr, nullptr, st);
}

template <int THREADS, int ITEMS>
int block_sort(const uint64_t* keys_in, const int* vals_in, uint64_t* keys_out, int* vals_out, int n,
               cudaStream_t s) {
    // per device (a process may drive several GPUs); a cheap host call
    CUDA_TRY(cudaFuncSetAttribute(k_block_sort<THREADS, ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sizeof(BlockSortSmem<THREADS, ITEMS>)));
    k_block_sort<THREADS, ITEMS><<<1, THREADS, sizeof(BlockSortSmem<THREADS, ITEMS>), s>>>(keys_in, vals_in, keys_out,
                                                                                  vals_out, n);
    CUDA_TRY(cudaGetLastError());
    return MHPC_OK;
}

// ------------------------------------------------------------------ scan
constexpr int kScanBlock = 256;
constexpr int kScanItems = 16;
constexpr int kScanChunk = kScanBlock * kScanItems;

__device__ __forceinline__ int block_excl_scan(int v, int* sw, int* total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(MHPC_FULL, x, o);
        if (lane >= o) x += t;
    }
    if (lane == 31) sw[w] = x;
    __syncthreads();
    if (w == 0) {
        int y = lane < (int)(blockDim.x >> 5) ? sw[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int t = __shfl_up_sync(MHPC_FULL, y, o);
            if (lane >= o) y += t;
        }
        sw[lane] = y;
    }
    __syncthreads();
    int before = w > 0 ? sw[w - 1] : 0;
    *total = sw[(blockDim.x >> 5) - 1];
    __syncthreads();
    return before + x - v;
}

__global__ void __launch_bounds__(kScanBlock) k_scan_reduce(const int* __restrict__ in, int n, int* bsum) {
    __shared__ int sw[32];
    long base = (long)blockIdx.x * kScanChunk;
    int s = 0;
    for (int i = 0; i < kScanItems; ++i) {
        long idx = base + i * kScanBlock + threadIdx.x;
        if (idx < n) s += in[idx];
    }
    int tot;
    block_excl_scan(s, sw, &tot);
    if (threadIdx.x == 0) bsum[blockIdx.x] = tot;
}

// (also the scan's total)
__global__ void __launch_bounds__(1024) k_scan_bsum(int* bsum, int nb, int* total) {
    __shared__ int sw[32];
    int carry = 0;
    for (int b0 = 0; b0 < nb; b0 += 1024) {
        int i = b0 + threadIdx.x;
        int v = i < nb ? bsum[i] : 0;
        int tot;
        int e = block_excl_scan(v, sw, &tot);
        if (i < nb) bsum[i] = carry + e;
        carry += tot;
    }
    if (threadIdx.x == 0) *total = carry;
}

__global__ void __launch_bounds__(kScanBlock) k_scan_down(const int* __restrict__ in, int* out, int n,
                                                          const int* __restrict__ bsum) {
    __shared__ int sw[32];
    __shared__ int tile[kScanChunk];
    long base = (long)blockIdx.x * kScanChunk;
    for (int i = 0; i < kScanItems; ++i) {
        long idx = base + i * kScanBlock + threadIdx.x;
        tile[i * kScanBlock + threadIdx.x] = idx < n ? in[idx] : 0;
    }
    __syncthreads();
    int loc[kScanItems];
    int s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        loc[i] = s;
        s += tile[threadIdx.x * kScanItems + i];
    }
    int tot;
    int e = block_excl_scan(s, sw, &tot);
    int carry = bsum[blockIdx.x] + e;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) tile[threadIdx.x * kScanItems + i] = carry + loc[i];
    __syncthreads();
    for (int i = 0; i < kScanItems; ++i) {
        long idx = base + i * kScanBlock + threadIdx.x;
        if (idx < n) out[idx] = tile[i * kScanBlock + threadIdx.x];
    }
}

constexpr size_t align256c(size_t b) { return (b + 255) & ~size_t(255); }

// look-back words or digit counts, whichever of the sizes up to n needs more
// (scratch made for n keys serves every smaller number too)
constexpr size_t look_bytes(long n) {
    const size_t a = sizeof(unsigned long long) * kPasses * kRadix * (size_t)tiles_of(n < 200000 ? n : 200000, 4);
    const size_t b = n <= kLookN ? 0 : sizeof(unsigned) * kRadix * (size_t)tiles_of(n, 8);
    return align256c(a > b ? a : b);
}

constexpr size_t scratch_formula(long n) {
    return align256c(sizeof(uint64_t) * (size_t)n) + align256c(sizeof(int) * (size_t)n) +
           align256c(sizeof(unsigned) * kPasses * kRadix) + align256c(sizeof(unsigned) * kPasses) +
           look_bytes(n);
}

}  // namespace

size_t sort_scratch_bytes(int n) { return scratch_formula(n); }

int sort_pairs_u64(const uint64_t* keys_in, const int* vals_in, uint64_t* keys_out, int* vals_out, int n,
                   void* scratch, size_t scratch_bytes, DevStatus* st, cudaStream_t s) {
    if (n < 0) return MHPC_ERR_ARG;
    if (n == 0) return MHPC_OK;
    if (!keys_in || !keys_out || !vals_out) return MHPC_ERR_ARG;
    if (!scratch || scratch_bytes < sort_scratch_bytes(n)) return MHPC_ERR_ARG;
    if (n <= 1024) return block_sort<256, 4>(keys_in, vals_in, keys_out, vals_out, n, s);
    if (n <= kBlockSortN) return block_sort<512, 8>(keys_in, vals_in, keys_out, vals_out, n, s);
    SortScratch S = carve(scratch, n);
    const bool lookback = n <= kLookN;
    const int items = pass_items(n);
    const long ntiles = tiles_of(n, items);
    unsigned* counts = reinterpret_cast<unsigned*>(S.look);
    if (lookback) {
        // zero histograms, tile counters and look-back words in one memset
        const size_t zero_bytes = (size_t)((char*)S.look - (char*)S.hist) +
                                  sizeof(unsigned long long) * kPasses * kRadix * (size_t)ntiles;
        CUDA_TRY(cudaMemsetAsync(S.hist, 0, zero_bytes, s));
        // (1024 keys a block or more: a block ends with up to 2048 global atomics)
        k_hist<<<grid_for(n, 4 * kBlock, 148 * 4), kBlock, 0, s>>>(keys_in, n, S.hist);
    }
    // per device (a process may drive several GPUs); cheap host calls
    CUDA_TRY(cudaFuncSetAttribute(k_pass<16, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sizeof(PassSmem<16>)));
    CUDA_TRY(cudaFuncSetAttribute(k_pass<12, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sizeof(PassSmem<12>)));
    const uint64_t* kin = keys_in;
    const int* vin = vals_in;
    for (int p = 0; p < kPasses; ++p) {
        uint64_t* kout = (p & 1) ? keys_out : S.keys_tmp;
        int* vout = (p & 1) ? vals_out : S.vals_tmp;
        unsigned* hist = S.hist + p * kRadix;
        if (lookback && items == 4) {
            k_pass<4, true><<<(int)ntiles, kBlock, sizeof(PassSmem<4>), s>>>(
                kin, vin, kout, vout, n, p, ntiles, hist, nullptr, S.tile_counter + p, S.look, st);
        } else if (lookback) {
            k_pass<16, true><<<(int)ntiles, kBlock, sizeof(PassSmem<16>), s>>>(
                kin, vin, kout, vout, n, p, ntiles, hist, nullptr, S.tile_counter + p, S.look, st);
        } else if (items == 8) {
            count_pass<8>(kin, vin, kout, vout, n, p, ntiles, hist, counts, st, s);
        } else {
            count_pass<12>(kin, vin, kout, vout, n, p, ntiles, hist, counts, st, s);
        }
        CUDA_TRY(cudaGetLastError());
        kin = kout;
        vin = vout;
    }
    return MHPC_OK;
}

// ------------------------------------------------- sort without allocation
// Some callers cannot allocate device memory: applications whose own pool
// reserves the device's memory at start-up (a cudaMalloc would fail or
// fragment it) and services that forbid allocation after initialisation.
// For them mhpc_sort_pairs_noalloc keeps its scratch in this file-scope
// device array, sized for kNoAllocMaxN keys.  Every GPU that loads the
// library holds the array until the process exits.
constexpr long kNoAllocMaxN = 1L << 20;
constexpr size_t kNoAllocStatusBytes = 256;
constexpr size_t kNoAllocBytes = scratch_formula(kNoAllocMaxN) + kNoAllocStatusBytes;
static __device__ __align__(256) unsigned char g_noalloc_sort_scratch[kNoAllocBytes];

namespace {

__global__ void k_copy_status(const DevStatus* st, int* out) { *out = st->code; }

// Device address of g_noalloc_sort_scratch on the current device.  The host
// symbol is only a stand-in for the device array, so the address is looked up
// once per device with that device current and cached.
std::mutex g_noalloc_mutex;
void* g_noalloc_ptr[256];

int noalloc_scratch(void** out) {
    int dev = 0;
    CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 256) return MHPC_ERR_ARG;
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_noalloc_sort_scratch) != cudaSuccess || !p) return MHPC_ERR_CUDA;
        g_noalloc_ptr[dev] = p;
    }
    *out = g_noalloc_ptr[dev];
    return MHPC_OK;
}

}  // namespace

extern "C" int mhpc_sort_noalloc_max_n(void) { return (int)kNoAllocMaxN; }

extern "C" int mhpc_sort_pairs_noalloc(const uint64_t* keys_in, const int* vals_in, uint64_t* keys_out,
                                       int* vals_out, int n, int* status_dev, void* stream) {
    if (n < 0) return MHPC_ERR_ARG;
    if (n > kNoAllocMaxN) return MHPC_ERR_CAPACITY;
    cudaStream_t s = (cudaStream_t)stream;
    void* base = nullptr;
    int rc = noalloc_scratch(&base);
    if (rc) return rc;
    DevStatus* st = reinterpret_cast<DevStatus*>((char*)base + kNoAllocBytes - kNoAllocStatusBytes);
    CUDA_TRY(cudaMemsetAsync(st, 0, sizeof(DevStatus), s));
    if (n > 0) {
        // sort_pairs_u64 clears the histograms, tile counters and look-back
        // words it needs before its first kernel
        rc = sort_pairs_u64(keys_in, vals_in, keys_out, vals_out, n, base, kNoAllocBytes - kNoAllocStatusBytes,
                            st, s);
        if (rc) return rc;
    }
    if (status_dev) {
        k_copy_status<<<1, 1, 0, s>>>(st, status_dev);
        CUDA_TRY(cudaGetLastError());
    }
    return MHPC_OK;
}

size_t scan_scratch_bytes(int n) {
    long nb = ((long)n + kScanChunk - 1) / kScanChunk;
    if (nb < 1) nb = 1;
    return align256(sizeof(int) * (size_t)nb);
}

int scan_exclusive_i32(const int* in, int* out, int n, void* scratch, cudaStream_t s) {
    if (n <= 0) {
        CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(int), s));
        return MHPC_OK;
    }
    int nb = (int)(((long)n + kScanChunk - 1) / kScanChunk);
    int* bsum = (int*)scratch;
    k_scan_reduce<<<nb, kScanBlock, 0, s>>>(in, n, bsum);
    k_scan_bsum<<<1, 1024, 0, s>>>(bsum, nb, out + n);
    k_scan_down<<<nb, kScanBlock, 0, s>>>(in, out, n, bsum);
    CUDA_TRY(cudaGetLastError());
    return MHPC_OK;
}
