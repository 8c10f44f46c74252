// Tile binning of visibility samples: a counting sort of samples by (w-slab, grid tile).
//
// The reference grids every sample straight into global memory with float atomics
// (SVDIntegratedImager.cu:1218-1293, 64 * K * 2 atomics per sample). Here samples are first
// binned by the tile that holds the origin of their ES footprint, so that each tile is gridded in
// shared memory by one CTA. The binning contract is bit-exact and shared with the CPU oracle:
//
//   p      = r * (cell_size * G)                FP64 (or the reference's FP32 rounding)
//   Q      = floor(p * 2^24)                    position quantised to 2^-24 cells
//   cell   = Q >> 24, frac = Q & (2^24 - 1)
//   lo     = frac ? cell - (W/2 - 1) : cell - W/2   (= ceil(p - W/2)),  hi = cell + W/2
//   clip   lo, hi to [-G/2, (G-1)/2] (SVDIntegratedImager.cu:1261-1267); drop if lo > hi
//          (strict mode: drop if the footprint leaves the grid)
//   tile1  = (lo1 + G/2) / T1, tile2 = (lo2 + G/2) / T2 (tiles may be rectangular)
//   slab   = clamp(floor((r3 - r3_min) / width), 0, nslab - 1)
//   key    = (slab * ntile1 + tile1) * ntile2 + tile2
#include "binning_rules.cuh"
#include "svdi_internal.cuh"

namespace svdi {

namespace {

using namespace binrules;

constexpr int kThreads = 256;
constexpr int kPerThread = 8;                       // samples per thread per scatter chunk
constexpr int kChunk = kThreads * kPerThread;       // samples per scatter block
constexpr int kSmemKeyLimit = 24576;                // keys aggregated in shared memory

// Per-block shared-memory histogram (warp-aggregated), flushed once per block.
__global__ void __launch_bounds__(kThreads) k_histogram(SampleSource src, GridGeom g, SlabParams sp,
                                                       unsigned int* __restrict__ counts, int n_keys,
                                                       unsigned long long* __restrict__ dropped,
                                                       const DevPlan* __restrict__ plan) {
    if (plan && first_thread()) {
        unsigned long long* const stamps = plan_stamps(plan);
        stamps[STAMP_BIN] = stamp_now();
        stamps[STAMP_FFT] = stamps[STAMP_END] = 0;  // maxima over the blocks of later kernels
    }
    if (plan) sp = plan->sp;
    extern __shared__ unsigned int sh[];
    const bool use_smem = n_keys <= kSmemKeyLimit;
    if (use_smem) {
        for (int k = threadIdx.x; k < n_keys; k += kThreads) sh[k] = 0;
        __syncthreads();
    }
    unsigned int ndrop = 0;
    const int lane = threadIdx.x & 31;
    const long long n = src.n;
    const long long stride = (long long)gridDim.x * kThreads;
    const long long n_round = ((n + stride - 1) / stride) * stride;
    for (long long idx = blockIdx.x * (long long)kThreads + threadIdx.x; idx < n_round; idx += stride) {
        int key = -2;
        if (idx < n) {
            key = sample_key(src, idx, g, sp).key;
            if (key < 0) ++ndrop;
        }
        const unsigned int peers = __match_any_sync(0xffffffffu, key);
        const int leader = __ffs(peers) - 1;
        if (key >= 0 && lane == leader) {
            const unsigned int c = __popc(peers);
            if (use_smem) atomicAdd(&sh[key], c);
            else atomicAdd(&counts[key], c);
        }
    }
    for (int o = 16; o > 0; o >>= 1) ndrop += __shfl_xor_sync(0xffffffffu, ndrop, o);
    if (lane == 0 && ndrop) atomicAdd(dropped, (unsigned long long)ndrop);
    if (use_smem) {
        __syncthreads();
        for (int k = threadIdx.x; k < n_keys; k += kThreads)
            if (sh[k]) atomicAdd(&counts[k], sh[k]);
    }
}

// Exclusive scan of the key counts (one block): offsets[0..n_keys], cursor = offsets. With
// kb_offsets, also the exclusive scan of ceil(count / kb_size): the K-blocks of kb_size records of
// one key each that the tensor-core gridder splits evenly over its CTAs. With chunk_key, for every
// chunk of chunk_size records the key its first record belongs to.
// The keys go through shared memory in tiles of kScanTile (coalesced loads and stores), each thread
// scanning kScanPer consecutive keys of a tile and the block combining the 1024 thread sums with warp
// shuffles; a running carry links the tiles.
constexpr int kScanPer = 4;               // keys per thread and tile
constexpr int kScanTile = kScanPer * 1024;

// Inclusive block-wide sum scan of one value per thread of a 1024-thread block; `tmp` holds 32 words
// of shared memory. Returns this thread's inclusive result and the block total.
__device__ __forceinline__ unsigned int block_scan(unsigned int v, unsigned int* tmp, unsigned int& total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    if (lane == 31) tmp[w] = v;
    __syncthreads();
    if (w == 0) {
        unsigned int x = tmp[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int u = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += u;
        }
        tmp[lane] = x;
    }
    __syncthreads();
    if (w > 0) v += tmp[w - 1];
    total = tmp[31];
    __syncthreads();
    return v;
}

// The key whose records hold the start of each chunk (chunk_size: a power of two): a key writes the chunks that
// start inside its records [run, run + c), and leaves them to its warp where they are many (mark_dense).
constexpr unsigned int kDenseChunks = 32;
__device__ __forceinline__ unsigned int first_chunk(unsigned int record, unsigned int chunk_size) {
    return (record >> (31 - __clz(chunk_size))) + ((record & (chunk_size - 1)) ? 1u : 0u);
}
__device__ __forceinline__ void mark_chunks(unsigned int* chunk_key, unsigned int chunk_size, unsigned int run,
                                            unsigned int c, unsigned int key) {
    if (c == 0 || c >= kDenseChunks * chunk_size) return;
    for (unsigned int ch = first_chunk(run, chunk_size), end = first_chunk(run + c, chunk_size); ch < end; ++ch)
        chunk_key[ch] = key;
}
// The chunks of the warp's dense keys, all lanes on one key at a time (one thread wrote the 32,700 chunks of a tile
// of 8.4 M samples in 1 ms). run, c, key: of this lane's first key; its kScanPer keys follow one another.
__device__ __forceinline__ void mark_dense(unsigned int* chunk_key, unsigned int chunk_size, unsigned int run,
                                           const unsigned int (&c)[kScanPer], unsigned int key) {
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
        const bool dense = c[k] >= kDenseChunks * chunk_size;
        for (unsigned int m = __ballot_sync(0xffffffffu, dense); m; m &= m - 1) {
            const int src = __ffs(m) - 1;
            const unsigned int from = __shfl_sync(0xffffffffu, run, src), n = __shfl_sync(0xffffffffu, c[k], src);
            const unsigned int owner = __shfl_sync(0xffffffffu, key + k, src);
            const unsigned int end = first_chunk(from + n, chunk_size);
            for (unsigned int ch = first_chunk(from, chunk_size) + (threadIdx.x & 31); ch < end; ch += 32)
                chunk_key[ch] = owner;
        }
        run += c[k];
    }
}

// Scan of the kScanTile keys from `base`, whose records and K-blocks follow `carry` and `kcarry`
// earlier ones; returns the tile's totals.
__device__ __forceinline__ void scan_tile(const unsigned int* __restrict__ counts, int base, int n_keys,
                                          unsigned int* __restrict__ offsets, unsigned int* __restrict__ cursor,
                                          unsigned int* __restrict__ kb_offsets, int kb_size,
                                          unsigned int* __restrict__ chunk_key, int chunk_size, unsigned int carry,
                                          unsigned int kcarry, unsigned int* tile, unsigned int* ktile,
                                          unsigned int* tmp, unsigned int& tot, unsigned int& ktot) {
    const int t = threadIdx.x;
    const int n = min(kScanTile, n_keys - base);
    for (int i = t; i < kScanTile; i += 1024) tile[i] = i < n ? counts[base + i] : 0u;
    __syncthreads();
    unsigned int c[kScanPer], s = 0, ks = 0;
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
        c[k] = tile[kScanPer * t + k];
        s += c[k];
        ks += (c[k] + kb_size - 1) / kb_size;
    }
    tot = ktot = 0;
    const unsigned int incl = block_scan(s, tmp, tot);
    const unsigned int kincl = kb_offsets ? block_scan(ks, tmp, ktot) : 0u;
    unsigned int run = carry + incl - s, krun = kcarry + kincl - ks;
    if (chunk_key && __any_sync(0xffffffffu, max(max(c[0], c[1]), max(c[2], c[3])) >= kDenseChunks * chunk_size))
        mark_dense(chunk_key, (unsigned int)chunk_size, run, c, (unsigned int)(base + kScanPer * t));
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
        if (chunk_key)
            mark_chunks(chunk_key, (unsigned int)chunk_size, run, c[k], (unsigned int)(base + kScanPer * t + k));
        tile[kScanPer * t + k] = run;
        run += c[k];
        ktile[kScanPer * t + k] = krun;
        krun += (c[k] + kb_size - 1) / kb_size;
    }
    __syncthreads();
    for (int i = t; i < n; i += 1024) {
        offsets[base + i] = tile[i];
        cursor[base + i] = tile[i];
        if (kb_offsets) kb_offsets[base + i] = ktile[i];
    }
    __syncthreads();
}

// One block over all keys.
__global__ void __launch_bounds__(1024) k_scan(const unsigned int* __restrict__ counts, int n_keys,
                                              unsigned int* __restrict__ offsets,
                                              unsigned int* __restrict__ cursor,
                                              unsigned int* __restrict__ kb_offsets, int kb_size,
                                              unsigned int* __restrict__ chunk_key, int chunk_size) {
    __shared__ __align__(16) unsigned int tile[kScanTile];
    __shared__ __align__(16) unsigned int ktile[kScanTile];
    __shared__ unsigned int tmp[32];
    unsigned int carry = 0, kcarry = 0;
    for (int base = 0; base < n_keys; base += kScanTile) {
        unsigned int tot, ktot;
        scan_tile(counts, base, n_keys, offsets, cursor, kb_offsets, kb_size, chunk_key, chunk_size, carry, kcarry, tile,
                  ktile, tmp, tot, ktot);
        carry += tot;
        kcarry += ktot;
    }
    if (threadIdx.x == 0) {
        offsets[n_keys] = carry;
        if (kb_offsets) kb_offsets[n_keys] = kcarry;
    }
}

// Many keys: a block per kScanTile keys, in two launches. The first writes each block's record and
// K-block totals; in the second every block adds up its predecessors' totals and scans its own tile.
// (147,456 keys of a 3072^2 grid at 8 x 8 tiles: 36 tiles one after another would take ~60 us.)
__global__ void __launch_bounds__(1024) k_scan_sums(const unsigned int* __restrict__ counts, int n_keys, int kb_size,
                                                   unsigned int* __restrict__ sums) {
    __shared__ unsigned int tmp[32];
    const int base = blockIdx.x * kScanTile;
    unsigned int s = 0, ks = 0;
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
        const int i = base + k * 1024 + (int)threadIdx.x;
        const unsigned int c = i < n_keys ? counts[i] : 0u;
        s += c;
        ks += (c + kb_size - 1) / kb_size;
    }
    unsigned int tot = 0, ktot = 0;
    block_scan(s, tmp, tot);
    block_scan(ks, tmp, ktot);
    if (threadIdx.x == 0) {
        sums[2 * blockIdx.x] = tot;
        sums[2 * blockIdx.x + 1] = ktot;
    }
}

__global__ void __launch_bounds__(1024) k_scan_tiles(const unsigned int* __restrict__ counts, int n_keys,
                                                    const unsigned int* __restrict__ sums,
                                                    unsigned int* __restrict__ offsets,
                                                    unsigned int* __restrict__ cursor,
                                                    unsigned int* __restrict__ kb_offsets, int kb_size,
                                                    unsigned int* __restrict__ chunk_key, int chunk_size) {
    __shared__ __align__(16) unsigned int tile[kScanTile];
    __shared__ __align__(16) unsigned int ktile[kScanTile];
    __shared__ unsigned int tmp[32];
    unsigned int s = 0, ks = 0, carry = 0, kcarry = 0;
    for (int b = threadIdx.x; b < (int)blockIdx.x; b += 1024) {
        s += sums[2 * b];
        ks += sums[2 * b + 1];
    }
    block_scan(s, tmp, carry);
    block_scan(ks, tmp, kcarry);
    unsigned int tot, ktot;
    scan_tile(counts, blockIdx.x * kScanTile, n_keys, offsets, cursor, kb_offsets, kb_size, chunk_key, chunk_size, carry,
              kcarry, tile, ktile, tmp, tot, ktot);
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
        offsets[n_keys] = carry + tot;
        if (kb_offsets) kb_offsets[n_keys] = kcarry + ktot;
    }
}

// NaN or +-Inf: all exponent bits set
__device__ __forceinline__ unsigned int nonfinite2(float a, float b) {
    return ((__float_as_uint(a) & 0x7f800000u) == 0x7f800000u) | ((__float_as_uint(b) & 0x7f800000u) == 0x7f800000u);
}

// Adds the warp's non-finite record count to *counter (one atomic per warp that saw any).
__device__ __forceinline__ void flush_nonfinite(unsigned long long* counter, unsigned int nbad) {
    if (!counter || !__any_sync(0xffffffffu, nbad != 0)) return;
    for (int o = 16; o > 0; o >>= 1) nbad += __shfl_xor_sync(0xffffffffu, nbad, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(counter, (unsigned long long)nbad);
}

// Scatter: block-aggregated reservation of output ranges per key, then 16-byte record writes.
__global__ void __launch_bounds__(kThreads) k_scatter(SampleSource src, GridGeom g, SlabParams sp,
                                                     unsigned int* __restrict__ cursor, int n_keys,
                                                     SampleRec* __restrict__ rec, float* __restrict__ rec_s,
                                                     unsigned int* __restrict__ vmax,
                                                     unsigned int* __restrict__ keymax,
                                                     const DevPlan* __restrict__ plan) {
    if (plan) {
        sp = plan->sp;
        src.inv_det = plan->inv_det;
    }
    extern __shared__ unsigned int sh[];  // [n_keys] counts, then [n_keys] bases
    unsigned int* cnt = sh;
    unsigned int* base = sh + n_keys;
    const bool use_smem = n_keys <= kSmemKeyLimit / 2;
    const int lane = threadIdx.x & 31;
    const long long n = src.n;
    float vm = 0.0f;  // max |record value| written by this thread
    unsigned int nbad = 0;  // non-finite records written by this thread
    for (long long c0 = (long long)blockIdx.x * kChunk; c0 < n; c0 += (long long)gridDim.x * kChunk) {
        KeyRec kr[kPerThread];
        unsigned int rank[kPerThread];
        if (use_smem) {
            for (int k = threadIdx.x; k < n_keys; k += kThreads) cnt[k] = 0;
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < kPerThread; ++i) {
            const long long idx = c0 + i * kThreads + threadIdx.x;
            kr[i].key = -2;
            if (idx < n) kr[i] = sample_key(src, idx, g, sp);
            const int key = kr[i].key;
            const unsigned int peers = __match_any_sync(0xffffffffu, key);
            const int leader = __ffs(peers) - 1;
            const unsigned int before = __popc(peers & ((1u << lane) - 1u));
            unsigned int b0 = 0;
            if (key >= 0 && lane == leader)
                b0 = use_smem ? atomicAdd(&cnt[key], __popc(peers)) : atomicAdd(&cursor[key], __popc(peers));
            b0 = __shfl_sync(0xffffffffu, b0, leader);
            rank[i] = b0 + before;
        }
        if (use_smem) {
            __syncthreads();
            for (int k = threadIdx.x; k < n_keys; k += kThreads) {
                const unsigned int c = cnt[k];
                base[k] = c ? atomicAdd(&cursor[k], c) : 0u;
            }
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < kPerThread; ++i) {
            const long long idx = c0 + i * kThreads + threadIdx.x;
            const int key = kr[i].key;
            if (key < 0) continue;
            const unsigned int pos = use_smem ? base[key] + rank[i] : rank[i];
            SampleRec r;
            r.xq = kr[i].xq;
            r.yq = kr[i].yq;
            r.vre = __fmul_rn(src.vr[idx], src.inv_det);
            r.vim = __fmul_rn(src.vi[idx], src.inv_det);
            rec[pos] = r;
            if (rec_s) rec_s[pos] = kr[i].s;
            nbad += nonfinite2(r.vre, r.vim);
            const float m = fmaxf(fabsf(r.vre), fabsf(r.vim));
            vm = fmaxf(vm, m);
            if (keymax && m > 0.0f) atomicMax(&keymax[key], __float_as_uint(m));
        }
        if (use_smem) __syncthreads();
    }
    flush_nonfinite(src.nonfinite, nbad);
    if (vmax) {  // non-negative floats order like their bit patterns
        const unsigned int mb = __reduce_max_sync(0xffffffffu, __float_as_uint(vm));
        if (lane == 0 && mb) atomicMax(vmax, mb);
    }
}

// Separable sources (r = s[chan] q[row], idx = row + chan R). A warp takes units of UR
// rows x one chunk of `lpr` channels (lpr a power of two <= 32): lane -> (row subset
// lane / lpr, channel lane % lpr), so consecutive lanes hold consecutive channels of one row. The
// channels of a baseline mostly share a tile, so runs of equal keys are long: one shared-memory or
// global atomic per run, and a run's records land in consecutive slots. No 64-bit division.
// UR = 16, or 4 where 16 would leave most of the chip idle: a unit is a serial chain of row steps (FP64 key
// rule, a run search, a returning cursor atomic in the scatter). 130 k samples: both and the scan 41 -> 27 us;
// 8.4 M samples keep 16, whose staging loads are whole 64-byte pieces. What bounds them is latency: 130
// (histogram) and 240 warp instructions per 32 samples at 50-70 % of the issue slots; four CTAs per SM for the
// scatter took it from 127 to 110 us at 8.4 M samples.
constexpr int kUnitRows = 16, kUnitRowsSmall = 4;

struct SepMap {
    int lpr;       // lanes per row (channels per chunk)
    int nch;       // channel chunks
    int nrt;       // row tiles of UR
    int C;
};

__device__ inline void unit_of(long long u, const SepMap& m, int& rt, int& ch) {
    rt = (int)(u / m.nch);
    ch = (int)(u - (long long)rt * m.nch);
}

// The lanes of a warp that place their records together. Runs of equal keys on consecutive lanes: consecutive
// channels of one baseline mostly stay in a tile and do not come back to one. One shuffle and one vote; a match over
// the warp costs several times that on the unit the atomics share (8.4 M samples of 64 channels: 195 instead of 185
// us).
template <bool ROWS>
struct LaneGroup {
    int first = 0, length = 0;
    __device__ __forceinline__ void find(int key, int lane) {
        const int before = __shfl_up_sync(0xffffffffu, key, 1);
        const unsigned int starts = __ballot_sync(0xffffffffu, lane == 0 || key != before);
        first = 31 - __clz(starts & (0xffffffffu >> (31 - lane)));
        const unsigned int after = starts & ~(0xffffffffu >> (31 - lane));
        length = (after ? __ffs(after) - 1 : 32) - first;
    }
    __device__ __forceinline__ int leader() const { return first; }
    __device__ __forceinline__ unsigned int count() const { return (unsigned int)length; }
    __device__ __forceinline__ unsigned int rank(int lane) const { return (unsigned int)(lane - first); }
    __device__ __forceinline__ unsigned int lanes() const { return (0xffffffffu >> (32 - length)) << first; }
};
// Several rows per warp (fewer than 17 channels): keys may repeat apart, as in the few tiles of a compact array, where
// each sample was an atomic of its own on one address (2 M samples of one channel in four tiles: binning 1.37 ms, with
// the match 0.17; spread over the grid 127 and 134 us). So many runs are matched.
template <>
struct LaneGroup<true> {
    unsigned int mask = 1;
    __device__ __forceinline__ void find(int key, int lane) {
        const int before = __shfl_up_sync(0xffffffffu, key, 1);
        const unsigned int starts = __ballot_sync(0xffffffffu, lane == 0 || key != before);
        if (__popc(starts) > 8) {
            mask = __match_any_sync(0xffffffffu, key);
            return;
        }
        const unsigned int upto = 0xffffffffu >> (31 - lane), after = starts & ~upto;
        mask = (after ? (after & (0u - after)) - 1u : 0xffffffffu) & (0xffffffffu << (31 - __clz(starts & upto)));
    }
    __device__ __forceinline__ int leader() const { return __ffs(mask) - 1; }
    __device__ __forceinline__ unsigned int count() const { return (unsigned int)__popc(mask); }
    __device__ __forceinline__ unsigned int rank(int lane) const { return (unsigned int)__popc(mask & ((1u << lane) - 1u)); }
    __device__ __forceinline__ unsigned int lanes() const { return mask; }
};

template <int UR, bool ROWS>
__global__ void __launch_bounds__(kThreads) k_histogram_sep(SampleSource src, SepMap m, GridGeom g, SlabParams sp,
                                                           unsigned int* __restrict__ counts, int n_keys,
                                                           unsigned long long* __restrict__ dropped,
                                                           const DevPlan* __restrict__ plan) {
    if (plan && first_thread()) {
        unsigned long long* const stamps = plan_stamps(plan);
        stamps[STAMP_BIN] = stamp_now();
        stamps[STAMP_FFT] = stamps[STAMP_END] = 0;  // maxima over the blocks of later kernels
    }
    if (plan) sp = plan->sp;
    extern __shared__ unsigned int sh[];
    const bool use_smem = n_keys <= kSmemKeyLimit;
    if (use_smem) {
        for (int k = threadIdx.x; k < n_keys; k += kThreads) sh[k] = 0;
        __syncthreads();
    }
    const int lane = threadIdx.x & 31;
    const int rps = 32 / m.lpr, sub = lane / m.lpr, coff = lane % m.lpr;
    const long long nunits = (long long)m.nrt * m.nch;
    const long long nwarps = (long long)gridDim.x * (kThreads / 32);
    unsigned int ndrop = 0;
    for (long long u = (long long)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5); u < nunits; u += nwarps) {
        int rt, ch;
        unit_of(u, m, rt, ch);
        const int c = ch * m.lpr + coff;
        const bool cvalid = c < m.C;
        const double sc = cvalid ? src.s[c] : 0.0;
        // every lane takes every step (the votes need the whole warp); rows past the unit have no key
        for (int i0 = 0; i0 < UR; i0 += rps) {
            const int i = i0 + sub;
            const long long row = (long long)rt * UR + i;
            int key = -2;
            if (cvalid && i < UR && row < src.R) {
                const double* q = src.q + row * 3;
                key = row_chan_key(sc, q[0], q[1], q[2], g, sp).key;
                if (key < 0) ++ndrop;
            }
            LaneGroup<ROWS> group;
            group.find(key, lane);
            if (key >= 0 && lane == group.leader()) {
                if (use_smem) atomicAdd(&sh[key], group.count());
                else atomicAdd(&counts[key], group.count());
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) ndrop += __shfl_xor_sync(0xffffffffu, ndrop, o);
    if (lane == 0 && ndrop) atomicAdd(dropped, (unsigned long long)ndrop);
    if (use_smem) {
        __syncthreads();
        for (int k = threadIdx.x; k < n_keys; k += kThreads)
            if (sh[k]) atomicAdd(&counts[k], sh[k]);
    }
}

// Scatter for separable sources: per unit, the warp stages the unit's collapsed visibilities in
// shared memory with row-contiguous loads, then writes each group's records to the slots one
// global atomic on the key's cursor reserved.
template <int UR, bool ROWS>
__global__ void __launch_bounds__(kThreads, 4) k_scatter_sep(SampleSource src, SepMap m, GridGeom g, SlabParams sp,
                                                         unsigned int* __restrict__ cursor,
                                                         SampleRec* __restrict__ rec, float* __restrict__ rec_s,
                                                         unsigned int* __restrict__ vmax,
                                                         unsigned int* __restrict__ keymax,
                                                         const DevPlan* __restrict__ plan) {
    if (plan) {
        sp = plan->sp;
        src.inv_det = plan->inv_det;
    }
    constexpr int kVisPitch = UR + 1;   // float2 pitch of a staged channel (bank-conflict free)
    __shared__ float2 stage[kThreads / 32][32 * kVisPitch];
    float2* my = stage[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int rps = 32 / m.lpr, sub = lane / m.lpr, coff = lane % m.lpr;
    const long long nunits = (long long)m.nrt * m.nch;
    const long long nwarps = (long long)gridDim.x * (kThreads / 32);
    const long long R = src.R;
    float vm = 0.0f;
    unsigned int nbad = 0;
    for (long long u = (long long)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5); u < nunits; u += nwarps) {
        int rt, ch;
        unit_of(u, m, rt, ch);
        const long long row0 = (long long)rt * UR;
        const int c0 = ch * m.lpr;
        // stage: UR lanes read UR consecutive rows of a channel, 32 / UR channels at a time
        __syncwarp();
        for (int k = 0; k < m.lpr; k += 32 / UR) {
            const int cc = k + lane / UR;
            const long long row = row0 + lane % UR;
            float2 v = make_float2(0.0f, 0.0f);
            if (c0 + cc < m.C && row < R) {
                const long long idx = row + (long long)(c0 + cc) * R;
                v = make_float2(src.vr[idx], src.vi[idx]);
            }
            my[cc * kVisPitch + lane % UR] = v;
        }
        __syncwarp();
        const int c = c0 + coff;
        const bool cvalid = c < m.C;
        const double sc = cvalid ? src.s[c] : 0.0;
        // every lane takes every step; a step's records are written after the next step's keys, so that the
        // latency of its cursor atomic is covered
        KeyRec last;
        last.key = -1;
        LaneGroup<ROWS> last_group;
        int last_i = 0;
        unsigned int last_base = 0;
        for (int i0 = 0; i0 < UR + rps; i0 += rps) {
            KeyRec kr;
            kr.key = -2;
            const int i = i0 + sub;
            LaneGroup<ROWS> group;
            unsigned int base = 0;
            if (i0 < UR) {
                const long long row = row0 + i;
                if (cvalid && i < UR && row < R) {
                    const double* q = src.q + row * 3;
                    kr = row_chan_key(sc, q[0], q[1], q[2], g, sp);
                }
                group.find(kr.key, lane);
                if (kr.key >= 0 && lane == group.leader()) base = atomicAdd(&cursor[kr.key], group.count());
            }
            if (i0 > 0) {
                const unsigned int b0 = __shfl_sync(0xffffffffu, last_base, last_group.leader());
                if (last.key >= 0) {
                    const unsigned int pos = b0 + last_group.rank(lane);
                    const float2 v = my[coff * kVisPitch + last_i];
                    SampleRec r;
                    r.xq = last.xq;
                    r.yq = last.yq;
                    r.vre = __fmul_rn(v.x, src.inv_det);
                    r.vim = __fmul_rn(v.y, src.inv_det);
                    rec[pos] = r;
                    if (rec_s) rec_s[pos] = last.s;
                    nbad += nonfinite2(r.vre, r.vim);
                    const float m = fmaxf(fabsf(r.vre), fabsf(r.vim));
                    vm = fmaxf(vm, m);
                    if (keymax) {  // the group's maximum, one atomic per group
                        const unsigned int gm = __reduce_max_sync(last_group.lanes(), __float_as_uint(m));
                        if (lane == last_group.leader() && gm) atomicMax(&keymax[last.key], gm);
                    }
                }
            }
            last = kr;
            last_i = i;
            last_group = group;
            last_base = base;
        }
    }
    flush_nonfinite(src.nonfinite, nbad);
    if (vmax) {  // non-negative floats order like their bit patterns
        const unsigned int mb = __reduce_max_sync(0xffffffffu, __float_as_uint(vm));
        if (lane == 0 && mb) atomicMax(vmax, mb);
    }
}

SepMap sep_map(const SampleSource& src, int unit_rows) {
    SepMap m{};
    m.C = (int)(src.n / src.R);
    m.lpr = 2;
    while (m.lpr < 32 && m.lpr < m.C) m.lpr <<= 1;
    m.nch = (m.C + m.lpr - 1) / m.lpr;
    m.nrt = (int)((src.R + unit_rows - 1) / unit_rows);
    return m;
}

// Rows per unit: short units until they fill four 8-warp blocks per SM.
int unit_rows(const SampleSource& src) {
    const long long chunks = (src.n / src.R + 31) / 32;
    return (src.R + kUnitRows - 1) / kUnitRows * chunks < 32LL * current_sm_count() ? kUnitRowsSmall : kUnitRows;
}

// Separable kernels need whole rows x channels and 32-bit unit and row counts.
bool use_sep(const SampleSource& src) {
    return !src.bin && src.R > 0 && src.n % src.R == 0 && src.n / src.R <= (1LL << 20) &&
           (src.R + kUnitRows - 1) / kUnitRows * ((src.n / src.R + 31) / 32) < (1LL << 31);
}

}  // namespace

int launch_histogram(const SampleSource& src, const GridGeom& g, const SlabParams& sp,
                     unsigned int* d_counts, int n_keys, unsigned long long* d_dropped,
                     cudaStream_t st, const DevPlan* d_plan) {
    const size_t smem = n_keys <= kSmemKeyLimit ? (size_t)n_keys * 4 : 0;
    if (use_sep(src)) {
        const int ur = unit_rows(src);
        const SepMap m = sep_map(src, ur);
        auto kern = m.lpr < 32 ? (ur == kUnitRows ? k_histogram_sep<kUnitRows, true> : k_histogram_sep<kUnitRowsSmall, true>)
                               : (ur == kUnitRows ? k_histogram_sep<kUnitRows, false> : k_histogram_sep<kUnitRowsSmall, false>);
        SVDI_TRY(ensure_dynamic_smem((const void*)kern, smem));
        const long long units = (long long)m.nrt * m.nch;
        long long blocks = (units + kThreads / 32 - 1) / (kThreads / 32);
        if (blocks > 4LL * current_sm_count()) blocks = 4LL * current_sm_count();   // a few units per warp: the shared histogram is flushed once
        if (blocks < 1) blocks = 1;
        kern<<<(int)blocks, kThreads, smem, st>>>(src, m, g, sp, d_counts, n_keys, d_dropped, d_plan);
        SVDI_LAUNCHED();
        return SVDI_OK;
    }
    SVDI_TRY(ensure_dynamic_smem((const void*)k_histogram, smem));
    long long blocks = (src.n + kThreads - 1) / kThreads;
    if (blocks > 8LL * current_sm_count()) blocks = 8LL * current_sm_count();
    if (blocks < 1) blocks = 1;
    k_histogram<<<(int)blocks, kThreads, smem, st>>>(src, g, sp, d_counts, n_keys, d_dropped, d_plan);
    SVDI_LAUNCHED();
    return SVDI_OK;
}

size_t scan_sums_words(long long n_keys) { return 2 * (size_t)((n_keys + kScanTile - 1) / kScanTile); }

int launch_scan(const unsigned int* d_counts, int n_keys, unsigned int* d_offsets,
                unsigned int* d_cursor, cudaStream_t st, unsigned int* d_kb_offsets, int kb_size,
                unsigned int* d_chunk_key, int chunk_size, unsigned int* d_sums) {
    if (!d_sums || n_keys <= kScanTile) {
        k_scan<<<1, 1024, 0, st>>>(d_counts, n_keys, d_offsets, d_cursor, d_kb_offsets, kb_size, d_chunk_key, chunk_size);
        SVDI_LAUNCHED();
        return SVDI_OK;
    }
    const int blocks = (n_keys + kScanTile - 1) / kScanTile;
    k_scan_sums<<<blocks, 1024, 0, st>>>(d_counts, n_keys, kb_size, d_sums);
    SVDI_LAUNCHED();
    k_scan_tiles<<<blocks, 1024, 0, st>>>(d_counts, n_keys, d_sums, d_offsets, d_cursor, d_kb_offsets, kb_size,
                                          d_chunk_key, chunk_size);
    SVDI_LAUNCHED();
    return SVDI_OK;
}

int launch_scatter(const SampleSource& src, const GridGeom& g, const SlabParams& sp,
                   unsigned int* d_cursor, int n_keys, SampleRec* d_rec, float* d_rec_s,
                   unsigned int* d_vmax, cudaStream_t st, unsigned int* d_keymax, const DevPlan* d_plan) {
    if (use_sep(src)) {
        const int ur = unit_rows(src);
        const SepMap m = sep_map(src, ur);
        auto kern = m.lpr < 32 ? (ur == kUnitRows ? k_scatter_sep<kUnitRows, true> : k_scatter_sep<kUnitRowsSmall, true>)
                               : (ur == kUnitRows ? k_scatter_sep<kUnitRows, false> : k_scatter_sep<kUnitRowsSmall, false>);
        const long long units = (long long)m.nrt * m.nch;
        long long blocks = (units + kThreads / 32 - 1) / (kThreads / 32);
        if (blocks > 8LL * current_sm_count()) blocks = 8LL * current_sm_count();
        if (blocks < 1) blocks = 1;
        kern<<<(int)blocks, kThreads, 0, st>>>(src, m, g, sp, d_cursor, d_rec, d_rec_s, d_vmax, d_keymax,
                                                        d_plan);
        SVDI_LAUNCHED();
        return SVDI_OK;
    }
    const size_t smem = n_keys <= kSmemKeyLimit / 2 ? (size_t)n_keys * 8 : 0;
    SVDI_TRY(ensure_dynamic_smem((const void*)k_scatter, smem));
    long long blocks = (src.n + kChunk - 1) / kChunk;
    if (blocks > 16LL * current_sm_count()) blocks = 16LL * current_sm_count();
    if (blocks < 1) blocks = 1;
    k_scatter<<<(int)blocks, kThreads, smem, st>>>(src, g, sp, d_cursor, n_keys, d_rec, d_rec_s, d_vmax, d_keymax,
                                                   d_plan);
    SVDI_LAUNCHED();
    return SVDI_OK;
}

}  // namespace svdi
