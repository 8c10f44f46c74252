// ES gridder on warp-level matrix instructions (support W <= 8, any number of Chebyshev terms).
//
// Samples arrive binned by 8 x 8 tiles of footprint origins (binning.cu), so every footprint of a
// tile lies in one 16 x 16 region of grid cells, and the region's sum over samples is a matrix
// product: C[row][col] = sum_k A[row][k] B[k][col], A the row weights and B the column weights times
// the visibility (16 complex columns = 32 real ones). A warp keeps the region in registers (16 x 32
// values, 16 per lane and term), so samples cost no memory reductions at all; the region is added to
// the moment plane with red.global.add.v2.f32 once per run of one tile's records.
//
// Precision: FP32 weights and values are split into FP16 hi + lo parts (22 significand bits, values
// scaled by the batch's largest |v| to 2^14, weights by 2^14), and hi hi + hi lo + lo hi are formed by
// mma.sync m16n8k16 with FP32 accumulation. Matrix accumulation truncates, so a product of at most 32 samples
// is added to the FP32 registers with an ordinary (rounding) FMA, which also undoes the scales; what it
// truncates, a measured mean of 1.0e-7 of the sum at every density tried (2,000 to 2 M samples on 96^2 and
// 192^2 grids), is put back by the last bit of the inverse scale.
//
// A footprint covers 8 consecutive rows of the 16, i.e. every residue mod 8 exactly once: the taps are
// staged by residue (8 words per sample and axis, one 32-bit word = hi | lo << 16) and the zero half
// of the operand is made with a mask, (residue >= origin) ? low half : high half.
//
// Work: chunks of consecutive records (the scan's table names each chunk's first tile key), taken by
// single warps from a counter; a batch of 32 records is staged lane-per-record (36 + 36 FMAs for the 16
// taps: the even and odd parts of a piece's polynomial also give the mirrored piece), then 16-record
// steps run for every tile segment the batch holds. Footprints that W x W taps cannot hold (exactly
// integer positions, W + 1 cells; clipped at the low grid edge) go straight to the plane, after the chunk's end.
//
// A tile's region and its right neighbour's share eight columns: a warp that moves on to that
// neighbour (the next key) keeps them in its registers and reduces only the left half.
//
// What bounds it: issue slots (32 warp instructions per sample at two terms: 11 staging, 11 products,
// the rest per tile), then the L2's reductions (16-byte reductions of 64-byte row pieces add 4.7 TB/s,
// 8-byte ones of 32-byte pieces 3.3 TB/s: hence the column order of b_row). Gridding stage, B200, against the
// fixed-point shared-memory gridder (gridder.cu, which keeps supports above 8 and the explicit tile
// sizes 32 and 64): 6.5 M samples, 2 terms, 3072^2 grid 0.541 -> 0.321 ms; 1.04 M, 2 terms, 1536^2
// 0.324 -> 0.085 ms; support 6 at 2048^2 0.590 -> 0.094 ms; 130 k samples, 8 terms, 384^2 0.119 ->
// 0.042 ms; 0.64 M samples, 59 terms, 2304^2 7.7 -> 3.1 ms. Error against 64 bits over 143 random images:
// median 0.86, at most 1.03 of that gridder's.
#include "svdi_internal.cuh"

#include <cuda_fp16.h>

#include <type_traits>

namespace svdi {

namespace {

constexpr int kPitch = 40;      // words per residue row of a staged batch: 32 records, rows 8 banks apart
constexpr int kWarps = 4;       // warps per CTA (they never synchronise with one another)
constexpr float kWeightScale = 16384.0f;  // 2^14

// Even and odd parts of the ES pieces in u = 2 f - 1: piece i = even + u odd, piece W - 1 - i = even -
// u odd. Row pieces carry the factor 2^14 of the FP16 split.
struct MmaPoly {
    float ex[4][5], ox[4][4];
    float ey[4][5], oy[4][4];
    float beta;
};

// n / d for 0 <= n < 2^26 and 1 <= d <= 2^26 as (n mul) >> shift, exact: mul = ceil(2^shift / d) with
// shift = 26 + ceil(log2 d), so the error n (mul d - 2^shift) / (d 2^shift) stays below 1 / d.
struct FastDiv {
    unsigned int mul, shift, d;
};
FastDiv fast_div(int d) {
    unsigned int s = 0;
    while ((1u << s) < (unsigned int)d) ++s;
    const unsigned long long p = 1ull << (26 + s);
    return {(unsigned int)((p + (unsigned long long)d - 1) / (unsigned long long)d), 26 + s, (unsigned int)d};
}
__device__ __forceinline__ int div_by(int n, const FastDiv& f) {
    return (int)(((unsigned long long)(unsigned int)n * f.mul) >> f.shift);
}

__device__ __forceinline__ void red_add_v4(float2* addr, float a, float b, float c, float d) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(a), "f"(b), "f"(c), "f"(d)
                 : "memory");
}

__device__ __forceinline__ void red_add_v2(float2* addr, float a, float b) {
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(addr), "f"(a), "f"(b) : "memory");
}

// Exact ES kernel psi(x) = exp(beta (sqrt(1 - x^2) - 1)) without cancellation (rare path).
__device__ __forceinline__ float es_exact(float beta, float x) {
    if (fabsf(x) > 1.0f) return 0.0f;
    return expf(-beta * x * x / (1.0f + sqrtf((1.0f - x) * (1.0f + x))));
}

__device__ __forceinline__ void mma_f16(float (&c)[4], const unsigned int (&a)[4], unsigned int b0, unsigned int b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// packed pairs of floats (one instruction for two FP32 operations)
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// the pair (x, y) as FP16 hi + lo, each value as one word hi | lo << 16
__device__ __forceinline__ void split2(unsigned long long xy, unsigned int& wx, unsigned int& wy) {
    const float2 v = unpack2(xy);
    const __half2 h = __floats2half2_rn(v.x, v.y);
    const float2 hf = __half22float2(h);
    const float2 d = unpack2(fma2(pack2(hf.x, hf.y), pack2(-1.0f, -1.0f), xy));  // exact
    const __half2 l = __floats2half2_rn(d.x, d.y);
    const unsigned int hb = *reinterpret_cast<const unsigned int*>(&h), lb = *reinterpret_cast<const unsigned int*>(&l);
    wx = __byte_perm(hb, lb, 0x5410);
    wy = __byte_perm(hb, lb, 0x7632);
}

template <int W>
__device__ __forceinline__ void taps(const float (&e)[4][5], const float (&o)[4][4], float u, float (&w)[W]) {
    const float v = u * u;
#pragma unroll
    for (int i = 0; i < W / 2; ++i) {
        const float ev = fmaf(fmaf(fmaf(fmaf(e[i][4], v, e[i][3]), v, e[i][2]), v, e[i][1]), v, e[i][0]);
        const float od = fmaf(fmaf(fmaf(o[i][3], v, o[i][2]), v, o[i][1]), v, o[i][0]);
        w[i] = fmaf(u, od, ev);
        w[W - 1 - i] = fmaf(-u, od, ev);
    }
}

// Sums of dense tiles. A tile of very many records would be added to its cells once per chunk, thousands of
// FP32 roundings at the size of the whole sum. So a group of 2^shift chunks that lies inside one tile is
// summed in a slot of its own, one per group and term, in the order of the accumulator registers; the
// group's last chunk adds the slot to the plane and leaves it and the group's arrival counter as zeros.
// Error against 64 bits of dense-core images (0.3 to 0.6 M samples, chunks added singly / through slots): 1.1e-6
// / 2.8e-7, 1.5e-6 / 5.3e-7, 5.1e-7 / 2.5e-7. Time: the wait for the arrival counter costs 2 us where all is
// dense (130 k samples in a few tiles, 8 terms: gridding 25 -> 27 us); fewer reductions of one address save 3 % at 6.5 M samples (0.331
// -> 0.318 ms).
struct DenseSlots {
    float4* sums;           // [group][term][kSlotWords]
    unsigned int* arrived;  // [group][term]
    unsigned int shift;
};
constexpr int kSlotWords = 128;  // 16-byte words per slot: 16 x 16 complex cells

template <int KC>
struct alignas(16) WarpStage {  // one after another in shared memory, read 8 bytes at a time
    unsigned int a[KC][8 * kPitch];      // [term][row residue][record]: T_n(s) times the row weight
    unsigned int b[16 * kPitch];         // [b_row(column residue) + (re, im)][record]: column weight times v
    __half oa[32], ob[32];               // footprint origins (row, column) in the region
    unsigned int rare;                   // batches of the chunk (8 at most) with rare records (rare_records)
};

// Column residues 0, 2, 4, 6 and then 1, 3, 5, 7, real and imaginary rows each: fragment tile (half,
// odd) holds columns 8 half + 2 q + odd, so a lane's two tiles of a half are adjacent cells.
__device__ __forceinline__ int b_row(int residue) { return (residue & 6) + 8 * (residue & 1); }

// CTAs per SM the register budget is set for
template <int KC>
constexpr int min_ctas() { return KC == 1 ? 5 : (KC == 2 ? 4 : 3); }

__device__ __forceinline__ void mma_f16_k8(float (&c)[4], unsigned int a0, unsigned int a1, unsigned int b0) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(b0));
}

// The B fragments (hi and lo parts of the four column tiles) of the 16 records from k0, records outside
// [lo, hi) as zeros. Register half h holds the plane columns of parity h of column / 8: the region's
// left half for an even tile (odd = 0), its right half for an odd one (odd = ~0).
struct BFrag {
    unsigned int h[4][2], l[4][2];
};
template <class Stage>
__device__ __forceinline__ void load_b(const Stage& st, int k0, int lo, int hi, int gr, int tq, __half2 res0,
                                       __half2 res1, unsigned int odd, BFrag& f) {
    const int kp = k0 + 2 * tq;
    const __half2 ob0 = *reinterpret_cast<const __half2*>(&st.ob[kp]);
    const __half2 ob1 = *reinterpret_cast<const __half2*>(&st.ob[kp + 8]);
    unsigned int s0 = 0xffffffffu, s8 = 0xffffffffu;
    if (lo > k0 || hi < k0 + 16) {
        auto in = [&](int k) { return k >= lo && k < hi; };
        s0 = (in(kp) ? 0xffffu : 0u) | (in(kp + 1) ? 0xffff0000u : 0u);
        s8 = (in(kp + 8) ? 0xffffu : 0u) | (in(kp + 9) ? 0xffff0000u : 0u);
    }
#pragma unroll
    for (int up = 0; up < 2; ++up) {  // column residues 2 (gr / 2) and 2 (gr / 2) + 1
        const unsigned int m0 = __hge2_mask(up ? res1 : res0, ob0) ^ odd, m1 = __hge2_mask(up ? res1 : res0, ob1) ^ odd;
        const uint2 w0 = *reinterpret_cast<const uint2*>(&st.b[(gr + 8 * up) * kPitch + kp]);
        const uint2 w1 = *reinterpret_cast<const uint2*>(&st.b[(gr + 8 * up) * kPitch + kp + 8]);
        const unsigned int h0 = __byte_perm(w0.x, w0.y, 0x5410), l0 = __byte_perm(w0.x, w0.y, 0x7632);
        const unsigned int h1 = __byte_perm(w1.x, w1.y, 0x5410), l1 = __byte_perm(w1.x, w1.y, 0x7632);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const unsigned int x0 = (half ? ~m0 : m0) & s0, x1 = (half ? ~m1 : m1) & s8;
            f.h[2 * half + up][0] = h0 & x0;
            f.h[2 * half + up][1] = h1 & x1;
            f.l[2 * half + up][0] = l0 & x0;
            f.l[2 * half + up][1] = l1 & x1;
        }
    }
}

template <class Stage>
__device__ __forceinline__ void load_a(const Stage& st, int t, int k0, int gr, int tq, unsigned int m0, unsigned int m1,
                                       unsigned int (&ahi)[4], unsigned int (&alo)[4]) {
    const int kp = k0 + 2 * tq;
    const uint2 w0 = *reinterpret_cast<const uint2*>(&st.a[t][gr * kPitch + kp]);
    const uint2 w1 = *reinterpret_cast<const uint2*>(&st.a[t][gr * kPitch + kp + 8]);
    const unsigned int h0 = __byte_perm(w0.x, w0.y, 0x5410), l0 = __byte_perm(w0.x, w0.y, 0x7632);
    const unsigned int h1 = __byte_perm(w1.x, w1.y, 0x5410), l1 = __byte_perm(w1.x, w1.y, 0x7632);
    ahi[0] = h0 & m0;
    ahi[1] = h0 & ~m0;
    ahi[2] = h1 & m1;
    ahi[3] = h1 & ~m1;
    alo[0] = l0 & m0;
    alo[1] = l0 & ~m0;
    alo[2] = l1 & m1;
    alo[3] = l1 & ~m1;
}

// acc += inv * (A B) over the NW windows of 16 records that start at k0 and k1 (k1 may lie inside the
// first window: its records below k0 + 16 are masked)
template <int NW, int KC>
__device__ __forceinline__ void products(const WarpStage<KC>& st, int k0, int k1, int lo, int hi, int gr, int tq,
                                         __half2 row_res, __half2 res0, __half2 res1, unsigned int odd, float inv,
                                         float (&acc)[KC][4][4]) {
    BFrag b[NW];
#pragma unroll
    for (int w = 0; w < NW; ++w) {
        const int k = w ? k1 : k0;
        asm volatile("" ::: "memory");  // one window's loads after the other's: registers are short
        load_b(st, k, w ? k0 + 16 : lo, hi, gr, tq, res0, res1, odd, b[w]);
    }
#pragma unroll
    for (int t = 0; t < KC; ++t) {
        float c[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) c[j][q] = 0.0f;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            unsigned int ahi[4], alo[4];
            const int k = (w ? k1 : k0) + 2 * tq;
            load_a(st, t, w ? k1 : k0, gr, tq, __hge2_mask(row_res, *reinterpret_cast<const __half2*>(&st.oa[k])),
                   __hge2_mask(row_res, *reinterpret_cast<const __half2*>(&st.oa[k + 8])), ahi, alo);
#pragma unroll
            for (int j = 0; j < 4; ++j) mma_f16(c[j], alo, b[w].h[j][0], b[w].h[j][1]);
#pragma unroll
            for (int j = 0; j < 4; ++j) mma_f16(c[j], ahi, b[w].l[j][0], b[w].l[j][1]);
#pragma unroll
            for (int j = 0; j < 4; ++j) mma_f16(c[j], ahi, b[w].h[j][0], b[w].h[j][1]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[t][j][q] = fmaf(c[j][q], (j & 1) ? -inv : inv, acc[t][j][q]);
    }
}

// acc += inv * (A B) over the window of 8 records that starts at k0: segments of few records
template <int KC>
__device__ __forceinline__ void products8(const WarpStage<KC>& st, int k0, int lo, int hi, int gr, int tq,
                                          __half2 row_res, __half2 res0, __half2 res1, unsigned int odd, float inv,
                                          float (&acc)[KC][4][4]) {
    const int kp = k0 + 2 * tq;
    const __half2 ob = *reinterpret_cast<const __half2*>(&st.ob[kp]);
    const unsigned int m = __hge2_mask(row_res, *reinterpret_cast<const __half2*>(&st.oa[kp]));
    const unsigned int s = (kp >= lo && kp < hi ? 0xffffu : 0u) | (kp + 1 >= lo && kp + 1 < hi ? 0xffff0000u : 0u);
    unsigned int bh[4], bl[4];
#pragma unroll
    for (int up = 0; up < 2; ++up) {
        const unsigned int mb = __hge2_mask(up ? res1 : res0, ob) ^ odd;
        const uint2 w = *reinterpret_cast<const uint2*>(&st.b[(gr + 8 * up) * kPitch + kp]);
        const unsigned int h = __byte_perm(w.x, w.y, 0x5410), l = __byte_perm(w.x, w.y, 0x7632);
        bh[up] = h & mb & s;
        bl[up] = l & mb & s;
        bh[2 + up] = h & ~mb & s;
        bl[2 + up] = l & ~mb & s;
    }
#pragma unroll
    for (int t = 0; t < KC; ++t) {
        const uint2 w = *reinterpret_cast<const uint2*>(&st.a[t][gr * kPitch + kp]);
        const unsigned int h = __byte_perm(w.x, w.y, 0x5410), l = __byte_perm(w.x, w.y, 0x7632);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            mma_f16_k8(c, l & m, l & ~m, bh[j]);
            mma_f16_k8(c, h & m, h & ~m, bl[j]);
            mma_f16_k8(c, h & m, h & ~m, bh[j]);
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[t][j][q] = fmaf(c[q], (j & 1) ? -inv : inv, acc[t][j][q]);
        }
    }
}

// A record whose footprint W x W taps cannot hold: exactly integer positions (W + 1 cells), or clipped at the low
// grid edge.
template <int W>
__device__ __forceinline__ bool odd_footprint(const SampleRec& r) {
    return (r.xq & 0xFFFFFF) == 0 || (r.yq & 0xFFFFFF) == 0 || (r.xq >> 24) < W / 2 - 1 || (r.yq >> 24) < W / 2 - 1;
}
// The larger component's magnitude as bits (in the order of the magnitudes; 0x7f800000 and up: not finite).
__device__ __forceinline__ unsigned int value_bits(const SampleRec& r) {
    return max(__float_as_uint(r.vre) & 0x7fffffffu, __float_as_uint(r.vim) & 0x7fffffffu);
}
constexpr unsigned int kNotFinite = 0x7f800000u;
// The batch's scale is its largest value's, and in a launch over several snapshots a batch may hold the records of
// two. So that one snapshot's values cannot cost another's records their bits, a record 2^20 times smaller than the
// largest, or not finite, is rare too (2^-19 of it, 22 bits of all others, is left to the split).
constexpr unsigned int kScaleSpan = 20u << 23;

// The rare records of the batch [b0, b1), whose keys are `key` or later (returns the last one): exact ES formula,
// lanes over cells, straight to the planes. Records at one position are summed first: autocorrelations and
// baselines without coordinates all lie at the origin, where one after another they took 2 us each of their warp, on
// the same 81 cells (2.1 M samples of 512 stations and their autocorrelations, 2 / 8 terms, 1024^2 image: call 812 /
// 1250 -> 439 / 731 us). Run when the chunk's sums are out of the registers; in the segment loop it takes as many.
template <int W, int KC>
__device__ __forceinline__ int rare_records(const SampleRec* __restrict__ rec, const float* __restrict__ rec_s,
                                            const unsigned int* __restrict__ offsets, unsigned int b0, unsigned int b1,
                                            int key, int key_lo, int key_hi, int G, const FastDiv& by_slab,
                                            const FastDiv& by_row, int K, float beta, float2* __restrict__ planes,
                                            int term0) {
    constexpr int HW = W / 2;
    const int lane = threadIdx.x & 31;
    const unsigned int mine = min(b0 + lane, b1 - 1);
    const SampleRec own = rec[mine];
    const float own_s = rec_s ? rec_s[mine] : 0.0f;
    const bool valid = b0 + lane < b1;
    const unsigned int own_bits = valid ? value_bits(own) : 0u;
    const bool plain = valid && !odd_footprint<W>(own) && own_bits < kNotFinite;
    const unsigned int largest = __reduce_max_sync(0xffffffffu, plain ? own_bits : 0u);
    unsigned int rm = __ballot_sync(0xffffffffu, valid && !(plain && (own_bits == 0u || own_bits + kScaleSpan >= largest)));
    const long long GG = (long long)G * G;
    while (rm) {
        const int js = __ffs(rm) - 1;
        const unsigned int p = b0 + js;
        unsigned int ends;  // the window of 32 keys from `key`
        while (!(ends = __ballot_sync(0xffffffffu, offsets[min(key + 1 + lane, key_hi)] > p))) {
            key += 32;
            ends = __ballot_sync(0xffffffffu, offsets[min(key + 32 * (lane + 1) * (lane + 1), key_hi)] > p);
            const int f = __clz(__brev(ends));
            key += 32 * f * f;
        }
        key += __ffs(ends) - 1;
        const int n = key - key_lo, slab = div_by(n, by_slab), rem = n - slab * (int)by_slab.d;
        const int t1 = div_by(rem, by_row), t2 = rem - t1 * (int)by_row.d;
        float2* const plane = planes + ((long long)slab * K + term0) * GG;
        const int xq = __shfl_sync(0xffffffffu, own.xq, js), yq = __shfl_sync(0xffffffffu, own.yq, js);
        const float s = __shfl_sync(0xffffffffu, own_s, js);
        const bool same = lane == js || ((rm >> lane & 1u) && own.xq == xq && own.yq == yq && own_s == s &&
                                         b0 + lane < offsets[key + 1]);
        rm &= ~__ballot_sync(0xffffffffu, same);
        float vre = same ? own.vre : 0.0f, vim = same ? own.vim : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            vre += __shfl_xor_sync(0xffffffffu, vre, o);
            vim += __shfl_xor_sync(0xffffffffu, vim, o);
        }
        const int rcx = xq >> 24, rcy = yq >> 24, rfx = xq & 0xFFFFFF, rfy = yq & 0xFFFFFF;
        const int lo_r = rfx ? rcx - (HW - 1) : rcx - HW, nr = rfx ? W : W + 1;
        const int lo_c = rfy ? rcy - (HW - 1) : rcy - HW, nc = rfy ? W : W + 1;
        const float px = (float)rfx * (1.0f / 16777216.0f), py = (float)rfy * (1.0f / 16777216.0f);
        for (int c = lane; c < nr * nc; c += 32) {
            const int i = c / nc, jj = c - i * nc;
            const int row = t1 * kMmaTile + lo_r + i, col = t2 * kMmaTile + lo_c + jj;
            if (row < 0 || col < 0 || row >= G || col >= G) continue;
            const float x = ((float)(lo_r + i - rcx) - px) / (float)HW;
            const float y = ((float)(lo_c + jj - rcy) - py) / (float)HW;
            const float kv = es_exact(beta, x) * es_exact(beta, y) * (((row + col) & 1) ? -1.0f : 1.0f);
            float2* d = plane + (long long)row * G + col;
            float tm2 = 1.0f, tm1 = s;
            for (int t = 0; t < term0; ++t) {
                const float tt = 2.0f * s * tm1 - tm2;
                tm2 = tm1;
                tm1 = tt;
            }
            for (int t = 0; t < KC; ++t) {
                red_add_v2(d + t * GG, kv * tm2 * vre, kv * tm2 * vim);
                const float tt = 2.0f * s * tm1 - tm2;
                tm2 = tm1;
                tm1 = tt;
            }
        }
    }
    return key;
}

template <int W, int KC>
__global__ void __launch_bounds__(32 * kWarps, min_ctas<KC>()) k_grid_mma(
    const SampleRec* __restrict__ rec, const float* __restrict__ rec_s, const unsigned int* __restrict__ offsets,
    const unsigned int* __restrict__ chunk_key, int chunk, unsigned int* __restrict__ work, int key_lo, int key_hi,
    GridGeom g, FastDiv by_slab, FastDiv by_row, int K, MmaPoly poly,
    float2* __restrict__ planes, int term_lo, int groups, DenseSlots dense, unsigned long long* __restrict__ stamps) {
    if (stamps && term_lo == 0 && first_thread()) stamps[STAMP_GRID] = stamp_now();
    constexpr int HW = W / 2;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    WarpStage<KC>& st = reinterpret_cast<WarpStage<KC>*>(smem)[warp];
    const int gr = lane >> 2, tq = lane & 3;  // fragment row (or column) group and quad lane
    const __half2 row_res = __half2half2(__int2half_rn(gr));
    const __half2 res0 = __half2half2(__int2half_rn(gr & 6)), res1 = __half2half2(__int2half_rn((gr & 6) + 1));
    // checkerboard of this lane's cells (row gr, columns 2 tq + odd; tile origins are even)
    const unsigned int neg = (gr & 1) ? 0x80000000u : 0u;
    const int G = (int)g.G;
    const unsigned int rec_lo = offsets[key_lo], rec_hi = offsets[key_hi];
    if (rec_lo >= rec_hi) return;
    const unsigned int ch_lo = rec_lo / chunk, n_ch = (rec_hi + chunk - 1) / chunk - ch_lo;
    const unsigned int n_work = n_ch * (unsigned int)groups;

    // the chunk of work item i: the chunks are taken from both ends inwards, since the grid's outer
    // tiles hold few records each and take the longest per chunk
    auto chunk_of = [&](unsigned int i) {
        const unsigned int ci = i / (unsigned int)groups;
        return ch_lo + ((ci & 1) ? n_ch - 1 - (ci >> 1) : (ci >> 1));
    };
    unsigned int item = 0, next = 0;
    if (lane == 0) {
        st.rare = 0u;
        item = atomicAdd(work, 1u);
    }
    item = __shfl_sync(0xffffffffu, item, 0);
    if (item >= n_work) return;
    unsigned int ch = chunk_of(item);
    // window of record ends of 32 keys, lane l: key kb + l; the chunk's first records
    int kb = max(key_lo, (int)chunk_key[ch]);
    unsigned int kw = offsets[min(kb + 1 + lane, key_hi)];
    SampleRec r = {0, 0, 0.0f, 0.0f};
    float sv = 0.0f;
    {
        const unsigned int i = max(rec_lo, ch * (unsigned int)chunk) + lane;
        if (i < min(rec_hi, (ch + 1) * (unsigned int)chunk)) {
            r = rec[i];
            if (rec_s) sv = rec_s[i];
        }
    }
    for (;;) {
        if (lane == 0) next = atomicAdd(work, 1u);  // its latency hides behind this chunk
        float acc[KC][4][4];
#pragma unroll
        for (int t = 0; t < KC; ++t)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[t][j][q] = 0.0f;
        const int term0 = term_lo + (int)(item % (unsigned int)groups) * KC;
        const bool need_s = !(KC == 1 && term0 == 0);
        const unsigned int c_beg = max(rec_lo, ch * (unsigned int)chunk);
        const unsigned int c_end = min(rec_hi, (ch + 1) * (unsigned int)chunk);
        int key = -1;                        // tile accumulated in the registers
        unsigned int kbeg = 0, kend = 0;     // its records in this chunk start and (in all) end here
        unsigned int nch = 0;                // the next chunk and its first key
        int nkb = 0;
        // a group of chunks inside one tile: its records' sum is formed in a slot (see DenseSlots)
        const unsigned int grp = ch >> dense.shift;
        const bool in_slot = ((grp + 1) << dense.shift) <= (rec_hi - 1) / (unsigned int)chunk &&
                             chunk_key[grp << dense.shift] == chunk_key[(grp + 1) << dense.shift];

        int t1 = 0, t2 = 0;                  // the tile's row and column
        float2* plane = planes;              // its slab's plane of term term0
        // adds register half h (the region's half `right`) to the plane and clears it; few records
        // (`count`) leave many cells untouched: those are not reduced
        auto add_half = [&](auto hc, int right, unsigned int count) {
            constexpr int h = decltype(hc)::value;
            const int row = t1 * kMmaTile + gr, col = (t2 + right) * kMmaTile + 2 * tq;
            float2* p0 = plane + (long long)row * G + col;
            const long long GG = (long long)G * G;
            const bool inside = t1 * kMmaTile + 16 <= G && (t2 + right + 1) * kMmaTile <= G && !(G & 1);  // 16-byte rows
            if (inside && count >= 8) {
#pragma unroll
                for (int t = 0; t < KC; ++t)
#pragma unroll
                    for (int hr = 0; hr < 2; ++hr)
                        red_add_v4(p0 + t * GG + 8 * hr * G, acc[t][2 * h][2 * hr], acc[t][2 * h][2 * hr + 1],
                                   acc[t][2 * h + 1][2 * hr], acc[t][2 * h + 1][2 * hr + 1]);
            } else {
#pragma unroll
                for (int t = 0; t < KC; ++t)
#pragma unroll
                    for (int hr = 0; hr < 2; ++hr) {
                        const float re0 = acc[t][2 * h][2 * hr], im0 = acc[t][2 * h][2 * hr + 1];
                        const float re1 = acc[t][2 * h + 1][2 * hr], im1 = acc[t][2 * h + 1][2 * hr + 1];
                        float2* d = p0 + t * GG + 8 * hr * G;
                        const bool on0 = re0 != 0.0f || im0 != 0.0f, on1 = re1 != 0.0f || im1 != 0.0f;
                        if (inside) {
                            if (on0 || on1) red_add_v4(d, re0, im0, re1, im1);
                        } else if (row + 8 * hr < G) {
                            if (on0 && col < G) red_add_v2(d, re0, im0);
                            if (on1 && col + 1 < G) red_add_v2(d + 1, re1, im1);
                        }
                    }
            }
#pragma unroll
            for (int t = 0; t < KC; ++t)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[t][2 * h][q] = acc[t][2 * h + 1][q] = 0.0f;
        };
        // moves on to tile `to` (-1: none): the right neighbour's region shares this one's right half,
        // which stays in its registers
        auto move_to = [&](int to, unsigned int count) {
            const bool next_right = key >= 0 && to == key + 1 && t2 + 1 < g.ntile2;
            if (key >= 0) {
                const int par = t2 & 1;
                if (par == 0 || !next_right) add_half(std::integral_constant<int, 0>(), par, count);
                if (par == 1 || !next_right) add_half(std::integral_constant<int, 1>(), 1 - par, count);
            }
            key = to;
            if (next_right) {
                ++t2;
            } else if (to >= 0) {
                const int n = to - key_lo, slab = div_by(n, by_slab), rem = n - slab * (int)by_slab.d;
                t1 = div_by(rem, by_row);
                t2 = rem - t1 * (int)by_row.d;
                plane = planes + ((long long)slab * K + term0) * ((long long)G * G);
            }
        };

        for (unsigned int b0 = c_beg; b0 < c_end; b0 += 32) {
            const unsigned int b1 = min(b0 + 32u, c_end);
            // ---- stage the batch, lane per record
            const bool valid = b0 + lane < b1;
            const int fxq = r.xq & 0xFFFFFF, fyq = r.yq & 0xFFFFFF;
            const int r0 = (r.xq >> 24) - (HW - 1), c0 = (r.yq >> 24) - (HW - 1);
            unsigned int vbits = valid ? value_bits(r) : 0u;
            bool fast = valid && !odd_footprint<W>(r) && vbits < kNotFinite;
            if (!fast) vbits = 0u;
            const unsigned int vmax = __reduce_max_sync(0xffffffffu, vbits);
            fast = fast && (vbits == 0u || vbits + kScaleSpan >= vmax);
            // |v| 2^se < 2^14
            const int se = max(-110, min(110, 14 - ((int)(vmax >> 23) - 126)));
            const float scale = fast ? __int_as_float((se + 127) << 23) : 0.0f;
            // (1 + 2^-23) 2^-(14 + se): the last bit makes up for the products' truncation towards zero
            const float inv = __uint_as_float(((unsigned int)(127 - 14 - se) << 23) | 1u | neg);
            if (valid && !fast) atomicOr(&st.rare, 1u << ((b0 - c_beg) / 32));
            if (vmax) {
                const int oa = fast ? r0 : 0, ob = fast ? c0 : 0;
                st.oa[lane] = __int2half_rn(oa);
                st.ob[lane] = __int2half_rn(ob);
                {
                    float w[W];
                    taps<W>(poly.ey, poly.oy, fmaf((float)fyq, 1.0f / 8388608.0f, -1.0f), w);
                    const unsigned long long v = fast ? pack2(r.vre * scale, r.vim * scale) : 0ull;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        unsigned int w0 = 0u, w1 = 0u;
                        if (i < W) split2(mul2(pack2(w[i < W ? i : 0], w[i < W ? i : 0]), v), w0, w1);
                        unsigned int* q = &st.b[b_row(ob + i) * kPitch + lane];
                        q[0] = w0;
                        q[kPitch] = w1;
                    }
                }
                {
                    float w[W];
                    taps<W>(poly.ex, poly.ox, fmaf((float)fxq, 1.0f / 8388608.0f, -1.0f), w);
                    float tm2 = 1.0f, tm1 = sv;  // T_0, T_1
                    if (need_s)
                        for (int t = 0; t < term0; ++t) {
                            const float tt = 2.0f * sv * tm1 - tm2;
                            tm2 = tm1;
                            tm1 = tt;
                        }
#pragma unroll
                    for (int t = 0; t < KC; ++t) {
                        // |T_n w| <= 1; T_0 = 1
#pragma unroll
                        for (int i = 0; i < 8; i += 2) {
                            unsigned int w0 = 0u, w1 = 0u;
                            if (i < W) {
                                const unsigned long long ww = pack2(w[i < W ? i : 0], w[i < W ? i + 1 : 0]);
                                split2(KC == 1 && !need_s ? ww : mul2(ww, pack2(tm2, tm2)), w0, w1);
                            }
                            st.a[t][((oa + i) & 7) * kPitch + lane] = w0;
                            st.a[t][((oa + i + 1) & 7) * kPitch + lane] = w1;
                        }
                        const float tt = 2.0f * sv * tm1 - tm2;
                        tm2 = tm1;
                        tm1 = tt;
                    }
                }
            }
            // the next batch's records (of the next chunk after the last batch), in flight during this
            // batch's products; the next chunk's first key likewise
            if (b0 == c_beg) {
                next = __shfl_sync(0xffffffffu, next, 0);
                if (next < n_work) {
                    nch = chunk_of(next);
                    nkb = max(key_lo, (int)chunk_key[nch]);
                }
            }
            {
                unsigned int i = b0 + 32 + lane, e = c_end;
                if (b1 == c_end) {
                    i = next < n_work ? max(rec_lo, nch * (unsigned int)chunk) + lane : rec_hi;
                    e = min(rec_hi, (nch + 1) * (unsigned int)chunk);
                }
                if (i < e) {
                    r = rec[i];
                    if (rec_s) sv = rec_s[i];
                }
            }
            __syncwarp();
            // ---- tile segments of the batch
            for (unsigned int p = b0; p < b1;) {
                if (p >= kend) {
                    // The next record's key. Past the window the keys between are empty tiles, mostly few, but a
                    // compact array's two w-slabs on a 3072^2 grid lie 147,000 apart, 2 ms window by window: from
                    // the second window on (kend marks it, free until the key is known) the warp looks (l + 1)^2
                    // windows ahead per step (8.4 M such samples, 2048^2 image: call 2.97 -> 1.07 ms; the 1024^2
                    // case's gridding 82.6 -> 84 us).
                    const unsigned int count = kend - kbeg;
                    unsigned int m;
                    kend = 0;
                    while (!(m = __ballot_sync(0xffffffffu, kw > p))) {
                        kb += 32;
                        if (kend) {
                            m = __ballot_sync(0xffffffffu, offsets[min(kb + 32 * (lane + 1) * (lane + 1), key_hi)] > p);
                            const int f = __clz(__brev(m));
                            kb += 32 * f * f;
                        }
                        kend = 1;
                        kw = offsets[min(kb + 1 + lane, key_hi)];
                    }
                    move_to(kb + __ffs(m) - 1, count);
                    kbeg = p;
                    kend = __shfl_sync(0xffffffffu, kw, __ffs(m) - 1);
                }
                const unsigned int s1 = min(kend, b1);
                const int lo = (int)(p - b0), hi = (int)(s1 - b0);
                p = s1;
                if (vmax) {
                    const unsigned int odd = (t2 & 1) ? 0xffffffffu : 0u;
                    // windows of 16 records from the segment's first pair, inside the batch
                    const int k0 = min(lo & ~1, 16), k8 = min(lo & ~1, 24);
                    if (hi <= k8 + 8)
                        products8<KC>(st, k8, lo, hi, gr, tq, row_res, res0, res1, odd, inv, acc);
                    else if (hi <= k0 + 16)
                        products<1, KC>(st, k0, 0, lo, hi, gr, tq, row_res, res0, res1, odd, inv, acc);
                    else
                        products<2, KC>(st, k0, 16, lo, hi, gr, tq, row_res, res0, res1, odd, inv, acc);
                }
            }
            __syncwarp();
        }
        if (next < n_work) kw = offsets[min(nkb + 1 + lane, key_hi)];
        bool to_plane = true;
        if (in_slot) {
            const size_t at = (size_t)grp * K + term0;
            float4* const slot = dense.sums + at * kSlotWords + lane;
#pragma unroll
            for (int t = 0; t < KC; ++t)
#pragma unroll
                for (int i = 0; i < 4; ++i)  // register half i / 2, rows gr + 8 (i & 1)
                    red_add_v4(reinterpret_cast<float2*>(slot + (4 * t + i) * 32), acc[t][i & 2][2 * (i & 1)],
                               acc[t][i & 2][2 * (i & 1) + 1], acc[t][(i & 2) + 1][2 * (i & 1)],
                               acc[t][(i & 2) + 1][2 * (i & 1) + 1]);
            __threadfence();
            __syncwarp();
            unsigned int arrived = 0;
            if (lane == 0) arrived = atomicInc(dense.arrived + at, (1u << dense.shift) - 1);  // back to 0 by itself
            arrived = __shfl_sync(0xffffffffu, arrived, 0);
            to_plane = arrived == (1u << dense.shift) - 1;  // the group's last chunk takes the sum to the plane
            if (to_plane) __threadfence();
#pragma unroll
            for (int t = 0; t < KC; ++t)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (to_plane) {
                        v = __ldcg(slot + (4 * t + i) * 32);
                        slot[(4 * t + i) * 32] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    }
                    acc[t][i & 2][2 * (i & 1)] = v.x;
                    acc[t][i & 2][2 * (i & 1) + 1] = v.y;
                    acc[t][(i & 2) + 1][2 * (i & 1)] = v.z;
                    acc[t][(i & 2) + 1][2 * (i & 1) + 1] = v.w;
                }
        }
        if (to_plane) move_to(-1, min(kend, c_end) - kbeg);
        unsigned int rare_batches = st.rare;
        if (rare_batches) {
            int rk = max(key_lo, (int)chunk_key[ch]);
            __syncwarp();
            if (lane == 0) st.rare = 0u;
            __syncwarp();
            for (; rare_batches; rare_batches &= rare_batches - 1) {
                const unsigned int b0 = c_beg + 32 * (__ffs(rare_batches) - 1);
                rk = rare_records<W, KC>(rec, need_s ? rec_s : nullptr, offsets, b0, min(b0 + 32u, c_end), rk, key_lo, key_hi,
                                         G, by_slab, by_row, K, poly.beta, planes, term0);
            }
        }
        if (next >= n_work) break;
        item = next;
        ch = nch;
        kb = nkb;
    }
    if (stamps && threadIdx.x == 0) atomicMax(stamps + STAMP_FFT, stamp_now());
}

template <int W, int KC>
int launch_kc(const SampleRec* d_rec, const float* d_rec_s, const unsigned int* d_offsets,
              const unsigned int* d_chunk_key, int chunk, unsigned int* d_work, int key_lo, int key_hi,
              const GridGeom& g, int K, const MmaPoly& poly, float2* d_planes, int term_lo, int groups,
              const DenseSlots& dense, int sm_count, cudaStream_t st, unsigned long long* d_stamps) {
    auto kern = k_grid_mma<W, KC>;
    const size_t smem = sizeof(WarpStage<KC>) * kWarps;
    SVDI_TRY(ensure_dynamic_smem((const void*)kern, smem, true));
    kern<<<sm_count * min_ctas<KC>(), 32 * kWarps, smem, st>>>(d_rec, d_rec_s, d_offsets, d_chunk_key, chunk, d_work,
                                                               key_lo, key_hi, g, fast_div(g.ntile * g.ntile2),
                                                               fast_div(g.ntile2), K, poly, d_planes, term_lo, groups, dense, d_stamps);
    SVDI_LAUNCHED();
    return SVDI_OK;
}

template <int W>
int launch_w(const SampleRec* d_rec, const float* d_rec_s, const unsigned int* d_offsets,
             const unsigned int* d_chunk_key, int chunk, unsigned int* d_work, int key_lo, int key_hi,
             const GridGeom& g, int K, const MmaPoly& poly, float2* d_planes, const DenseSlots& dense, int sm_count,
             cudaStream_t st, unsigned long long* d_stamps) {
    int t0 = 0;
    if (K >= 4) {
        const int n = K / 4;
        SVDI_TRY((launch_kc<W, 4>(d_rec, d_rec_s, d_offsets, d_chunk_key, chunk, d_work, key_lo, key_hi, g, K,
                                  poly, d_planes, t0, n, dense, sm_count, st, d_stamps)));
        t0 += 4 * n;
    }
    if (K - t0 >= 2) {
        SVDI_TRY((launch_kc<W, 2>(d_rec, d_rec_s, d_offsets, d_chunk_key, chunk, d_work + 1, key_lo, key_hi, g, K,
                                  poly, d_planes, t0, 1, dense, sm_count, st, d_stamps)));
        t0 += 2;
    }
    if (K - t0 >= 1)
        SVDI_TRY((launch_kc<W, 1>(d_rec, d_rec_s, d_offsets, d_chunk_key, chunk, d_work + 2, key_lo, key_hi, g, K,
                                  poly, d_planes, t0, 1, dense, sm_count, st, d_stamps)));
    return SVDI_OK;
}

}  // namespace

// Records per chunk: small inputs need many chunks to fill 148 SMs x 12-20 warps, large ones lose more to
// the extra reductions of tiles split between chunks (6.5 M samples: 64 / 128 / 256 / 512 records 0.52 /
// 0.41 / 0.40 / 0.42 ms; 1.04 M samples: 64 / 128 records 0.107 / 0.14 ms, 32 no faster). Below 64 records for
// each of 148 x 12 warps a chunk's own time counts: 24 k samples, 8 terms, whole call 110 us with 64, 106 with 32
// (130 k samples: 141.6 / 141.7).
int mma_chunk(long long n) { return n >= 2000000 ? 256 : n >= 64 * 148 * 12 ? 64 : 32; }

namespace {
// Chunks per slot, as a power of two: 32 (136 additions per cell instead of 4360 where 0.28 M samples share one
// tile), and more where the slots of all groups and terms would exceed 32 MiB.
unsigned int slot_shift(long long n, int K) {
    unsigned int shift = 5;
    while (((n / mma_chunk(n)) >> shift) * K * kSlotWords * (long long)sizeof(float4) > (32LL << 20)) ++shift;
    return shift;
}
size_t slot_count(long long n, int K) { return (size_t)((n / mma_chunk(n)) >> slot_shift(n, K)) * (size_t)K; }
}  // namespace

size_t mma_slot_bytes(long long n, int K) { return slot_count(n, K) * (kSlotWords * sizeof(float4) + sizeof(unsigned int)); }

int launch_grid_mma(const SampleRec* d_rec, const float* d_rec_s, const unsigned int* d_offsets,
                    const unsigned int* d_chunk_key, long long n, void* d_slots, unsigned int* d_work, bool work_cleared,
                    int n_keys, int key_lo, int key_hi, const GridGeom& g, int K, const EsPoly& poly, float2* d_planes,
                    int sm_count, cudaStream_t st, unsigned long long* d_stamps) {
    if (key_lo < 0 || key_hi > n_keys || key_lo >= key_hi || key_hi - key_lo > (1 << 26) || g.T != kMmaTile ||
        g.T2 != kMmaTile) {
        set_error("matrix gridder: bad key range or tile size");
        return SVDI_ERR_INTERNAL;
    }
    if (!work_cleared) SVDI_CUDA(cudaMemsetAsync(d_work, 0, 3 * sizeof(unsigned int), st));
    const int chunk = mma_chunk(n);
    const DenseSlots dense{static_cast<float4*>(d_slots),
                           reinterpret_cast<unsigned int*>(static_cast<float4*>(d_slots) + slot_count(n, K) * kSlotWords),
                           slot_shift(n, K)};
    MmaPoly p{};
    p.beta = poly.beta;
    for (int i = 0; i < g.W / 2; ++i)
        for (int d = 0; d <= kPolyDeg; ++d) {
            (d & 1 ? p.oy[i][d / 2] : p.ey[i][d / 2]) = poly.c[i][d];
            (d & 1 ? p.ox[i][d / 2] : p.ex[i][d / 2]) = poly.c[i][d] * kWeightScale;
        }
    switch (g.W) {
        case 6: return launch_w<6>(d_rec, d_rec_s, d_offsets, d_chunk_key, chunk, d_work, key_lo, key_hi, g, K, p, d_planes, dense, sm_count, st, d_stamps);
        case 8: return launch_w<8>(d_rec, d_rec_s, d_offsets, d_chunk_key, chunk, d_work, key_lo, key_hi, g, K, p, d_planes, dense, sm_count, st, d_stamps);
        default:
            set_error("matrix gridder: ES support must be 6 or 8");
            return SVDI_ERR_UNSUPPORTED;
    }
}

}  // namespace svdi
