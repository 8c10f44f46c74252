// Second pass of the pruned inverse 2-D FFT: the column transforms of the N columns the
// recombination reads, in shared memory, for grid sizes G = 2^a 3^b 5^c 7^d, 16 <= G <= 12288.
//
// cuFFT transforms a strided column batch of a large plane at a fraction of the bandwidth of its
// contiguous row transforms (6144-row columns: ~1.1 TB/s). Here a CTA takes CB adjacent columns
// whole (G x CB complex values, CB * 8-byte row segments, up to 192 KB of shared memory) and runs a
// mixed-radix decimation-in-frequency FFT over the rows. Pass p with radix R and stride S (the product of
// the later radices) takes the R elements b R S + j + S m (m < R) of a column, forms their inverse DFT
// (e^{+2 pi i m k / R}), multiplies element k by e^{+2 pi i j k / (R S)} and writes it back to
// b R S + j + S k. The block comes in by asynchronous copies, all of them in flight at once (a first pass
// straight from the plane, a radix of loads per thread at a time, was slower: 6144 rows 0.33 -> 0.42 ms per
// plane); the last pass writes the output rows (a table gives the output row of each butterfly's first
// element, the others follow G / R apart) straight to the plane. The transform is the inverse, unnormalised one,
// as cuFFT's CUFFT_INVERSE.
//
// What bounds it: latency of one tile's passes (one or two CTAs per SM, 43 % of the issue slots at 3072 rows),
// so fewer and shorter accesses count. The twiddles (FP64-rounded) lie in one table per pass, pairs of them
// 16 bytes, j running fastest: neighbouring threads read one line. Against entries j k G / (R S) of a single
// table e^{+2 pi i t / G} and a table look-up per output row (columns alone): 2 planes of 1536 rows 24 -> 20 us, of
// 3072 rows 98 -> 88 us, 116 planes of 6144 rows 22 -> 18 ms.
//
// Shared-memory rows are swizzled: block row r sits at row r ^ (f(r >> 3) & mask), f(x) = x ^
// (x >> 2) ^ (x >> 4), mask = 16 / CB - 1 (the rows that share a 128-byte bank line). The last
// passes take rows R or 2 R apart in a warp, which without it fall on the same banks (a 6144-row
// block lost half its shared-memory wavefronts to conflicts).
#include "svdi_internal.cuh"

#include <cmath>
#include <vector>

namespace svdi {

namespace {


__device__ __forceinline__ float2 c_add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 c_sub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 c_mul(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 c_i(float2 a) { return make_float2(-a.y, a.x); }    // i a

// inverse DFTs (e^{+2 pi i m k / R}) in place
__device__ __forceinline__ void dft2(float2& a, float2& b) {
    const float2 t = a;
    a = c_add(t, b);
    b = c_sub(t, b);
}

__device__ __forceinline__ void dft3(float2& a, float2& b, float2& c) {
    constexpr float kS = 0.866025403784438647f;  // sqrt(3) / 2
    const float2 t1 = c_add(b, c), t2 = c_sub(b, c);
    const float2 m = make_float2(fmaf(-0.5f, t1.x, a.x), fmaf(-0.5f, t1.y, a.y));
    const float2 r = make_float2(-kS * t2.y, kS * t2.x);  // i sqrt(3)/2 (b - c)
    a = c_add(a, t1);
    b = c_add(m, r);
    c = c_sub(m, r);
}

__device__ __forceinline__ void dft5(float2& a, float2& b, float2& c, float2& d, float2& e) {
    constexpr float kC1 = 0.309016994374947424f, kC2 = -0.809016994374947424f;  // cos(2 pi / 5), cos(4 pi / 5)
    constexpr float kS1 = 0.951056516295153572f, kS2 = 0.587785252292473129f;   // sines
    const float2 p1 = c_add(b, e), q1 = c_sub(b, e), p2 = c_add(c, d), q2 = c_sub(c, d);
    const float2 x = make_float2(a.x + kC1 * p1.x + kC2 * p2.x, a.y + kC1 * p1.y + kC2 * p2.y);
    const float2 y = make_float2(a.x + kC2 * p1.x + kC1 * p2.x, a.y + kC2 * p1.y + kC1 * p2.y);
    const float2 u = make_float2(-(kS1 * q1.y + kS2 * q2.y), kS1 * q1.x + kS2 * q2.x);  // i (S1 q1 + S2 q2)
    const float2 v = make_float2(-(kS2 * q1.y - kS1 * q2.y), kS2 * q1.x - kS1 * q2.x);  // i (S2 q1 - S1 q2)
    a = c_add(a, c_add(p1, p2));
    b = c_add(x, u);
    e = c_sub(x, u);
    c = c_add(y, v);
    d = c_sub(y, v);
}

__device__ __forceinline__ void dft7(float2 (&v)[16]) {
    constexpr float kC[3] = {0.623489801858733531f, -0.222520933956314404f, -0.900968867902419126f};
    constexpr float kS[3] = {0.781831482468029809f, 0.974927912181823607f, 0.433883739117558120f};
    float2 p[3], q[3];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        p[m] = c_add(v[m + 1], v[6 - m]);
        q[m] = c_sub(v[m + 1], v[6 - m]);
    }
    const float2 a = v[0];
    v[0] = c_add(a, c_add(p[0], c_add(p[1], p[2])));
#pragma unroll
    for (int k = 1; k <= 3; ++k) {
        float2 x = a, u = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int m = 1; m <= 3; ++m) {
            const int t = (k * m) % 7, i = t <= 3 ? t : 7 - t;  // cos and |sin| of 2 pi t / 7
            const float c = kC[i - 1], sn = t <= 3 ? kS[i - 1] : -kS[i - 1];
            x = make_float2(fmaf(c, p[m - 1].x, x.x), fmaf(c, p[m - 1].y, x.y));
            u = make_float2(fmaf(-sn, q[m - 1].y, u.x), fmaf(sn, q[m - 1].x, u.y));
        }
        v[k] = c_add(x, u);
        v[7 - k] = c_sub(x, u);
    }
}

__device__ __forceinline__ void dft4(float2& a, float2& b, float2& c, float2& d) {
    const float2 s0 = c_add(a, c), d0 = c_sub(a, c), s1 = c_add(b, d), d1 = c_sub(b, d);
    a = c_add(s0, s1);
    c = c_sub(s0, s1);
    b = c_add(d0, c_i(d1));
    d = c_sub(d0, c_i(d1));
}

__device__ __forceinline__ void dft8(float2 (&v)[16]) {
    constexpr float kC = 0.707106781186547524f;
    dft4(v[0], v[2], v[4], v[6]);
    dft4(v[1], v[3], v[5], v[7]);
    // odd half times e^{+2 pi i k / 8}, k = 0..3
    const float2 o1 = make_float2(kC * (v[3].x - v[3].y), kC * (v[3].x + v[3].y));
    const float2 o2 = c_i(v[5]);
    const float2 o3 = make_float2(-kC * (v[7].x + v[7].y), kC * (v[7].x - v[7].y));
    const float2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
    v[0] = c_add(e0, o0);
    v[4] = c_sub(e0, o0);
    v[1] = c_add(e1, o1);
    v[5] = c_sub(e1, o1);
    v[2] = c_add(e2, o2);
    v[6] = c_sub(e2, o2);
    v[3] = c_add(e3, o3);
    v[7] = c_sub(e3, o3);
}

__device__ __forceinline__ void dft16(float2 (&v)[16]) {
    // x[b + 4 a]: four radix-4 DFTs over a, twiddles e^{+2 pi i b k1 / 16}, four over b;
    // y[k1 + 4 k2] = sum_b e^{2 pi i b k2 / 4} e^{2 pi i b k1 / 16} Z_b[k1]
    constexpr float kC1 = 0.923879532511286756f, kS1 = 0.382683432365089772f, kC = 0.707106781186547524f;
#pragma unroll
    for (int b = 0; b < 4; ++b) dft4(v[b], v[b + 4], v[b + 8], v[b + 12]);
    // Z_b[k1] sits in v[b + 4 k1]
    v[5] = c_mul(v[5], make_float2(kC1, kS1));     // b 1, k1 1: e^{i pi / 8}
    v[9] = c_mul(v[9], make_float2(kC, kC));       // b 1, k1 2: e^{i pi / 4}
    v[13] = c_mul(v[13], make_float2(kS1, kC1));   // b 1, k1 3: e^{3 i pi / 8}
    v[6] = c_mul(v[6], make_float2(kC, kC));       // b 2, k1 1
    v[10] = c_i(v[10]);                            // b 2, k1 2: i
    v[14] = c_mul(v[14], make_float2(-kC, kC));    // b 2, k1 3: e^{3 i pi / 4}
    v[7] = c_mul(v[7], make_float2(kS1, kC1));     // b 3, k1 1: e^{3 i pi / 8}
    v[11] = c_mul(v[11], make_float2(-kC, kC));    // b 3, k1 2: e^{3 i pi / 4}
    v[15] = c_mul(v[15], make_float2(-kC1, -kS1)); // b 3, k1 3: e^{9 i pi / 8}
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) dft4(v[4 * k1], v[4 * k1 + 1], v[4 * k1 + 2], v[4 * k1 + 3]);
    // y[k1 + 4 k2] now sits in v[4 k1 + k2]: transpose the 4 x 4 index
    float2 t;
    t = v[1]; v[1] = v[4]; v[4] = t;
    t = v[2]; v[2] = v[8]; v[8] = t;
    t = v[3]; v[3] = v[12]; v[12] = t;
    t = v[6]; v[6] = v[9]; v[9] = t;
    t = v[7]; v[7] = v[13]; v[13] = t;
    t = v[11]; v[11] = v[14]; v[14] = t;
}

__device__ __forceinline__ void dft9(float2 (&v)[16]) {
    // x[b + 3 a]: radix-3 DFTs over a, twiddles e^{+2 pi i b k1 / 9}, radix-3 over b: y[k1 + 3 k2]
#pragma unroll
    for (int b = 0; b < 3; ++b) dft3(v[b], v[b + 3], v[b + 6]);
    constexpr float kC1 = 0.766044443118978035f, kS1 = 0.642787609686539326f;  // 2 pi / 9
    constexpr float kC2 = 0.173648177666930349f, kS2 = 0.984807753012208059f;  // 4 pi / 9
    constexpr float kC4 = -0.939692620785908384f, kS4 = 0.342020143325668733f; // 8 pi / 9
    v[4] = c_mul(v[4], make_float2(kC1, kS1));  // b 1, k1 1
    v[7] = c_mul(v[7], make_float2(kC2, kS2));  // b 1, k1 2
    v[5] = c_mul(v[5], make_float2(kC2, kS2));  // b 2, k1 1
    v[8] = c_mul(v[8], make_float2(kC4, kS4));  // b 2, k1 2
#pragma unroll
    for (int k1 = 0; k1 < 3; ++k1) dft3(v[3 * k1], v[3 * k1 + 1], v[3 * k1 + 2]);
    // y[k1 + 3 k2] now sits in v[3 k1 + k2]: transpose the 3 x 3 index
    float2 t;
    t = v[1]; v[1] = v[3]; v[3] = t;
    t = v[2]; v[2] = v[6]; v[6] = t;
    t = v[5]; v[5] = v[7]; v[7] = t;
}

// Prime-factor forms (no twiddles): R = 3 Q, input (Q a + 3 b) mod R -> radix-3 DFTs over a, radix-Q DFTs over b;
// bin (Q Q' k1 + 3 T k2) mod R, Q Q' = 1 mod 3, 3 T = 1 mod Q, ends where input (Q k1 + 3 k2) mod R was.
__device__ __forceinline__ void dft12(float2 (&v)[16]) {
#pragma unroll
    for (int b = 0; b < 4; ++b) dft3(v[3 * b % 12], v[(4 + 3 * b) % 12], v[(8 + 3 * b) % 12]);
#pragma unroll
    for (int a = 0; a < 3; ++a) dft4(v[4 * a], v[(4 * a + 3) % 12], v[(4 * a + 6) % 12], v[(4 * a + 9) % 12]);
    float2 y[12];
#pragma unroll
    for (int i = 0; i < 12; ++i) y[(4 * (i / 4) + 9 * (i % 4)) % 12] = v[(4 * (i / 4) + 3 * (i % 4)) % 12];
#pragma unroll
    for (int i = 0; i < 12; ++i) v[i] = y[i];
}

__device__ __forceinline__ void dft24(float2 (&v)[24]) {
#pragma unroll
    for (int b = 0; b < 8; ++b) dft3(v[3 * b % 24], v[(8 + 3 * b) % 24], v[(16 + 3 * b) % 24]);
    float2 y[24];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        float2 t[16];
#pragma unroll
        for (int b = 0; b < 8; ++b) t[b] = v[(8 * a + 3 * b) % 24];
        dft8(t);
#pragma unroll
        for (int k = 0; k < 8; ++k) y[(16 * a + 9 * k) % 24] = t[k];
    }
#pragma unroll
    for (int i = 0; i < 24; ++i) v[i] = y[i];
}

template <int R>
__device__ __forceinline__ void dft_r(float2 (&v)[16]) {
    if constexpr (R == 2) dft2(v[0], v[1]);
    else if constexpr (R == 3) dft3(v[0], v[1], v[2]);
    else if constexpr (R == 4) dft4(v[0], v[1], v[2], v[3]);
    else if constexpr (R == 5) dft5(v[0], v[1], v[2], v[3], v[4]);
    else if constexpr (R == 7) dft7(v);
    else if constexpr (R == 8) dft8(v);
    else if constexpr (R == 9) dft9(v);
    else if constexpr (R == 12) dft12(v);
    else dft16(v);
}

// asynchronous global -> shared copies of 8 or 16 bytes (the block's rows stay in flight together)
__device__ __forceinline__ void cp_async8(float2* dst, const float2* src) {
    const unsigned int d = (unsigned int)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(float2* dst, const float2* src) {
    const unsigned int d = (unsigned int)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// the shared-memory row of block row r (file comment)
__device__ __forceinline__ int srow(int r, int mask) {
    const int x = r >> 3;
    return r ^ ((x ^ (x >> 2) ^ (x >> 4)) & mask);
}

// The CTA's columns in the plane: `pl` the first of them, ncb of them inside the run; pairs of columns are
// read and written as 16 bytes where both lie in it and are aligned (al16).
struct Columns {
    float2* pl;
    long long G;
    int ncb;
    bool al16;
    // columns past the block's end are zero
    __device__ __forceinline__ void load(float2* dst, long long row, int c) const {
        const float2* p = pl + row * G + c;
        if (al16 && c + 1 < ncb) {
            cp_async16(dst, p);
        } else {
            if (c < ncb) cp_async8(dst, p);
            else dst[0] = make_float2(0.0f, 0.0f);
            if (c + 1 < ncb) cp_async8(dst + 1, p + 1);
            else dst[1] = make_float2(0.0f, 0.0f);
        }
    }
    __device__ __forceinline__ void store(long long row, int c, float2 a, float2 b) const {
        float2* p = pl + row * G + c;
        if (al16 && c + 1 < ncb) {
            *reinterpret_cast<float4*>(p) = make_float4(a.x, a.y, b.x, b.y);
        } else {
            if (c < ncb) p[0] = a;
            if (c + 1 < ncb) p[1] = b;
        }
    }
};

// one pass of radix R over the CTA's G x CB block (see the file comment); LAST: to the plane
template <int R, int NT, bool LAST>
__device__ __forceinline__ void col_pass(float2* __restrict__ sh, const Columns& cols, int G, int lcb,
                                         const ColFftPass& P, const float2* __restrict__ tw,
                                         const int* __restrict__ out_row) {
    // a thread takes one butterfly of two adjacent columns: 16-byte accesses and the twiddles loaded once
    // for both
    const int S = P.stride, CP = 1 << (lcb - 1);
    const int nbf = (G / R) << (lcb - 1);
    const int mask = (16 >> lcb) - 1;  // lcb <= 4
    for (int t = threadIdx.x; t < nbf; t += NT) {
        const int c = (t & (CP - 1)) * 2, q = t >> (lcb - 1);
        const int b = (int)(((unsigned int)q * P.div_mul) >> P.div_shift), j = q - b * S;
        const int base = b * R * S + j;
        float2 v[16], u[16];
#pragma unroll
        for (int m = 0; m < R; ++m) {
            const float4 w = *reinterpret_cast<const float4*>(sh + (srow(base + S * m, mask) << lcb) + c);
            v[m] = make_float2(w.x, w.y);
            u[m] = make_float2(w.z, w.w);
        }
        dft_r<R>(v);
        dft_r<R>(u);
        if (!LAST) {  // the last pass has S = 1
#pragma unroll
            for (int k = 1; k < R; k += 2) {
                const float4 w = __ldg(reinterpret_cast<const float4*>(tw) + P.tw_at + (k / 2) * S + j);
                v[k] = c_mul(v[k], make_float2(w.x, w.y));
                u[k] = c_mul(u[k], make_float2(w.x, w.y));
                if (k + 1 < R) {
                    v[k + 1] = c_mul(v[k + 1], make_float2(w.z, w.w));
                    u[k + 1] = c_mul(u[k + 1], make_float2(w.z, w.w));
                }
            }
        }
        const int row0 = LAST ? __ldg(&out_row[base]) : 0;
#pragma unroll
        for (int m = 0; m < R; ++m) {
            if (LAST)
                cols.store(row0 + m * (G / R), c, v[m], u[m]);  // the last digit of the output row
            else
                *reinterpret_cast<float4*>(sh + (srow(base + S * m, mask) << lcb) + c) =
                    make_float4(v[m].x, v[m].y, u[m].x, u[m].y);
        }
    }
}

// a first pass of radix 24, a thread one column: two would not fit the registers
template <int NT>
__device__ __forceinline__ void pass24(float2* __restrict__ sh, int G, int lcb, const ColFftPass& P,
                                       const float2* __restrict__ tw) {
    const int S = P.stride, mask = (16 >> lcb) - 1;
    for (int t = threadIdx.x; t < S << lcb; t += NT) {
        const int c = t & ((1 << lcb) - 1), j = t >> lcb;
        float2 v[24];
#pragma unroll
        for (int m = 0; m < 24; ++m) v[m] = sh[(srow(j + S * m, mask) << lcb) + c];
        dft24(v);
#pragma unroll
        for (int k = 1; k < 24; k += 2) {
            const float4 w = __ldg(reinterpret_cast<const float4*>(tw) + P.tw_at + (k / 2) * S + j);
            v[k] = c_mul(v[k], make_float2(w.x, w.y));
            if (k + 1 < 24) v[k + 1] = c_mul(v[k + 1], make_float2(w.z, w.w));
        }
#pragma unroll
        for (int m = 0; m < 24; ++m) sh[(srow(j + S * m, mask) << lcb) + c] = v[m];
    }
}

template <int NT, bool LAST>
__device__ __forceinline__ void any_pass(float2* __restrict__ sh, const Columns& cols, int G, int lcb,
                                         const ColFftPass& P, const float2* __restrict__ tw,
                                         const int* __restrict__ out_row) {
    switch (P.radix) {
        case 2: col_pass<2, NT, LAST>(sh, cols, G, lcb, P, tw, out_row); break;
        case 3: col_pass<3, NT, LAST>(sh, cols, G, lcb, P, tw, out_row); break;
        case 4: col_pass<4, NT, LAST>(sh, cols, G, lcb, P, tw, out_row); break;
        case 5: col_pass<5, NT, LAST>(sh, cols, G, lcb, P, tw, out_row); break;
        case 7: col_pass<7, NT, LAST>(sh, cols, G, lcb, P, tw, out_row); break;
        case 8: col_pass<8, NT, LAST>(sh, cols, G, lcb, P, tw, out_row); break;
        case 9: col_pass<9, NT, LAST>(sh, cols, G, lcb, P, tw, out_row); break;
        case 12: col_pass<12, NT, LAST>(sh, cols, G, lcb, P, tw, out_row); break;
        case 24:
            if constexpr (!LAST) pass24<NT>(sh, G, lcb, P, tw);
            break;
        default: col_pass<16, NT, LAST>(sh, cols, G, lcb, P, tw, out_row); break;
    }
}

// NT threads; NT = 256: two CTAs per SM and more (blocks of up to 96 KB), NT = 512: one (up to 192 KB)
template <int NT>
__global__ void __launch_bounds__(NT, 512 / NT) k_fft_cols(float2* __restrict__ planes, int G, long long c0,
                                                             int ncols, ColFftPlan P,
                                                             const float2* __restrict__ tw,
                                                             const int* __restrict__ out_row) {
    extern __shared__ __align__(16) float2 sh[];
    const int lcb = P.lcb, CB = 1 << lcb;
    const int cb0 = blockIdx.x * CB;
    Columns cols;
    cols.pl = planes + (long long)blockIdx.y * G * G + c0 + cb0;
    cols.G = G;
    cols.ncb = min(CB, ncols - cb0);
    cols.al16 = ((c0 + cb0) & 1) == 0;  // G even keeps every row aligned alike
    for (int i = threadIdx.x; i < (G << (lcb - 1)); i += NT) {
        const int r = i >> (lcb - 1), c = (i & ((CB >> 1) - 1)) * 2;
        cols.load(sh + (srow(r, (16 >> lcb) - 1) << lcb) + c, r, c);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    for (int p = 0; p + 1 < P.npass; ++p) {
        any_pass<NT, false>(sh, cols, G, lcb, P.pass[p], tw, out_row);
        __syncthreads();
    }
    any_pass<NT, true>(sh, cols, G, lcb, P.pass[P.npass - 1], tw, out_row);
}

}  // namespace

// Radices of G: the largest power of two first, then the odd ones, then the remaining powers of two; empty
// when G has a prime factor above 7 or fewer than two radices.
static std::vector<int> col_radices(long long G) {
    int k2 = 0, k3 = 0;
    std::vector<int> odd, two;
    long long g = G;
    while (g % 2 == 0) g /= 2, ++k2;
    while (g % 3 == 0) g /= 3, ++k3;
    while (g % 5 == 0) g /= 5, odd.push_back(5);
    while (g % 7 == 0) g /= 7, odd.push_back(7);
    if (g != 1 || k2 == 0) return {};
    for (; k3 >= 2; k3 -= 2) odd.push_back(9);
    // a lone 3 joins a 4 or an 8 where that saves a pass (24 first: see pass24). Whole FFT, us: 1536 rows = 8 3 8 8
    // -> 16 12 8, 2 planes 38 -> 36; 3072 = 16 3 8 8 -> 16 12 16, 8 planes 542 -> 523; 6144 = 16 3 16 8 -> 24 16 16,
    // 2 planes 626 -> 605; 1500 = 4 5 5 5 3 -> 5 5 5 12, 4 planes 79 -> 75
    int first = 0;
    if (k3 && (k2 % 4 == 1 || k2 % 4 == 2) && k2 >= 2) odd.push_back(12), k2 -= 2;
    else if (k3 && k2 % 4 == 3 && k2 > 3) first = 24, k2 -= 3;
    else if (k3) odd.push_back(3);
    // 16s with a tail of 8s and 4s (no radix-2 pass beside a larger one: 2^5 = 8 4, 2^9 = 8 8 8)
    switch (k2 % 4) {
        case 1:
            if (k2 == 1) two = {2};
            else if (k2 == 5) two = {8, 4}, k2 = 0;
            else two = {8, 8, 8}, k2 -= 9;
            break;
        case 2:
            if (k2 == 2) two = {4};
            else two = {8, 8}, k2 -= 6;
            break;
        case 3: two = {8}; k2 -= 3; break;
    }
    if (two.empty() || two[0] > 4 || k2 > 2)
        for (; k2 >= 4; k2 -= 4) two.insert(two.begin(), 16);
    std::vector<int> rad;
    if (first) rad.push_back(first);
    if (!two.empty()) rad.push_back(two[0]);
    rad.insert(rad.end(), odd.begin(), odd.end());
    if (!two.empty()) rad.insert(rad.end(), two.begin() + 1, two.end());
    if (rad.size() < 2 || rad.size() > kColFftPasses) return {};
    return rad;
}

// log2 of the columns per CTA: the largest power of two up to 16 with G * CB * 8 bytes <= 96 KB where that gives
// blocks above 64 KB or 8 columns (two CTAs per SM overlap their copies and passes), else <= 192 KB (one CTA per
// SM); at least 1: the passes take pairs of columns. Whole FFT, us, at 96 / 192 KB: 1536 rows, 8 planes 126 /
// 138; 2304, 8 planes 290 / 300; 3072, 2 planes 146 / 152; but 1792, 2 planes 50 / 48; 2048, 2 planes 56 / 54;
// 3584, 2 planes 220 / 214; 6144, 2 planes 648 / 626.
static int col_fft_lcb(long long G, long long columns) {
    const long long cap = G <= 1536 || (G > 2048 && G <= 3072) ? 96 * 1024 : 192 * 1024;
    int lcb = 1;
    while (lcb < 4 && G * (2LL << lcb) * 8 <= cap) ++lcb;
    // few columns: narrower blocks until there is a CTA per SM (8 planes of 288 / 384 rows: 19.5 / 25.6 us with
    // two CTAs per SM asked for, 17.4 / 21.5 us with one)
    while (lcb > 2 && (columns >> lcb) < 148) --lcb;
    return lcb;
}

// Where it is used: every grid size it supports measured at or below cuFFT's strided column plan (whole FFT,
// rows by cuFFT in both; us): 288 rows, 8 planes 58 -> 17; 720, 8 planes 91 -> 42; 1500, 4 planes 126 -> 75; 1536,
// 2 planes 52 -> 36; 2304, 8 planes 407 -> 290; 3072, 2 planes 185 -> 146; 3584, 2 planes 341 -> 214; 4500, 2
// planes 1037 -> 370; 6144, 2 planes 1025 -> 605.
bool col_fft_supported(long long G) {
    if (G < 16 || G > 12288) return false;
    return !col_radices(G).empty();
}

int make_col_fft(long long G, long long columns, ColFftPlan& P, float2** d_tw, int** d_perm) {
    const std::vector<int> rad = col_radices(G);
    if (!col_fft_supported(G)) {
        set_error("column FFT: unsupported grid size");
        return SVDI_ERR_UNSUPPORTED;
    }
    P = ColFftPlan{};
    P.npass = (int)rad.size();
    std::vector<float2> tw;
    long long before = 1;  // product of the earlier radices = G / (R S)
    for (int p = 0; p < P.npass; ++p) {
        long long S = 1;
        for (int q = p + 1; q < P.npass; ++q) S *= rad[q];
        P.pass[p].radix = rad[p];
        P.pass[p].stride = (int)S;
        P.pass[p].tw_at = (int)(tw.size() / 2);
        if (p + 1 < P.npass)  // pairs k, k + 1 of twiddles e^{2 pi i j k / (R S)}, runs over j
            for (int k = 1; k < rad[p]; k += 2)
                for (long long j = 0; j < S; ++j)
                    for (int i = k; i < k + 2; ++i) {
                        const long long t = j * i * before % G;
                        const double a = 2.0 * 3.14159265358979323846 * (double)t / (double)G;
                        tw.push_back(make_float2((float)std::cos(a), (float)std::sin(a)));
                    }
        // mul = ceil(2^shift / S), shift = 14 + ceil(log2 S): the quotient is off by less than q / 2^14 / S < 1 / S
        unsigned int shift = 14;
        while ((1LL << (shift - 14)) < S) ++shift;
        P.pass[p].div_mul = (unsigned int)(((1LL << shift) + S - 1) / S);
        P.pass[p].div_shift = shift;
        before *= rad[p];
    }
    P.lcb = col_fft_lcb(G, columns);
    // the digit-reversed position of each output row
    std::vector<int> perm((size_t)G);
    for (long long nrow = 0; nrow < G; ++nrow) {
        long long t = nrow, pos = 0;
        for (int p = 0; p < P.npass; ++p) {
            const long long k = t % rad[p];
            t /= rad[p];
            pos += k * P.pass[p].stride;
        }
        perm[(size_t)pos] = (int)nrow;  // block row pos holds output row nrow
    }
    SVDI_CUDA(cudaMalloc(d_tw, tw.size() * sizeof(float2)));
    SVDI_CUDA(cudaMalloc(d_perm, (size_t)G * sizeof(int)));
    SVDI_CUDA(cudaMemcpy(*d_tw, tw.data(), tw.size() * sizeof(float2), cudaMemcpyHostToDevice));
    SVDI_CUDA(cudaMemcpy(*d_perm, perm.data(), (size_t)G * sizeof(int), cudaMemcpyHostToDevice));
    return SVDI_OK;
}

int launch_col_fft(float2* d_planes, int nplanes, long long G, long long c0, long long ncols, const ColFftPlan& P,
                   const float2* d_tw, const int* d_perm, cudaStream_t st) {
    const size_t bank_rows = (size_t)16 >> P.lcb;  // the swizzle permutes rows within runs of this length
    const size_t smem = ((size_t)G + bank_rows - 1) / bank_rows * bank_rows * ((size_t)1 << P.lcb) * sizeof(float2);
    const dim3 grid((unsigned)((ncols + (1LL << P.lcb) - 1) >> P.lcb), (unsigned)nplanes);
    if (smem <= 96 * 1024) {
        SVDI_TRY(ensure_dynamic_smem((const void*)k_fft_cols<256>, smem, true));
        k_fft_cols<256><<<grid, 256, smem, st>>>(d_planes, (int)G, c0, (int)ncols, P, d_tw, d_perm);
    } else {
        SVDI_TRY(ensure_dynamic_smem((const void*)k_fft_cols<512>, smem, true));
        k_fft_cols<512><<<grid, 512, smem, st>>>(d_planes, (int)G, c0, (int)ncols, P, d_tw, d_perm);
    }
    SVDI_LAUNCHED();
    return SVDI_OK;
}

}  // namespace svdi
