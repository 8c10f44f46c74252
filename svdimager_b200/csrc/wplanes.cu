// Imaging through w planes: the error-target rule's path for large w ranges.
//
// The reference (and this library's other rules) expands e^{2 pi i r3 t3} in Chebyshev polynomials per
// w-slab: every sample enters all K terms of its slab, and nslab K planes are transformed. Where only an
// error target is asked for, the third axis can be interpolated like the other two: with planes w_p = lo +
// (p - (W/2 - 1)) dw and an ES kernel psi of W planes,
//   e^{2 pi i r3 t3} = (1 / psi^(dw t3)) sum_p psi(v - p) e^{2 pi i w_p t3},  v = (r3 - lo) / dw + W/2 - 1,
// so a sample enters W planes only, and dw = 1 / (2 sigma max|t3|) gives sigma alpha / pi + W planes. The
// image is a real part, and Re(V e^{i phi}) = Re(V* e^{-i phi}): samples with r3 < 0 enter as their mirror
// image (-r, V*), which halves the w range. Wide field of 4 slabs x 59 terms (236 moments): 116 planes.
//
// Gridding: planes hold 0.1 samples per 8 x 8 tile and plane there, so a cell is touched about once, and
// reductions into cleared planes cost a read, a write and the clearing of every cell from DRAM. Instead the
// samples are binned by 8 x 8 tiles of their (mirrored) footprint origins and every cell is owned: a CTA takes
// 16 x 16 cells of all planes and stages the samples of the nine tiles whose footprints reach them; its warps
// take four planes at a time in registers and write each cell once (zeros included: no clearing). Blocks of
// many samples are split into parts, which add by reductions to cells cleared first. Samples on exactly
// integer positions or at the grid edge are added by reductions afterwards. Figures at launch_grid_w.
#include "binning_rules.cuh"
#include "svdi_internal.cuh"

namespace svdi {

namespace {

using namespace binrules;

constexpr int kWarps = 4;
constexpr int kMaxW = 12;          // planes per sample
constexpr int kCells = 16;         // side of a CTA's block of cells
constexpr int kWarpPlanes = 4;     // planes of a warp
constexpr int kPart = 32 * kWarps; // records of one CTA (a thread stages one): a block with more is split

__device__ __forceinline__ void red_add_v4(float2* addr, float a, float b, float c, float d) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(a), "f"(b), "f"(c), "f"(d)
                 : "memory");
}

__device__ __forceinline__ void red_add_v2(float2* addr, float a, float b) {
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(addr), "f"(a), "f"(b) : "memory");
}

__device__ __forceinline__ float es_exact(float beta, float x) {
    if (fabsf(x) > 1.0f) return 0.0f;
    return expf(-beta * x * x / (1.0f + sqrtf((1.0f - x) * (1.0f + x))));
}

// Taps 0 .. W - 1 at fraction f (u = 2 f - 1): mirrored pieces share the even and odd parts.
template <int W>
__device__ __forceinline__ void taps(const EsPoly& p, float u, float* w) {
    const float v = u * u;
#pragma unroll
    for (int i = 0; i < W / 2; ++i) {
        const float* c = p.c[i];
        const float ev = fmaf(fmaf(fmaf(fmaf(c[8], v, c[6]), v, c[4]), v, c[2]), v, c[0]);
        const float od = fmaf(fmaf(fmaf(c[7], v, c[5]), v, c[3]), v, c[1]);
        w[i] = fmaf(u, od, ev);
        w[W - 1 - i] = fmaf(-u, od, ev);
    }
}
static_assert(kPolyDeg == 8, "taps() is written for degree 8");

// A sample of a separable source as the planes take it: mirrored to r3 >= 0, position split into cell and
// 24-bit fraction per axis, first plane and fraction on the w axis.
struct WSample {
    int c1, c2, f1, f2;  // cells relative to the grid centre, fractions
    int p0;
    float f3;
    bool kept, mirrored, rare;
};

__device__ __forceinline__ WSample w_sample(const SampleSource& src, unsigned int row, int c, const GridGeom& g,
                                            const WPlanes& wp) {
    WSample o;
    const double* q = src.q + (long long)row * 3;
    const double sc = src.s[c];
    const double r1 = __dmul_rn(sc, q[0]), r2 = __dmul_rn(sc, q[1]), r3 = __dmul_rn(sc, q[2]);
    double p1 = grid_pos(r1, g), p2 = grid_pos(r2, g);
    int tile, qrel;
    // the binned gridders' inclusion rule, on the sample as it is
    o.kept = quantise_axis(p1, g, g.T, tile, qrel) && quantise_axis(p2, g, g.T2, tile, qrel);
    o.mirrored = r3 < 0.0;
    o.rare = false;
    o.c1 = o.c2 = o.f1 = o.f2 = o.p0 = 0;
    o.f3 = 0.0f;
    if (!o.kept) return o;
    if (o.mirrored) {
        p1 = -p1;
        p2 = -p2;
    }
    const long long q1 = floor_to_int(p1 * 16777216.0), q2 = floor_to_int(p2 * 16777216.0);
    o.c1 = (int)(q1 >> 24);
    o.c2 = (int)(q2 >> 24);
    o.f1 = (int)(q1 & 0xFFFFFF);
    o.f2 = (int)(q2 & 0xFFFFFF);
    const double w = __dmul_rn(fabs(r3) - wp.lo, wp.inv_dw);  // >= 0 up to rounding
    o.p0 = max(0, min((int)(floor_to_int(w * 16777216.0) >> 24), wp.P - wp.W));
    o.f3 = fminf(1.0f, fmaxf(0.0f, (float)(w - (double)o.p0)));
    const int hw = g.W / 2, G = (int)g.G;
    const int a1 = o.c1 - (hw - 1) - (int)g.gmin, a2 = o.c2 - (hw - 1) - (int)g.gmin;  // plane row, column
    const int low = o.mirrored ? 1 : 0;  // -G / 2 mirrors G / 2, which is not on the grid
    o.rare = o.f1 == 0 || o.f2 == 0 || a1 < low || a2 < low || a1 + g.W > G || a2 + g.W > G;
    return o;
}

// A binned sample (32 bytes): origin of its footprint in the plane, fractions, first plane, value.
struct __align__(16) WRec {
    int a1, a2, f1, f2;
    int p0;
    float f3, vre, vim;
};

constexpr int kThreads = 256;

// The samples by channel runs of a row: sample k of the launch is channel k % C of row k / C, so consecutive
// lanes hold consecutive channels of one baseline and mostly share a tile.
template <bool SCATTER>
__global__ void __launch_bounds__(kThreads) k_bin_w(SampleSource src, GridGeom g, WPlanes wp, int nt, int C,
                                                    unsigned int* __restrict__ counts, WRec* __restrict__ rec) {
    const int lane = threadIdx.x & 31;
    const long long n = src.n, stride = (long long)gridDim.x * kThreads;
    for (long long k0 = blockIdx.x * (long long)kThreads + (threadIdx.x & ~31); k0 < n; k0 += stride) {
        const unsigned int k = (unsigned int)(k0 + lane);
        int key = -1;
        WSample o;
        unsigned int row = 0;
        int c = 0;
        if (k0 + lane < n) {
            row = k / (unsigned int)C;
            c = (int)(k - row * (unsigned int)C);
            o = w_sample(src, row, c, g, wp);
            if (o.kept && !o.rare)
                key = ((o.c1 - (g.W / 2 - 1) - (int)g.gmin) >> 3) * nt + ((o.c2 - (g.W / 2 - 1) - (int)g.gmin) >> 3);
        }
        // runs of equal keys on consecutive lanes: one atomic each
        const int before = __shfl_up_sync(0xffffffffu, key, 1);
        const unsigned int starts = __ballot_sync(0xffffffffu, lane == 0 || key != before);
        const int first = 31 - __clz(starts & (0xffffffffu >> (31 - lane)));
        const unsigned int after = starts & ~(0xffffffffu >> (31 - lane));
        const int length = (after ? __ffs(after) - 1 : 32) - first;
        unsigned int at = 0;
        if (key >= 0 && lane == first) {
            if (SCATTER) at = atomicAdd(&counts[key], (unsigned int)length);
            else atomicAdd(&counts[key], (unsigned int)length);
        }
        if (SCATTER) {
            at = __shfl_sync(0xffffffffu, at, first);
            if (key >= 0) {
                const long long idx = (long long)row + (long long)c * src.R;
                const float vim = __fmul_rn(src.vi[idx], src.inv_det);
                WRec r;
                r.a1 = o.c1 - (g.W / 2 - 1) - (int)g.gmin;
                r.a2 = o.c2 - (g.W / 2 - 1) - (int)g.gmin;
                r.f1 = o.f1;
                r.f2 = o.f2;
                r.p0 = o.p0;
                r.f3 = o.f3;
                r.vre = __fmul_rn(src.vr[idx], src.inv_det);
                r.vim = o.mirrored ? -vim : vim;
                rec[at + (unsigned int)(lane - first)] = r;
            }
        }
    }
}

// A staged sample of a CTA: its taps on the block's 16 rows and 16 columns (checkerboard sign in the rows; zero
// where the footprint does not reach) and on its planes, three zeros either side.
struct __align__(16) Staged {
    float wx[kCells], wy[kCells];
    float wz[kMaxW + 6];
    float2 v;
};

// packed pairs of floats
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

// The records whose footprints reach block (by, bx): three runs, of the tile rows 2 by - 1 .. 2 by + 1.
struct Runs {
    unsigned int beg[3], len[3];
    __device__ __forceinline__ unsigned int total() const { return len[0] + len[1] + len[2]; }
    __device__ __forceinline__ unsigned int record(unsigned int i) const {
        if (i < len[0]) return beg[0] + i;
        i -= len[0];
        return i < len[1] ? beg[1] + i : beg[2] + (i - len[1]);
    }
};
__device__ __forceinline__ Runs block_runs(const unsigned int* __restrict__ offsets, int nt, int by, int bx) {
    Runs r;
    const int tc0 = max(0, 2 * bx - 1), tc1 = min(nt - 1, 2 * bx + 1);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int tr = 2 * by - 1 + k;
        const bool on = tr >= 0 && tr < nt;
        r.beg[k] = on ? offsets[tr * nt + tc0] : 0u;
        r.len[k] = on ? offsets[tr * nt + tc1 + 1] - r.beg[k] : 0u;
    }
    return r;
}

// A block with more than kPart records is shared by several CTAs, which add to its cells instead of writing
// them (a compact array's core holds most of its samples: one CTA per block took 1.8 ms where the whole
// snapshot takes 0.2). list[0] counts the further parts, entries (block, part) follow; their blocks' cells are
// cleared here.
__global__ void __launch_bounds__(256) k_split_w(const unsigned int* __restrict__ offsets, int G, int nt, int nplanes,
                                                 unsigned int* __restrict__ list, float2* __restrict__ planes) {
    __shared__ unsigned int parts, at;
    const int nb = (G + kCells - 1) / kCells;
    for (int b = blockIdx.x; b < nb * nb; b += gridDim.x) {
        const int by = b / nb, bx = b - by * nb;
        if (threadIdx.x == 0) {
            parts = (block_runs(offsets, nt, by, bx).total() + kPart - 1) / kPart;
            if (parts > 1) at = atomicAdd(list, parts - 1);
        }
        __syncthreads();
        if (parts > 1) {
            for (unsigned int k = 1 + threadIdx.x; k < parts; k += 256) {
                list[2 * (at + k)] = (unsigned int)b;
                list[2 * (at + k) + 1] = k;
            }
            const int rows = min(kCells, G - by * kCells), cols = min(kCells, G - bx * kCells);
            float2* base = planes + (long long)by * kCells * G + bx * kCells;
            for (int i = threadIdx.x; i < nplanes * kCells * kCells; i += 256) {
                const int p = i / (kCells * kCells), r = i / kCells % kCells, c = i % kCells;
                if (r < rows && c < cols) base[(long long)p * G * G + (long long)r * G + c] = make_float2(0.0f, 0.0f);
            }
        }
        __syncthreads();
    }
}

// blockIdx.x < number of blocks: part 0 of that block; beyond: the listed further parts in turn.
template <int W, int WZ>
__global__ void __launch_bounds__(32 * kWarps, 20 / kWarps) k_grid_w(const WRec* __restrict__ rec,
                                                           const unsigned int* __restrict__ offsets,
                                                           const unsigned int* __restrict__ list, int G, int nt,
                                                           EsPoly pxy, EsPoly pz, int plane_lo, int plane_hi,
                                                           float2* __restrict__ planes) {
    extern __shared__ __align__(16) unsigned char smem[];
    Staged* st = reinterpret_cast<Staged*>(smem);
    __shared__ int n_st, next_planes, st_p0[kPart];  // staged samples; the next planes to take; first planes
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nb = (G + kCells - 1) / kCells, nblocks = nb * nb;
    // this lane's cells: rows 2 r2, 2 r2 + 1 and columns 4 c4 .. 4 c4 + 3, (re, im) pairs per plane
    const int r2 = lane >> 2, c4 = lane & 3;
    const long long GG = (long long)G * G;
    const bool listed = (int)blockIdx.x >= nblocks;
    const unsigned int n_listed = listed ? list[0] : 0u;
    for (unsigned int e = listed ? blockIdx.x - nblocks : 0u; !listed || e < n_listed; e += gridDim.x - nblocks) {
        const int b = listed ? (int)list[2 * (e + 1)] : (int)blockIdx.x;
        const unsigned int part = listed ? list[2 * (e + 1) + 1] : 0u;
        const int by = b / nb, bx = b - by * nb;
        const int row0 = by * kCells, col0 = bx * kCells;
        const Runs runs = block_runs(offsets, nt, by, bx);
        const unsigned int total = runs.total();
        // ---- stage the samples of the part that reach the block's cells and the launch's planes
        if (threadIdx.x == 0) {
            n_st = 0;
            next_planes = kWarps;
        }
        __syncthreads();
        const unsigned int i = part * kPart + threadIdx.x;
        if (i < total) {
            const WRec r = rec[runs.record(i)];
            const int d1 = r.a1 - row0, d2 = r.a2 - col0;
            if (d1 > -W && d1 < kCells && d2 > -W && d2 < kCells && r.p0 < plane_hi && r.p0 + WZ > plane_lo) {
                const int at = atomicAdd(&n_st, 1);
                Staged& s = st[at];
                st_p0[at] = r.p0;
                float t[W];
                taps<W>(pxy, fmaf((float)r.f1, 1.0f / 8388608.0f, -1.0f), t);
#pragma unroll
                for (int q = 0; q < kCells; ++q) s.wx[q] = 0.0f;
#pragma unroll
                for (int q = 0; q < W; ++q)
                    if ((unsigned int)(d1 + q) < (unsigned int)kCells) s.wx[d1 + q] = (d1 + q) & 1 ? -t[q] : t[q];
                taps<W>(pxy, fmaf((float)r.f2, 1.0f / 8388608.0f, -1.0f), t);
#pragma unroll
                for (int q = 0; q < kCells; ++q) s.wy[q] = 0.0f;
#pragma unroll
                for (int q = 0; q < W; ++q)
                    if ((unsigned int)(d2 + q) < (unsigned int)kCells) s.wy[d2 + q] = (d2 + q) & 1 ? -t[q] : t[q];
                float z[WZ];
                taps<WZ>(pz, fmaf(2.0f, r.f3, -1.0f), z);
#pragma unroll
                for (int q = 0; q < 3; ++q) s.wz[q] = s.wz[3 + WZ + q] = 0.0f;
#pragma unroll
                for (int q = 0; q < WZ; ++q) s.wz[3 + q] = z[q];
                s.v = make_float2(r.vre, r.vim);
            }
        }
        __syncthreads();
        const int n = n_st;
        const bool add = total > (unsigned int)kPart;
        // ---- four planes at a time, taken by the warps as they come free (low planes hold most samples): add the
        // samples that reach them, then the cells. A lane's four columns are 32 bytes, four lanes a 128-byte
        // row piece.
        for (int group = warp;;) {
            const int mine = plane_lo + group * kWarpPlanes;
            if (mine >= plane_hi) break;
            unsigned long long acc[kWarpPlanes][8];
#pragma unroll
            for (int p = 0; p < kWarpPlanes; ++p)
#pragma unroll
                for (int q = 0; q < 8; ++q) acc[p][q] = 0ull;
            for (int j0 = 0; j0 < n; j0 += 32) {
              const int o_lane = mine - (j0 + lane < n ? st_p0[j0 + lane] : -1000000);
              unsigned int todo = __ballot_sync(0xffffffffu, o_lane > -kWarpPlanes && o_lane < WZ);
              while (todo) {
                const int jj = __ffs(todo) - 1;
                todo &= todo - 1;
                const Staged& s = st[j0 + jj];
                const int o = __shfl_sync(0xffffffffu, o_lane, jj);  // the first of the four planes among the sample's
                const float2 wx = *reinterpret_cast<const float2*>(&s.wx[2 * r2]);
                const float4 wy = *reinterpret_cast<const float4*>(&s.wy[4 * c4]);
                const unsigned long long v = *reinterpret_cast<const unsigned long long*>(&s.v);
                const unsigned long long v0 = mul2(v, pack2(wx.x, wx.x)), v1 = mul2(v, pack2(wx.y, wx.y));
                unsigned long long kv[8];
                kv[0] = mul2(v0, pack2(wy.x, wy.x));
                kv[1] = mul2(v0, pack2(wy.y, wy.y));
                kv[2] = mul2(v0, pack2(wy.z, wy.z));
                kv[3] = mul2(v0, pack2(wy.w, wy.w));
                kv[4] = mul2(v1, pack2(wy.x, wy.x));
                kv[5] = mul2(v1, pack2(wy.y, wy.y));
                kv[6] = mul2(v1, pack2(wy.z, wy.z));
                kv[7] = mul2(v1, pack2(wy.w, wy.w));
#pragma unroll
                for (int p = 0; p < kWarpPlanes; ++p) {
                    const float z = s.wz[o + 3 + p];
                    const unsigned long long zz = pack2(z, z);
#pragma unroll
                    for (int q = 0; q < 8; ++q) acc[p][q] = fma2(kv[q], zz, acc[p][q]);
                }
              }
            }
            const int col = col0 + 4 * c4;
#pragma unroll
            for (int p = 0; p < kWarpPlanes; ++p) {
                if (mine + p >= plane_hi) break;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int row = row0 + 2 * r2 + h;
                    if (row >= G) continue;
                    float2* d = planes + (long long)(mine + p - plane_lo) * GG + (long long)row * G + col;
                    const unsigned long long* a = &acc[p][4 * h];
                    if (add) {
#pragma unroll
                        for (int q = 0; q < 4; q += 2) {
                            const float2 x = unpack2(a[q]), y = unpack2(a[q + 1]);
                            if (x.x == 0.0f && x.y == 0.0f && y.x == 0.0f && y.y == 0.0f) continue;
                            if (col + q + 1 < G) red_add_v4(d + q, x.x, x.y, y.x, y.y);  // 16-byte aligned: G, col even
                            else if (col + q < G) red_add_v2(d + q, x.x, x.y);
                        }
                    } else if (col + 3 < G) {
                        *reinterpret_cast<ulonglong2*>(d) = make_ulonglong2(a[0], a[1]);
                        *reinterpret_cast<ulonglong2*>(d + 2) = make_ulonglong2(a[2], a[3]);
                    } else {
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (col + q < G) *reinterpret_cast<unsigned long long*>(d + q) = a[q];
                    }
                }
            }
            if (lane == 0) group = atomicAdd(&next_planes, 1);
            group = __shfl_sync(0xffffffffu, group, 0);
        }
        if (!listed) break;
        __syncthreads();  // the next part's staging overwrites this one's
    }
}

// The samples that the tiles leave out -- exactly integer positions (W + 1 cells) and footprints at the grid
// edge: the cells the reference rule keeps of the sample as it is, mirrored with it (column G / 2 is column
// -G / 2 of the periodic transform) -- and, with `dropped`, the counts of dropped and non-finite samples.
template <int W, int WZ>
__global__ void __launch_bounds__(kThreads) k_rare_w(SampleSource src, GridGeom g, WPlanes wp, EsPoly pz, int C,
                                                     int plane_lo, int plane_hi, float2* __restrict__ planes,
                                                     unsigned long long* __restrict__ dropped) {
    constexpr int HW = W / 2;
    const int lane = threadIdx.x & 31;
    const int G = (int)g.G, gmin = (int)g.gmin, gmax = (int)g.gmax;
    const long long GG = (long long)G * G;
    const long long n = src.n, stride = (long long)gridDim.x * kThreads;
    unsigned int ndrop = 0, nbad = 0;
    for (long long k0 = blockIdx.x * (long long)kThreads + (threadIdx.x & ~31); k0 < n; k0 += stride) {
        WSample o;
        o.kept = o.rare = o.mirrored = false;
        o.c1 = o.c2 = o.f1 = o.f2 = o.p0 = 0;
        o.f3 = 0.0f;
        float vre = 0.0f, vim = 0.0f;
        if (k0 + lane < n) {
            const unsigned int k = (unsigned int)(k0 + lane), row = k / (unsigned int)C;
            const int c = (int)(k - row * (unsigned int)C);
            o = w_sample(src, row, c, g, wp);
            if (!o.kept) ++ndrop;
            if (o.kept && (dropped || o.rare)) {
                const long long idx = (long long)row + (long long)c * src.R;
                vre = __fmul_rn(src.vr[idx], src.inv_det);
                vim = __fmul_rn(src.vi[idx], src.inv_det);
                nbad += (((__float_as_uint(vre) & 0x7f800000u) == 0x7f800000u) |
                         ((__float_as_uint(vim) & 0x7f800000u) == 0x7f800000u));
                if (o.mirrored) vim = -vim;
            }
        }
        unsigned int todo = __ballot_sync(0xffffffffu, o.rare);
        while (todo) {
            const int j = __ffs(todo) - 1;
            todo &= todo - 1;
            const int c1 = __shfl_sync(0xffffffffu, o.c1, j), f1 = __shfl_sync(0xffffffffu, o.f1, j);
            const int c2 = __shfl_sync(0xffffffffu, o.c2, j), f2 = __shfl_sync(0xffffffffu, o.f2, j);
            const int p0 = __shfl_sync(0xffffffffu, o.p0, j), m = __shfl_sync(0xffffffffu, o.mirrored ? -1 : 1, j);
            const float f3 = __shfl_sync(0xffffffffu, o.f3, j);
            const float re = __shfl_sync(0xffffffffu, vre, j), im = __shfl_sync(0xffffffffu, vim, j);
            float z[WZ];
            taps<WZ>(pz, fmaf(2.0f, f3, -1.0f), z);
            const int lo1 = f1 ? c1 - (HW - 1) : c1 - HW, n1 = f1 ? W : W + 1;
            const int lo2 = f2 ? c2 - (HW - 1) : c2 - HW, n2 = f2 ? W : W + 1;
            const float x0 = (float)f1 * (1.0f / 16777216.0f), y0 = (float)f2 * (1.0f / 16777216.0f);
            for (int e = lane; e < n1 * n2; e += 32) {
                int y = lo1 + e / n2, x = lo2 + e % n2;
                const float kv = es_exact(wp.beta_xy, ((float)(y - c1) - x0) / (float)HW) *
                                 es_exact(wp.beta_xy, ((float)(x - c2) - y0) / (float)HW);
                if (m * y < gmin || m * y > gmax || m * x < gmin || m * x > gmax) continue;
                if (y > gmax) y -= G;
                if (x > gmax) x -= G;
                const float sg = ((y - gmin + x - gmin) & 1) ? -kv : kv;
#pragma unroll
                for (int q = 0; q < WZ; ++q) {
                    if (p0 + q < plane_lo || p0 + q >= plane_hi) continue;
                    red_add_v2(planes + (long long)(p0 + q - plane_lo) * GG + (long long)(y - gmin) * G + (x - gmin),
                               sg * z[q] * re, sg * z[q] * im);
                }
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        ndrop += __shfl_xor_sync(0xffffffffu, ndrop, o);
        nbad += __shfl_xor_sync(0xffffffffu, nbad, o);
    }
    if (lane == 0 && dropped) {
        if (ndrop) atomicAdd(dropped, (unsigned long long)ndrop);
        if (nbad && src.nonfinite) atomicAdd(src.nonfinite, (unsigned long long)nbad);
    }
}

int bin_blocks(long long n) {
    return (int)std::max<long long>(1, std::min<long long>((n + kThreads - 1) / kThreads, 8LL * current_sm_count()));
}

template <int W, int WZ>
int launch_planes(const SampleSource& src, const GridGeom& g, const WPlanes& wp, const EsPoly& pxy, const EsPoly& pz,
                  const void* d_rec, const unsigned int* d_offsets, unsigned int* d_list, int plane_lo, int plane_hi,
                  float2* d_planes, unsigned long long* d_dropped, cudaStream_t st) {
    const int G = (int)g.G, nt = w_tiles(g.G), nb = (G + kCells - 1) / kCells, nblocks = nb * nb;
    SVDI_CUDA(cudaMemsetAsync(d_list, 0, sizeof(unsigned int), st));
    k_split_w<<<std::min(nblocks, 8 * current_sm_count()), 256, 0, st>>>(d_offsets, G, nt, plane_hi - plane_lo, d_list,
                                                                        d_planes);
    SVDI_LAUNCHED();
    const size_t smem = sizeof(Staged) * kPart;
    auto kern = k_grid_w<W, WZ>;
    SVDI_TRY(ensure_dynamic_smem((const void*)kern, smem));
    const long long extra = std::min<long long>((long long)w_list_words(src.n) / 2, 4LL * current_sm_count());
    kern<<<(unsigned)(nblocks + extra), 32 * kWarps, smem, st>>>(static_cast<const WRec*>(d_rec), d_offsets, d_list, G, nt, pxy, pz, plane_lo,
                                          plane_hi, d_planes);
    SVDI_LAUNCHED();
    k_rare_w<W, WZ><<<bin_blocks(src.n), kThreads, 0, st>>>(src, g, wp, pz, (int)(src.n / src.R), plane_lo, plane_hi,
                                                            d_planes, d_dropped);
    SVDI_LAUNCHED();
    return SVDI_OK;
}

}  // namespace

int w_tiles(long long G) { return (int)((G + 7) / 8); }
size_t w_record_bytes() { return sizeof(WRec); }
// a record lies in the runs of at most four blocks, and a block with r records has fewer than r / kPart
// further parts
size_t w_list_words(long long n) { return 2 * ((size_t)n * 4 / kPart + 2); }

int launch_bin_w(const SampleSource& src, const GridGeom& g, const WPlanes& wp, unsigned int* d_counts,
                 unsigned int* d_offsets, unsigned int* d_cursor, unsigned int* d_sums, void* d_rec, cudaStream_t st) {
    const int nt = w_tiles(g.G), C = (int)(src.n / src.R);
    k_bin_w<false><<<bin_blocks(src.n), kThreads, 0, st>>>(src, g, wp, nt, C, d_counts, nullptr);
    SVDI_LAUNCHED();
    SVDI_TRY(launch_scan(d_counts, nt * nt, d_offsets, d_cursor, st, nullptr, 32, nullptr, 512, d_sums));
    k_bin_w<true><<<bin_blocks(src.n), kThreads, 0, st>>>(src, g, wp, nt, C, d_cursor, static_cast<WRec*>(d_rec));
    SVDI_LAUNCHED();
    return SVDI_OK;
}

// What bounds it: instruction issue (about 600 warp instructions a sample, its 100 taps in 10 planes) where
// samples are dense, else writing the planes (116 of 6144^2: 35 GB, 5.4 ms at 6.5 TB/s). Against one reduction
// per sample and cell into cleared planes, B200, binning and clearing included: 5.2 M samples, 116 planes of
// 6144^2 25 -> 10.5 ms; 0.64 M, 46 planes of 2304^2 1.34 -> 1.12 ms; 2.9 M, 33 planes of 1536^2 4.8 -> 3.3 ms.
// Four warps a CTA: eight are 10.0 ms on the first and 1.23 ms on the second.
int launch_grid_w(const SampleSource& src, const GridGeom& g, const WPlanes& wp, const EsPoly& pxy, const EsPoly& pz,
                  const void* d_rec, const unsigned int* d_offsets, unsigned int* d_list, int plane_lo, int plane_hi,
                  float2* d_planes, unsigned long long* d_dropped, cudaStream_t st) {
#define SVDI_W(A, B)                                                                                             \
    if (g.W == A && wp.W == B)                                                                                   \
        return launch_planes<A, B>(src, g, wp, pxy, pz, d_rec, d_offsets, d_list, plane_lo, plane_hi, d_planes,      \
                                   d_dropped, st)
    SVDI_W(8, 10);
    SVDI_W(8, 12);
    SVDI_W(6, 10);
    SVDI_W(6, 12);
#undef SVDI_W
    set_error("w planes: unsupported kernel widths");
    return SVDI_ERR_INTERNAL;
}

}  // namespace svdi
