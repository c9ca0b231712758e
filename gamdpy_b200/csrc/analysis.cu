// analysis.cu -- radial distribution function and structure factor on B200.
//
// RDF (calculators/calculator_radial_distribution.py:76-107): every ordered
// pair i != j with dist_sq < r_max^2 is counted in bin int(d / width) of its
// (type_i, type_j) histogram, with the reference's mixed precision: dist_sq
// in float32 (orthorhombic.py:59-73), the range test and d / width in
// float64, d = sqrt(dist_sq) in float32.  Counts are exact integers (uint64).
// dist_sq is symmetric bit for bit (the minimum image of -dr is -dr's), so
// each unordered pair is evaluated once and counted in both orders.
//   * r_max >= min(L)/3 (or more than 2^28 cells): all pairs, j tiles staged
//     in shared memory.
//   * smaller r_max: particles sorted into cells (counting sort) of edge >=
//     r_max in y and z and that or half of it in x; a warp takes 32 slots of
//     an x-row of cells against its own row and four neighbouring rows.  Same
//     pair set, so the same counts.
// A pair in range is binned from an approximate root and one comparison with
// the bins' edges in dist_sq, which a kernel finds first (k_rdf_edges).
// Per-block histograms live in shared memory (uint32, each unordered pair
// once) and are flushed with 64-bit atomics in both orders.
//
// S(q) (calculators/calculator_structure_factor.py:131-156, :185-203):
// rho_q = N_f^-1/2 sum_i f_i exp(i q.r_i) with q = 2 pi n / L.  Because q is
// on the reciprocal lattice, exp(i q.r) = e_x(nx) e_y(ny) e_z(nz) with
// e_d(k) = exp(2 pi i k r_d / L_d); each block tabulates e_d(k) for a tile of
// particles in shared memory (sincospi, float32), float32 sums within a tile
// and float64 across tiles.
//   * sets that pack into runs along an axis (two q-vectors a run or more): a
//     thread takes a run of eight and shares the product of the two other
//     factors among them (k_sq_runs).
//   * other sets: a thread takes up to four q-vectors, two complex products
//     each a particle (k_sq).
// The two differ by float32's rounding (1e-5 of rho_q / N^(1/2)).
#include <cuda_runtime.h>
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "../../include/gamdb200.h"
#include "gdb_internal.cuh"

using namespace gdb;

extern "C" {
const float4 *gdb_internal_pos(gdb_sim *h);
const int *gdb_internal_orig(gdb_sim *h);
cudaStream_t gdb_internal_stream(gdb_sim *h);
const float *gdb_internal_box(gdb_sim *h);
int gdb_internal_n(gdb_sim *h);
int gdb_internal_ntypes(gdb_sim *h);
int gdb_internal_dev(gdb_sim *h);
int gdb_internal_uploaded(gdb_sim *h);
char *gdb_internal_err(gdb_sim *h);
cudaEvent_t gdb_internal_event(gdb_sim *h, int k);
void gdb_internal_set_analysis_ms(gdb_sim *h, float ms);
}

// Device time of one handle call: events on the handle's stream around its
// device work (nothing for the stand-alone calculators, h == NULL).
static cudaError_t timing_begin(gdb_sim *h, cudaStream_t st) {
    return h ? cudaEventRecord(gdb_internal_event(h, 0), st) : cudaSuccess;
}
static cudaError_t timing_end(gdb_sim *h, cudaStream_t st) {
    return h ? cudaEventRecord(gdb_internal_event(h, 1), st) : cudaSuccess;
}
static void timing_store(gdb_sim *h) {
    float ms = 0.f;
    if (h && cudaEventElapsedTime(&ms, gdb_internal_event(h, 0), gdb_internal_event(h, 1)) == cudaSuccess)
        gdb_internal_set_analysis_ms(h, ms);
}

static int aset(gdb_sim *h, int code, const char *msg, cudaError_t e = cudaSuccess) {
    snprintf(gdb_internal_err(h), 512, "%s%s%s", msg, e != cudaSuccess ? ": " : "",
             e != cudaSuccess ? cudaGetErrorString(e) : "");
    return code;
}

#define ACK(call)                                                     \
    do {                                                              \
        cudaError_t e_ = (call);                                      \
        if (e_ != cudaSuccess) return aset(h, GDB_ERR_CUDA, #call, e_); \
    } while (0)

namespace {

constexpr int RDF_THREADS = 256;
constexpr int RDF_WARPS = RDF_THREADS / 32;
constexpr int RDF_TILE = RDF_THREADS;     // j positions staged per block (all-pairs path)
constexpr int RDF_SMEM_MAX_BINS = 12288;  // uint32 entries kept in shared memory
// Dynamic shared memory that a kernel may be launched with: one value for every
// call, as calls of several threads set it (a thread that sets less than
// another is about to launch with would fail that launch).
constexpr int RDF_HIST_MAX = (2 * RDF_SMEM_MAX_BINS + 1) * (int)sizeof(unsigned);  // histograms and bin edges
constexpr int SQ_SMEM_MAX = 200 * 1024, SQ_RUN_SMEM_MAX = 224 * 1024;

template <bool B>
struct RdfTag {
    static constexpr bool value = B;
};

struct RdfArgs {
    int n, nt, bins;
    float Lx, Ly, Lz;
    // smallest float32 >= r_max^2 and >= r_max: for a float32 x,
    // (double)x < r_max^2  <=>  x < r2f, so the range tests stay in float32
    float r2f, rf;
    double width, inv_width;  // r_max / bins and its rounded reciprocal
    float guess;              // (1 - 2e-6) / width, for the first guess of a bin
    const float *edge;        // bins + 1 bin edges in dist_sq (k_rdf_edges)
    unsigned long long *out;
};

// int(d / width) as the float64 division gives it.  q = d * (1 / width) is
// within 2.3e-16 q of d / width and the rounded quotient within 1.2e-16, so
// their floors can differ only when an integer k >= 1 lies within
// 3.3e-16 k of q; such quotients (|q - k| <= 1e-12 k) take the division.
__device__ __forceinline__ int rdf_bin(const RdfArgs &a, float d) {
    const double q = (double)d * a.inv_width;
    const double k = rint(q);
    int b = (k >= 1.0 && fabs(q - k) <= 1e-12 * k) ? (int)__ddiv_rn((double)d, a.width) : (int)q;
    // d < r_max, yet d / width can round up to `bins`; the reference would
    // index past its array there, this keeps the count in range
    return b < a.bins ? b : a.bins - 1;
}

// Bin edges in dist_sq.  A pair is counted when d2 < r2f and sqrt(d2) < rf,
// in bin rdf_bin(sqrt(d2)); all three grow with d2, so the pairs of bin k are
// exactly those with edge[k] <= d2 < edge[k + 1], where edge[k] is the
// smallest float32 that is out of range or has a bin >= k.  Non-negative
// floats are ordered as their bit patterns: 31 halvings find it.  The counting
// loop then needs neither the exact root nor float64.  (Histograms in global
// memory need edge[bins] only: `first`.)
__global__ void k_rdf_edges(RdfArgs a, float *edge, int first) {
    const int k = first + blockIdx.x * blockDim.x + threadIdx.x;
    if (k > a.bins) return;
    unsigned lo = 0, hi = 0x7f800000u;  // +inf is out of range
    while (lo < hi) {
        const unsigned mid = (lo + hi) >> 1;
        const float d2 = __uint_as_float(mid);
        const float d = __fsqrt_rn(d2);
        const bool at = !(d2 < a.r2f && d < a.rf) || (k < a.bins && rdf_bin(a, d) >= k);
        if (at)
            hi = mid;
        else
            lo = mid + 1;
    }
    edge[k] = __uint_as_float(lo);
}

// One pair in range (d2 < edge[bins]).  In histograms that fit shared memory
// (SH: at most RDF_SMEM_MAX_BINS bins) one count of the unordered pair in
// (t_i, t_j), rdf_flush gives every pair both orders; in histograms in global
// memory both orders at once, one addition where they are the same entry (what
// bounds those is the additions: N 100 000, 40 000 bins, all pairs, 23.6 ms, 58.6 with two additions for every pair and the
// bins searched among the edges).
// SH: a guess of the bin from the approximate root, corrected against the
// edges.  The guess d / width (1 - 2e-6) is below d / width by more than its rounding
// errors (5e-7 of it) and by less than 0.04, so its floor is the bin or the
// one before: one edge decides.  The float is truncated to the bin by
// subtracting a half, adding 1.5 2^23 (whose ulp is 1) and reading the
// mantissa: the conversion instruction runs at an eighth of the rate.
template <bool SH>
__device__ __forceinline__ void rdf_count(const RdfArgs &a, const float *edge, float d2, int row, int col,
                                          unsigned *hist) {
    if (SH) {
        float root;
        asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(root) : "f"(d2));
        const int b = __float_as_int(__fadd_rn(__fmaf_rn(root, a.guess, -0.5f), 12582912.0f)) - 0x4b400000;
        atomicAdd(&hist[row + b + (d2 >= edge[b + 1] ? 1 : 0)], 1u);
    } else {
        const int b = rdf_bin(a, __fsqrt_rn(d2));
        if (row == col) {
            atomicAdd(&a.out[row + b], 2ull);
        } else {
            atomicAdd(&a.out[row + b], 1ull);
            atomicAdd(&a.out[col + b], 1ull);
        }
    }
}

// dist_sq of a lane's particle to the staged positions q .. q + 3, two to a
// register pair.  MIC: magnitude of the minimum image per component, as the
// reference's; without it the plain difference, which callers use only where
// it gives the same pairs in range and the same dist_sq for them.
template <bool MIC>
__device__ __forceinline__ f32x2 rdf_diff(f32x2 pj, f32x2 mpi, float L) {
    f32x2 d = add2(pj, mpi);
    if (MIC) {
        float d0, d1;
        unpack2(d, d0, d1);
        d = pack2(mic_abs(d0, L), mic_abs(d1, L));
    }
    return d;
}
template <bool FMA>
__device__ __forceinline__ f32x2 rdf_norm(f32x2 dx, f32x2 dy, f32x2 dz) {
    if (FMA) return fma2(dz, dz, fma2(dy, dy, mul2(dx, dx)));
    // rounded products: the scalar intrinsics are never contracted (measured:
    // a packed multiply and add were)
    float x[2], y[2], z[2], d[2];
    unpack2(dx, x[0], x[1]);
    unpack2(dy, y[0], y[1]);
    unpack2(dz, z[0], z[1]);
#pragma unroll
    for (int k = 0; k < 2; k++)
        d[k] = __fadd_rn(__fadd_rn(__fmul_rn(x[k], x[k]), __fmul_rn(y[k], y[k])), __fmul_rn(z[k], z[k]));
    return pack2(d[0], d[1]);
}

// Positions staged for the counting loops, one array per coordinate (a
// 16-byte load gives four of them); a place past the last position holds NaN
// and is in range of nothing.
template <int N>
struct RdfStage {
    float x[N], y[N], z[N];
    int t[N];
    __device__ __forceinline__ void put(int k, float4 p, bool valid) {
        x[k] = valid ? p.x : __int_as_float(0x7fffffff);
        y[k] = p.y;
        z[k] = p.z;
        t[k] = ptype_of(p);
    }
};

// Lane's particle i (negated coordinates mx, my, mz) against the staged
// positions [q0, q0 + 32).  First pass: every candidate's dist_sq goes to
// the warp's d2s[q][lane] and in-range candidates set bit q of the lane's
// mask; bits q <= lim are dropped (j at or before i in the same row or tile).
// Second pass: every lane counts its own hits, one per round.  SHARED: the
// histograms are in shared memory (a kernel each way: with both in one, the
// loops are scheduled worse: LJ below 1.39 to 1.67 ms against 1.23).
template <bool FMA, bool MIC, bool SHARED, int N>
__device__ __forceinline__ void rdf_warp_tile(const RdfArgs &a, f32x2 mx, f32x2 my, f32x2 mz, int ti, bool act,
                                              const RdfStage<N> &st, int q0, int lim, float *d2s, int lane,
                                              const float *edge, float last, unsigned *hist) {
    unsigned mask = 0;
#pragma unroll
    for (int q = 0; q < 32; q += 4) {
        const ulonglong2 X = *reinterpret_cast<const ulonglong2 *>(&st.x[q0 + q]);
        const ulonglong2 Y = *reinterpret_cast<const ulonglong2 *>(&st.y[q0 + q]);
        const ulonglong2 Z = *reinterpret_cast<const ulonglong2 *>(&st.z[q0 + q]);
        const f32x2 e = rdf_norm<FMA>(rdf_diff<MIC>(X.x, mx, a.Lx), rdf_diff<MIC>(Y.x, my, a.Ly),
                                      rdf_diff<MIC>(Z.x, mz, a.Lz));
        const f32x2 f = rdf_norm<FMA>(rdf_diff<MIC>(X.y, mx, a.Lx), rdf_diff<MIC>(Y.y, my, a.Ly),
                                      rdf_diff<MIC>(Z.y, mz, a.Lz));
        float d[4];
        unpack2(e, d[0], d[1]);
        unpack2(f, d[2], d[3]);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            d2s[(q + k) * 32 + lane] = d[k];
            if (d[k] < last) mask |= 1u << (q + k);
        }
    }
    if (lim >= 31)
        mask = 0;
    else if (lim >= 0)
        mask &= ~0u << (lim + 1);
    if (!act) mask = 0;
    // each lane reads back its own column of d2s
    auto rounds = [&](auto one_tag) {
        constexpr bool ONE = decltype(one_tag)::value;  // one histogram
        while (mask) {
            const int q = __ffs(mask) - 1;
            mask &= mask - 1u;
            const float d2 = d2s[q * 32 + lane];
            int row = 0, col = 0;
            if (!ONE) {
                const int tj = st.t[q0 + q];
                row = (ti * a.nt + tj) * a.bins;
                col = (tj * a.nt + ti) * a.bins;
            }
            rdf_count<SHARED>(a, edge, d2, row, col, hist);
        }
    };
    if (a.nt == 1)
        rounds(RdfTag<true>{});
    else
        rounds(RdfTag<false>{});
    __syncwarp();
}

// Shared memory of a counting block: the warps' d2s, then (when the
// histograms fit) the bin edges and the histograms.
__device__ __forceinline__ const float *rdf_begin(const RdfArgs &a, unsigned char *tail, unsigned *&hist, int total,
                                                  bool shared) {
    if (!shared) {
        hist = nullptr;
        return a.edge;
    }
    float *edge = (float *)tail;
    hist = (unsigned *)(edge + a.bins + 1);
    for (int k = threadIdx.x; k <= a.bins; k += blockDim.x) edge[k] = a.edge[k];
    for (int k = threadIdx.x; k < total; k += blockDim.x) hist[k] = 0;
    __syncthreads();
    return edge;
}

// Block histograms of unordered pairs to the ordered counts.
__device__ __forceinline__ void rdf_flush(const RdfArgs &a, unsigned *hist, int total) {
    __syncthreads();
    for (int k = threadIdx.x; k < total; k += blockDim.x) {
        const int pair = k / a.bins, b = k - pair * a.bins;
        const unsigned long long c =
            (unsigned long long)hist[k] + hist[((pair % a.nt) * a.nt + pair / a.nt) * a.bins + b];
        if (c) atomicAdd(&a.out[k], c);
    }
}

// All pairs, each unordered pair once.  Tiles of RDF_TILE particles; i-tile b
// meets j-tiles b + k (mod T) for k = 0 .. T/2 (k = 0: j > i; for even T the
// tile pair at distance T/2 belongs to the lower tile), so every i-tile has
// the same work; blockIdx.y takes slice y of that k range (small systems still
// fill the GPU).
template <bool FMA, bool SHARED>
__global__ void __launch_bounds__(RDF_THREADS) k_rdf_allpairs(RdfArgs a, const float4 *pos) {
    extern __shared__ __align__(16) unsigned char smraw[];
    RdfStage<RDF_TILE> &tile = *(RdfStage<RDF_TILE> *)smraw;
    float *d2s = (float *)(smraw + sizeof(RdfStage<RDF_TILE>));  // [RDF_WARPS][32][32]
    unsigned *hist;
    const int total = a.nt * a.nt * a.bins;
    const float *edge = rdf_begin(a, (unsigned char *)(d2s + RDF_WARPS * 1024), hist, total, SHARED);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float *wd2 = d2s + w * 1024;
    const float last = edge[a.bins];  // in range: d2 < last (k_rdf_edges)
    const int T = (a.n + RDF_TILE - 1) / RDF_TILE;
    const int b = blockIdx.x;
    const int i = b * RDF_TILE + threadIdx.x;
    const bool act = i < a.n;
    const float4 pi = act ? pos[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const f32x2 mx = pack2(-pi.x, -pi.x), my = pack2(-pi.y, -pi.y), mz = pack2(-pi.z, -pi.z);
    const int ti = ptype_of(pi);
    const int kmax = (T % 2 == 0 && b >= T / 2) ? T / 2 - 1 : T / 2;
    const int per = (T / 2 + gridDim.y) / gridDim.y;  // ceil((T / 2 + 1) / S)
    const int k_end = min(kmax + 1, ((int)blockIdx.y + 1) * per);
    for (int k = blockIdx.y * per; k < k_end; k++) {
        const int jt = (b + k) % T;
        const int j0 = jt * RDF_TILE;
        const int jn = min(RDF_TILE, a.n - j0);
        __syncthreads();
        const bool valid = (int)threadIdx.x < jn;
        tile.put(threadIdx.x, valid ? pos[j0 + threadIdx.x] : pi, valid);
        __syncthreads();
        for (int q0 = 0; q0 < jn; q0 += 32)
            rdf_warp_tile<FMA, true, SHARED>(a, mx, my, mz, ti, act, tile, q0, k == 0 ? i - (j0 + q0) : -1, wd2, lane, edge,
                                     last, hist);
    }
    if (SHARED) rdf_flush(a, hist, total);
}

// Cell coordinate of the cell search (the same roundings wherever it is used).
// A coordinate at the high face, or so close to it that its cell rounds up to
// nc, stays in the last cell, beside the coordinates it can be subtracted from.
__device__ __forceinline__ int rdf_cell(float r, float L, int nc) {
    const float f = __fmul_rn(__fadd_rn(__fdiv_rn(r, L), 0.5f), (float)nc);
    if (!(f == f)) return 0;
    if (f == (float)nc && r <= 0.5f * L) return nc - 1;
    int c = (int)floorf(f) % nc;
    return c < 0 ? c + nc : c;
}

// Cell search for r_max < L/3: particles sorted by cell, x fastest; cells of
// edge >= r_max in y and z (at least 3 per side) and >= r_max / 2 in x (of
// half the edge where cells are full, see rdf_device).  A unit of work is 32 consecutive slots of one x-row of cells
// (unit u: row u / K, slots 32 (u % K) on, K = units of the fullest row; units
// past a row's end are empty), taken a unit per warp: every lane has a
// particle, whatever a cell holds.  With [xa, xb] the x-cells of the unit's
// first and last slot, its neighbours are the slots of the x-cells xa - 2 ..
// xb + 2, contiguous but for the periodic wrap, of its own row (j > i) and of
// the 4 rows of the half shell in (y, z).  Each pair of neighbouring rows is
// visited from exactly one side, each pair of particles once.
//
// Plain differences between a unit and a row part that is not reached across
// a face, in grids of at least 5 cells in y and z and windows under half of
// the x-cells: the components are then below 2 L / 5 or L / 2, which the
// minimum image leaves unchanged.  When any position lies outside [-L/2, L/2]
// (*outside set by the binning) every unit takes the minimum image.
//
// What bounds it is instruction issue (69 % of the slots), then the shared
// memory that the two passes go through (59 % of its rate).  Measured on B200, LJ, 1 000 188
// particles, r_max 5, 1000 bins: a call 3.80 ms with a warp per cell and hits
// compacted into a ring for a float64 bin, 1.23 ms here.
template <bool FMA, bool SHARED>
__global__ void __launch_bounds__(RDF_THREADS) k_rdf_cells(RdfArgs a, const float4 *spos, const int *start,
                                                           const int *outside, int ncx, int ncy, int ncz) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    RdfStage<32> &js = ((RdfStage<32> *)smraw)[w];
    float *d2s = (float *)(smraw + RDF_WARPS * sizeof(RdfStage<32>));
    unsigned *hist;
    const int total = a.nt * a.nt * a.bins;
    const float *edge = rdf_begin(a, (unsigned char *)(d2s + RDF_WARPS * 1024), hist, total, SHARED);
    float *wd2 = d2s + w * 1024;
    const float last = edge[a.bins];  // in range: d2 < last (k_rdf_edges)
    const bool inside = *outside == 0;
    const int ncell = ncx * ncy * ncz;
    const int K = start[ncell + 1];
    const long long units = (long long)ncy * ncz * K;
    for (long long u = (long long)blockIdx.x * RDF_WARPS + w; u < units; u += (long long)gridDim.x * RDF_WARPS) {
        const int row = (int)(u / K);
        const int h1 = start[(row + 1) * ncx];
        const int i0 = start[row * ncx] + 32 * (int)(u % K);
        if (i0 >= h1) continue;
        const int cy = row % ncy, cz = row / ncy;
        const int i = i0 + lane;
        const bool act = i < h1;
        const float4 pi = spos[act ? i : h1 - 1];
        const int ti = ptype_of(pi);
        const f32x2 mx = pack2(-pi.x, -pi.x), my = pack2(-pi.y, -pi.y), mz = pack2(-pi.z, -pi.z);
        const int cx = rdf_cell(pi.x, a.Lx, ncx);
        const int xa = __shfl_sync(0xffffffffu, cx, 0), xb = __shfl_sync(0xffffffffu, cx, 31);
        const bool narrow = inside && ncy >= 5 && ncz >= 5 && 2 * (xb - xa + 3) < ncx;
        // x-cells [lo, hi) of a row, and the wrapped rest [lo2, hi2)
        int lo = xa - 2, hi = xb + 3, lo2 = 0, hi2 = 0;
        if (hi - lo >= ncx) {
            lo = 0;
            hi = ncx;
        } else if (lo < 0) {
            lo2 = lo + ncx;
            hi2 = ncx;
            lo = 0;
        } else if (hi > ncx) {
            lo2 = 0;
            hi2 = hi - ncx;
            hi = ncx;
        }
        for (int s = 0; s < 10; s++) {
            // rows (0, 0), (1, 0), (-1, 1), (0, 1), (1, 1) in (y, z); s odd: the wrapped rest
            const int k = s >> 1;
            if ((s & 1) && hi2 <= lo2) continue;
            const int dy = k == 0 ? 0 : (k == 1 ? 1 : k - 3), dz = k >= 2 ? 1 : 0;
            const int y = (cy + dy + ncy) % ncy, z = (cz + dz) % ncz;
            const int base = (z * ncy + y) * ncx;
            const bool plain = narrow && !(s & 1) && y == cy + dy && z == cz + dz;
            int j0 = start[base + ((s & 1) ? lo2 : lo)];
            const int j1 = start[base + ((s & 1) ? hi2 : hi)];
            if (k == 0) j0 = max(j0, i0);  // own row: slots from the unit's first on
            for (; j0 < j1; j0 += 32) {
                __syncwarp();
                const bool valid = j0 + lane < j1;
                js.put(lane, valid ? spos[j0 + lane] : pi, valid);
                __syncwarp();
                const int lim = k == 0 ? i - j0 : -1;
                if (plain)
                    rdf_warp_tile<FMA, false, SHARED>(a, mx, my, mz, ti, act, js, 0, lim, wd2, lane, edge, last, hist);
                else
                    rdf_warp_tile<FMA, true, SHARED>(a, mx, my, mz, ti, act, js, 0, lim, wd2, lane, edge, last, hist);
            }
        }
    }
    if (SHARED) rdf_flush(a, hist, total);
}

// cell binning for the cell search: a counting sort of the positions;
// *outside = 1 when a coordinate is outside [-L/2, L/2] (or not a number)
__global__ void k_bin_cells(const float4 *pos, int n, float Lx, float Ly, float Lz, int ncx, int ncy, int ncz,
                            int *pcell, int *prank, int *count, int *outside) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p = pos[i];
    const float r[3] = {p.x, p.y, p.z};
    const float L[3] = {Lx, Ly, Lz};
    const int nc[3] = {ncx, ncy, ncz};
    int c[3];
    bool out = false;
    for (int k = 0; k < 3; k++) {
        const float h = 0.5f * L[k];
        out = out || !(r[k] >= -h && r[k] <= h);
        c[k] = rdf_cell(r[k], L[k], nc[k]);
    }
    if (out) *outside = 1;
    const int cid = (c[2] * ncy + c[1]) * ncx + c[0];
    pcell[i] = cid;
    prank[i] = atomicAdd(&count[cid], 1);
}
// exclusive prefix sum of the cell counts (start[ncell] = total) and the
// 32-particle units of the fullest row of ncx cells (start[ncell + 1]), one
// block of 1024 threads, each over a contiguous run of cells
constexpr int SCAN_THREADS = 1024;
__global__ void __launch_bounds__(SCAN_THREADS) k_cells_scan(const int *count, int *start, int ncell, int ncx) {
    __shared__ int wsum[SCAN_THREADS / 32];
    __shared__ int rmax;
    if (threadIdx.x == 0) rmax = 0;
    const int per = (ncell + SCAN_THREADS - 1) / SCAN_THREADS;
    const int c0 = min(ncell, (int)threadIdx.x * per), c1 = min(ncell, c0 + per);
    int s = 0;
    for (int c = c0; c < c1; c++) s += count[c];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = s;  // inclusive scan within the warp
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    if (w == 0) {
        int v = wsum[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += y;
        }
        wsum[lane] = v;
    }
    __syncthreads();
    int run = x - s + (w > 0 ? wsum[w - 1] : 0);
    for (int c = c0; c < c1; c++) {
        start[c] = run;
        run += count[c];
    }
    if (threadIdx.x == SCAN_THREADS - 1) start[ncell] = run;
    __syncthreads();  // every start is written
    int m = 0;
    for (int r = threadIdx.x; r < ncell / ncx; r += SCAN_THREADS) m = max(m, start[(r + 1) * ncx] - start[r * ncx]);
    atomicMax(&rmax, m);
    __syncthreads();
    if (threadIdx.x == 0) start[ncell + 1] = (rmax + 31) / 32;
}

__global__ void k_cells_scatter(const float4 *pos, const int *pcell, const int *prank, const int *start,
                                float4 *spos, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    spos[start[pcell[i]] + prank[i]] = pos[i];
}

// ---------------------------------------------------------------------------
// S(q)
// ---------------------------------------------------------------------------
constexpr int SQ_TILE = 32;      // particles per shared-memory tile
constexpr int SQ_THREADS = 256;  // q-vectors per block
constexpr int SQ_CHUNK = 8192;   // particles per block (grid y)
constexpr int SQ_RUN_THREADS = 640;  // most items per block (k_sq_runs): 20 warps at 96 registers

struct SqArgs {
    const float4 *pos;
    const int *orig;
    const float *ff;  // user order, may be null
    int n, nq;
    const int *nvec;  // nq x 3
    int kmin[3], klen[3];
    float invL[3];
    double *acc;  // nq x 2
};

// One (particle, q) term of rho_q: (e_x e_y) e_z, times the form factor w
// when weighted, added to (tr, ti).  The roundings are written out, so every
// kernel that sums with it gives the same float32 partial sums.
__device__ __forceinline__ void sq_term(float2 ex, float2 ey, float2 ez, float w, bool weighted, float &tr,
                                        float &ti) {
    const float xr = __fmaf_rn(ex.x, ey.x, -__fmul_rn(ex.y, ey.y));
    const float xi = __fmaf_rn(ex.x, ey.y, __fmul_rn(ex.y, ey.x));
    const float cr = __fmaf_rn(xr, ez.x, -__fmul_rn(xi, ez.y));
    const float ci = __fmaf_rn(xr, ez.y, __fmul_rn(xi, ez.x));
    if (weighted) {
        tr = __fmaf_rn(w, cr, tr);
        ti = __fmaf_rn(w, ci, ti);
    } else {
        tr = __fadd_rn(tr, cr);
        ti = __fadd_rn(ti, ci);
    }
}

// One block: QPT x SQ_THREADS q-vectors (q = blockIdx.x QPT 256 + k 256 + t)
// against SQ_CHUNK particles.  Per tile of SQ_TILE particles the block
// tabulates e_d(k) = exp(2 pi i k x_d / L_d) once (sincospif, float32) and
// every thread accumulates its QPT q-vectors from the table: two complex
// products per (particle, q), float32 within a tile, float64 across tiles.
template <int QPT, bool FF>
__global__ void __launch_bounds__(SQ_THREADS) k_sq(SqArgs a) {
    extern __shared__ float2 tab[];  // [SQ_TILE][klen0 + klen1 + klen2]
    __shared__ float wsh[SQ_TILE];
    __shared__ float4 psh[SQ_TILE];
    const int k0 = a.klen[0], k01 = a.klen[0] + a.klen[1];
    const int row = k01 + a.klen[2];
    int ix[QPT], iy[QPT], iz[QPT];
#pragma unroll
    for (int k = 0; k < QPT; k++) {
        const int q = (blockIdx.x * QPT + k) * SQ_THREADS + threadIdx.x;
        ix[k] = 0, iy[k] = 0, iz[k] = 0;  // inactive slots read entry 0 and are not stored
        if (q < a.nq) {
            ix[k] = a.nvec[3 * q] - a.kmin[0];
            iy[k] = a.nvec[3 * q + 1] - a.kmin[1] + k0;
            iz[k] = a.nvec[3 * q + 2] - a.kmin[2] + k01;
        }
    }
    double sr[QPT], si[QPT];
#pragma unroll
    for (int k = 0; k < QPT; k++) sr[k] = si[k] = 0.0;
    // this thread's table entries: (pl0, col0) then steps of SQ_THREADS
    const int dpl = SQ_THREADS / row, dcol = SQ_THREADS % row;
    const int pl0 = threadIdx.x / row, col0 = threadIdx.x % row;
    const int p_begin = blockIdx.y * SQ_CHUNK;
    const int p_end = min(a.n, p_begin + SQ_CHUNK);
    for (int p0 = p_begin; p0 < p_end; p0 += SQ_TILE) {
        const int np = min(SQ_TILE, p_end - p0);
        __syncthreads();
        if (threadIdx.x < np) {
            psh[threadIdx.x] = a.pos[p0 + threadIdx.x];
            if (FF) wsh[threadIdx.x] = a.ff[a.orig[p0 + threadIdx.x]];
        }
        __syncthreads();
        for (int pl = pl0, col = col0; pl < np;) {
            const int d = (col >= k0) + (col >= k01);
            const int kk = col - (d == 0 ? 0 : (d == 1 ? k0 : k01)) + a.kmin[d];
            const float4 p = psh[pl];
            const float x = d == 0 ? p.x : (d == 1 ? p.y : p.z);
            float sn, cs;
            sincospif(2.0f * (float)kk * (x * a.invL[d]), &sn, &cs);
            tab[pl * row + col] = make_float2(cs, sn);
            col += dcol;
            pl += dpl;
            if (col >= row) {
                col -= row;
                pl++;
            }
        }
        __syncthreads();
        float tr[QPT], ti[QPT];
#pragma unroll
        for (int k = 0; k < QPT; k++) tr[k] = ti[k] = 0.f;
        for (int pl = 0; pl < np; pl++) {
            const float2 *t = tab + pl * row;
            const float w = FF ? wsh[pl] : 1.0f;
#pragma unroll
            for (int k = 0; k < QPT; k++) {
                sq_term(t[ix[k]], t[iy[k]], t[iz[k]], w, FF, tr[k], ti[k]);
            }
        }
#pragma unroll
        for (int k = 0; k < QPT; k++) {
            sr[k] += tr[k];
            si[k] += ti[k];
        }
    }
#pragma unroll
    for (int k = 0; k < QPT; k++) {
        const int q = (blockIdx.x * QPT + k) * SQ_THREADS + threadIdx.x;
        if (q < a.nq) {
            atomicAdd(&a.acc[2 * q], sr[k]);
            atomicAdd(&a.acc[2 * q + 1], si[k]);
        }
    }
}

// Runs of q-vectors: an item is one pair (a, b) of components along two of the
// axes and SQ_Z consecutive components along the third (the run axis).  A
// thread owns an item: per particle it multiplies e_a(a) e_b(b) and adds its
// products with the run's SQ_Z factors, so a term costs two packed
// multiply-adds and 10 bytes of shared memory, against two complex products
// and 24 bytes in k_sq.  float32 within a tile of SQ_TILE particles, float64
// across tiles, as k_sq.  What bounds it is the 6 shared loads a run (76 % of
// the shared memory's rate; 60 % of the issue slots).  Measured on B200 with 1 000 188 particles and 3778 q-vectors in
// an octant: a call 4.04 ms with k_sq, 1.51 here, 1.34 of it this kernel; with
// one table and two barriers a tile 1.38, with two items a thread (320
// threads) 1.57 to 1.85, with two blocks an SM at 48 registers 1.59.  Items
// beyond SQ_RUN_THREADS take another block that tabulates the particles again:
// a call of 10^6 particles with 640 items takes 2.35 ms, with 641 2.95, with
// 1280 3.78.
constexpr int SQ_Z = 8;
struct SqRunArgs {
    const float4 *pos;
    const int *orig;
    const float *ff;  // user order, may be null
    int n, nitems;
    int chunk;        // particles per block, a multiple of SQ_TILE
    const int4 *items;  // table columns of a, b and of the run's first entry (even); w unused
    int axis[3];        // coordinate of each third of the table: a, b, run axis
    int kmin[3], klen[3];  // klen[0] + klen[1] and klen[2] even (16-byte loads of the run)
    float invL[3];         // 1 / box length, by third of the table
    double *acc;  // [2 SQ_Z][nitems]: re and im of entry z at rows 2 z, 2 z + 1
};

template <bool FF>
__global__ void __launch_bounds__(SQ_RUN_THREADS, 1) k_sq_runs(SqRunArgs a) {
    extern __shared__ __align__(16) float2 rtab[];  // two tables [SQ_TILE][klen0 + klen1 + klen2]
    __shared__ float wsh[3][SQ_TILE];
    __shared__ float xsh[2][3][SQ_TILE];  // coordinate / box length along a, b and the run axis
    const int k0 = a.klen[0], k01 = a.klen[0] + a.klen[1];
    const int row = k01 + a.klen[2];
    const int item = blockIdx.x * blockDim.x + threadIdx.x;
    const int4 it = a.items[min(item, a.nitems - 1)];  // threads past the end repeat the last item, unstored
    const int ca = it.x, cb = it.y, cz = it.z;
    // the thread's float64 sums stay in shared memory (touched once per tile):
    // their 32 registers cost a third of the warps an SM holds
    double *sum = reinterpret_cast<double *>(rtab + 2 * SQ_TILE * row) + threadIdx.x;
#pragma unroll
    for (int j = 0; j < 2 * SQ_Z; j++) sum[j * blockDim.x] = 0.0;
    const int dpl = blockDim.x / row, dcol = blockDim.x % row;
    const int pl0 = threadIdx.x / row, col0 = threadIdx.x % row;
    const int p_begin = blockIdx.y * a.chunk;
    const int p_end = min(a.n, p_begin + a.chunk);
    const int tiles = (p_end - p_begin + SQ_TILE - 1) / SQ_TILE;
    // particle of tile t that this thread (one of the first SQ_TILE) stages; a
    // place past the end repeats the last particle and is not summed
    auto fetch = [&](int t, float4 &p, float &w) {
        const int k = min(p_begin + t * SQ_TILE + (int)threadIdx.x, p_end - 1);
        p = a.pos[k];
        if (FF) w = a.ff[a.orig[k]];
    };
    auto stage = [&](int t, float4 p, float w) {
#pragma unroll
        for (int d = 0; d < 3; d++)
            xsh[t & 1][d][threadIdx.x] = (a.axis[d] == 0 ? p.x : (a.axis[d] == 1 ? p.y : p.z)) * a.invL[d];
        if (FF) wsh[t % 3][threadIdx.x] = w;
    };
    auto tabulate = [&](int t) {
        float2 *tab = rtab + (t & 1) * SQ_TILE * row;
        for (int pl = pl0, col = col0; pl < SQ_TILE;) {
            const int d = (col >= k0) + (col >= k01);
            const int kk = col + (d == 0 ? a.kmin[0] : (d == 1 ? a.kmin[1] - k0 : a.kmin[2] - k01));
            float sn, cs;
            sincospif(2.0f * (float)kk * xsh[t & 1][d][pl], &sn, &cs);
            tab[pl * row + col] = make_float2(cs, sn);
            col += dcol;
            pl += dpl;
            if (col >= row) {
                col -= row;
                pl++;
            }
        }
    };
    const bool loader = threadIdx.x < SQ_TILE;
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
    float w = 0.f;
    for (int t = 0; t < 2; t++)
        if (loader) {
            fetch(t, p, w);
            stage(t, p, w);
        }
    __syncthreads();
    tabulate(0);
    __syncthreads();
    // one barrier a tile: the next tile's table is made beside this tile's
    // sums, from the positions loaded a tile before
    for (int t = 0; t < tiles; t++) {
        if (loader) fetch(t + 2, p, w);
        if (t + 1 < tiles) tabulate(t + 1);
        const int np = min(SQ_TILE, p_end - p_begin - t * SQ_TILE);
        const float2 *tab = rtab + (t & 1) * SQ_TILE * row;
        // sums of x_re (z_re, z_im) and x_im (z_re, z_im), x = e_a e_b
        f32x2 pz[SQ_Z], qz[SQ_Z];
#pragma unroll
        for (int z = 0; z < SQ_Z; z++) pz[z] = qz[z] = 0ull;
#pragma unroll 2
        for (int pl = 0; pl < np; pl++) {
            const float2 *e = tab + pl * row;
            const float2 ea = e[ca], eb = e[cb];
            float re = __fmaf_rn(ea.x, eb.x, -__fmul_rn(ea.y, eb.y));
            float im = __fmaf_rn(ea.x, eb.y, __fmul_rn(ea.y, eb.x));
            if (FF) {
                re *= wsh[t % 3][pl];
                im *= wsh[t % 3][pl];
            }
            const f32x2 xr = pack2(re, re), xi = pack2(im, im);
            const ulonglong2 *zr = reinterpret_cast<const ulonglong2 *>(e + cz);
#pragma unroll
            for (int z = 0; z < SQ_Z; z += 2) {
                const ulonglong2 g = zr[z / 2];
                pz[z] = fma2(xr, g.x, pz[z]);
                qz[z] = fma2(xi, g.x, qz[z]);
                pz[z + 1] = fma2(xr, g.y, pz[z + 1]);
                qz[z + 1] = fma2(xi, g.y, qz[z + 1]);
            }
        }
#pragma unroll
        for (int z = 0; z < SQ_Z; z++) {
            float pr, pi, qr, qi;
            unpack2(pz[z], pr, pi);
            unpack2(qz[z], qr, qi);
            sum[(2 * z) * blockDim.x] += pr - qi;
            sum[(2 * z + 1) * blockDim.x] += pi + qr;
        }
        if (loader) stage(t + 2, p, w);  // (the table of tile t, the last to use this place, is made)
        __syncthreads();
    }
    if (item < a.nitems)
        for (int j = 0; j < 2 * SQ_Z; j++) atomicAdd(&a.acc[(size_t)j * a.nitems + item], sum[j * blockDim.x]);
}

template <int QPT>
static void launch_sq(dim3 grid, size_t smem, cudaStream_t st, const SqArgs &a) {
    if (a.ff)
        k_sq<QPT, true><<<grid, SQ_THREADS, smem, st>>>(a);
    else
        k_sq<QPT, false><<<grid, SQ_THREADS, smem, st>>>(a);
}

// ---------------------------------------------------------------------------
// trajectory dynamics (tools/calc_dynamics.py:6-75)
// ---------------------------------------------------------------------------
constexpr int DYN_THREADS = 256;
constexpr int DYN_MAX_TYPES = 8;

// Frame pair p (frames f0 -> f1, each 2 x n x 3 float32: positions, then
// image counts): dR = (r1 - r0) + (i1 - i0) L in float32 as the reference,
// dR^2 summed over x, y, z in float32; per type the float64 sums of dR^2,
// (dR^2)^2 and cos(q_t dR_k) over particles and components, into
// acc[(p * nt + t) * 3 + {0, 1, 2}].
__global__ void __launch_bounds__(DYN_THREADS) k_dynamics(const float *frames, int n, const int *ptype, int nt,
                                                          float Lx, float Ly, float Lz, const int2 *pairs,
                                                          const double *q, double *acc) {
    __shared__ double red[DYN_MAX_TYPES * 3];
    for (int k = threadIdx.x; k < nt * 3; k += blockDim.x) red[k] = 0.0;
    __syncthreads();
    const int2 pr = pairs[blockIdx.y];
    const float *A = frames + (size_t)pr.x * 2 * n * 3;
    const float *B = frames + (size_t)pr.y * 2 * n * 3;
    const float L[3] = {Lx, Ly, Lz};
    double s[DYN_MAX_TYPES][3];
#pragma unroll
    for (int t = 0; t < DYN_MAX_TYPES; t++) s[t][0] = s[t][1] = s[t][2] = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int t = ptype[i];
        float d[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const float dr = __fsub_rn(B[3 * i + k], A[3 * i + k]);
            const float di = __fsub_rn(B[3 * n + 3 * i + k], A[3 * n + 3 * i + k]);
            d[k] = __fadd_rn(dr, __fmul_rn(di, L[k]));
        }
        const float sq = __fadd_rn(__fadd_rn(__fmul_rn(d[0], d[0]), __fmul_rn(d[1], d[1])), __fmul_rn(d[2], d[2]));
        const double qt = q[t];
        const double c = cos((double)d[0] * qt) + cos((double)d[1] * qt) + cos((double)d[2] * qt);
#pragma unroll
        for (int u = 0; u < DYN_MAX_TYPES; u++)
            if (u == t) {
                s[u][0] += sq;
                s[u][1] += (double)__fmul_rn(sq, sq);
                s[u][2] += c;
            }
    }
    for (int t = 0; t < nt; t++)
        for (int k = 0; k < 3; k++) {
            const double v = warp_sum(s[t][k]);
            if ((threadIdx.x & 31) == 0) atomicAdd(&red[t * 3 + k], v);
        }
    __syncthreads();
    for (int k = threadIdx.x; k < nt * 3; k += blockDim.x)
        atomicAdd(&acc[(size_t)blockIdx.y * nt * 3 + k], red[k]);
}

__global__ void k_pack_pos(int n, const float *r, const int *pt, float4 *pos, int *orig) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    pos[i] = make_float4(r[3 * i], r[3 * i + 1], r[3 * i + 2], __int_as_float(pt ? pt[i] : 0));
    orig[i] = i;
}

}  // namespace

// ---------------------------------------------------------------------------
// host implementations working on device-resident positions
// ---------------------------------------------------------------------------
// smallest float32 >= x
static float float_at_or_above(double x) {
    float f = (float)x;
    if ((double)f < x) f = nextafterf(f, INFINITY);
    return f;
}

static int rdf_device(gdb_sim *h, cudaStream_t st, const float4 *pos, int n, const float *box, int nt, int bins,
                      double r_max, uint64_t *out_host) {
    if (bins < 1 || nt < 1) return aset(h, GDB_ERR_ARG, "rdf: bins and ntypes must be positive");
    // the kernels index the nt^2 histograms and the bins' edges by int
    if ((double)nt * nt * bins > 2147483647.0 || bins > 2147483646)
        return aset(h, GDB_ERR_ARG, "rdf: more than 2^31 - 1 histogram entries");
    float minL = fminf(box[0], fminf(box[1], box[2]));
    // the reference: min_box_dim float32, (min_box_dim / 2) float64
    const double half = (double)minL / 2.0;
    if (r_max <= 0.0) r_max = half;
    if (r_max > half) return aset(h, GDB_ERR_ARG, "rdf: r_max must not exceed min(L)/2");
    RdfArgs a;
    a.n = n;
    a.nt = nt;
    a.bins = bins;
    a.Lx = box[0];
    a.Ly = box[1];
    a.Lz = box[2];
    a.r2f = float_at_or_above(r_max * r_max);
    a.rf = float_at_or_above(r_max);
    a.width = r_max / (double)bins;
    a.inv_width = 1.0 / a.width;
    a.guess = (float)(a.inv_width * (1.0 - 2e-6));
    const char *fm = getenv("GDB_NBLIST_FMA");
    const bool fma = !(fm && fm[0] == '0');
    const size_t total = (size_t)nt * nt * bins;
    ACK(timing_begin(h, st));
    unsigned long long *dout = nullptr;  // the counts, then the bins' edges
    ACK(pool_alloc((unsigned char **)&dout,
                   total * sizeof(unsigned long long) + ((size_t)bins + 1) * sizeof(float), st));
    ACK(cudaMemsetAsync(dout, 0, total * sizeof(unsigned long long), st));
    a.out = dout;
    float *dedge = (float *)(dout + total);
    a.edge = dedge;
    // histograms and bin edges in shared memory
    const bool shared = total <= (size_t)RDF_SMEM_MAX_BINS;
    const size_t hist_bytes = shared ? total * sizeof(unsigned) + ((size_t)bins + 1) * sizeof(float) : 0;
    const int first = shared ? 0 : bins;
    k_rdf_edges<<<(bins - first) / 128 + 1, 128, 0, st>>>(a, dedge, first);
    int nc[3];
    bool cells = true;
    for (int k = 0; k < 3; k++) {
        // edge slightly above r_max so float32 rounding of the cell
        // coordinate can never separate a pair closer than r_max by two cells
        const double edges = box[k] / (r_max * (1.0 + 1e-4));
        if (edges < 3.0) cells = false;
        nc[k] = (int)floor(edges);
    }
    // cells of half the edge in x from 12 particles a whole one on: the search
    // gains from the narrower windows, the counts' scan loses (a call, us,
    // whole and half: N 300 000 at 4 a cell 839 and 1030, at 12 804 and 816,
    // at 24 865 and 830, at 128 1537 and 1240; N 30 000 at 0.01 3510 and 7505)
    const int ncx2 = cells ? (int)floor(2.0 * (box[0] / (r_max * (1.0 + 1e-4)))) : 0;
    const long long yz = (long long)nc[1] * nc[2];
    if (cells && ncx2 * yz > (1LL << 28)) cells = false;  // r_max tiny against L: fall back to all pairs
    if (cells && 6 * ncx2 * yz <= n) nc[0] = ncx2;
    const long long ncell = cells ? nc[0] * yz : 0;
    if (!cells) {
        const size_t smem = sizeof(RdfStage<RDF_TILE>) + RDF_WARPS * 1024 * sizeof(float) + hist_bytes;
        const int T = (n + RDF_TILE - 1) / RDF_TILE;
        int dev = 0, sms = 0, per_sm = 0;
        ACK(cudaGetDevice(&dev));
        ACK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        auto kern = shared ? (fma ? k_rdf_allpairs<true, true> : k_rdf_allpairs<false, true>)
                           : (fma ? k_rdf_allpairs<true, false> : k_rdf_allpairs<false, false>);
        ACK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(smem - hist_bytes) + RDF_HIST_MAX));
        ACK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, RDF_THREADS, smem));
        // slices of the tile-distance range: about two waves of blocks in all
        const int slots = sms * std::max(per_sm, 1);
        const int S = std::max(1, std::min(T / 2 + 1, (2 * slots + T - 1) / T));
        kern<<<dim3(T, S), RDF_THREADS, smem, st>>>(a, pos);
        ACK(cudaGetLastError());
    } else {
        int *count = nullptr, *start = nullptr, *pcell = nullptr, *prank = nullptr;
        float4 *spos = nullptr;
        ACK(pool_alloc(&count, (ncell + 1) * sizeof(int), st));  // [ncell]: the outside flag
        ACK(pool_alloc(&start, (ncell + 2) * sizeof(int), st));
        ACK(pool_alloc(&pcell, (size_t)n * sizeof(int), st));
        ACK(pool_alloc(&prank, (size_t)n * sizeof(int), st));
        ACK(pool_alloc(&spos, (size_t)n * sizeof(float4), st));
        ACK(cudaMemsetAsync(count, 0, (ncell + 1) * sizeof(int), st));
        const int g = (n + 255) / 256;
        k_bin_cells<<<g, 256, 0, st>>>(pos, n, box[0], box[1], box[2], nc[0], nc[1], nc[2], pcell, prank, count,
                                      count + ncell);
        k_cells_scan<<<1, SCAN_THREADS, 0, st>>>(count, start, (int)ncell, nc[0]);
        k_cells_scatter<<<g, 256, 0, st>>>(pos, pcell, prank, start, spos, n);
        const size_t smem = RDF_WARPS * (sizeof(RdfStage<32>) + 1024 * sizeof(float)) + hist_bytes;
        int dev = 0, sms = 0, per_sm = 0;
        ACK(cudaGetDevice(&dev));
        ACK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        auto kern = shared ? (fma ? k_rdf_cells<true, true> : k_rdf_cells<false, true>)
                           : (fma ? k_rdf_cells<true, false> : k_rdf_cells<false, false>);
        ACK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(smem - hist_bytes) + RDF_HIST_MAX));
        ACK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, RDF_THREADS, smem));
        const int grid = sms * std::max(per_sm, 1);  // warps stride over the units
        kern<<<grid, RDF_THREADS, smem, st>>>(a, spos, start, count + ncell, nc[0], nc[1], nc[2]);
        ACK(cudaGetLastError());
        ACK(cudaFreeAsync(count, st));
        ACK(cudaFreeAsync(start, st));
        ACK(cudaFreeAsync(pcell, st));
        ACK(cudaFreeAsync(prank, st));
        ACK(cudaFreeAsync(spos, st));
    }
    std::vector<unsigned long long> tmp(total);
    ACK(timing_end(h, st));
    ACK(cudaMemcpyAsync(tmp.data(), dout, total * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st));
    ACK(cudaFreeAsync(dout, st));
    ACK(cudaStreamSynchronize(st));
    timing_store(h);
    for (size_t k = 0; k < total; k++) out_host[k] += tmp[k];
    return GDB_OK;
}

// Items of k_sq_runs for a set of q-vectors, along the run axis that needs the
// fewest; entry[q] is the q-vector's place in the accumulators, z * nitems +
// item.
struct SqRuns {
    int axis[3], kmin[3], klen[3];
    std::vector<int4> items;
    std::vector<int> entry;
};

// One bit per cell of a bounding grid, columns of nz cells along a run axis.
struct SqGrid {
    int axis[3], kmin[3], klen[3];
    std::vector<uint64_t> bits;
    std::vector<unsigned> cell;  // by q-vector
    void mark(int nq, const int32_t *nvec, const int lo[3], const int len[3], int run) {
        axis[0] = run == 0 ? 1 : 0;
        axis[1] = run == 2 ? 1 : 2;
        axis[2] = run;
        for (int d = 0; d < 3; d++) {
            kmin[d] = lo[axis[d]];
            klen[d] = len[axis[d]];
        }
        bits.assign(((size_t)klen[0] * klen[1] * klen[2] + 63) / 64, 0);
        cell.resize(nq);
        const unsigned s1 = klen[2], s0 = klen[1] * s1;  // (modulo 2^32; a cell's number is below 2^31)
        const unsigned off = kmin[0] * s0 + kmin[1] * s1 + kmin[2];
        const int32_t *v0 = nvec + axis[0], *v1 = nvec + axis[1], *v2 = nvec + axis[2];
        for (size_t q = 0; q < (size_t)nq; q++) {
            const unsigned c = (unsigned)v0[3 * q] * s0 + (unsigned)v1[3 * q] * s1 + (unsigned)v2[3 * q] - off;
            cell[q] = c;
            bits[c / 64] |= 1ull << (c % 64);
        }
    }
    // at most as many as there are runs: the marked cells without another
    // among the seven before them
    size_t runs_at_least() const {
        size_t count = 0;
        uint64_t last = 0;
        for (const uint64_t m : bits) {
            if (!m) {
                last = 0;
                continue;
            }
            unsigned __int128 before = ((unsigned __int128)m << 64 | last) << 1;  // marked 1, then 1 to 7 before
            before |= before << 1;
            before |= before << 2;
            before |= before << 3;
            count += __builtin_popcountll(m & ~(uint64_t)(before >> 64));
            last = m;
        }
        return count;
    }
    // the runs in the order of their cells: f(first cell marked, its column,
    // start of the run)
    template <class F>
    void runs(F f) const {
        const unsigned nz = klen[2];
        for (unsigned pos = 0, w = 0; (w = pos / 64) < bits.size();) {
            const uint64_t m = bits[w] >> (pos % 64);
            if (!m) {
                pos = 64 * (w + 1);
                continue;
            }
            pos += __builtin_ctzll(m);
            const unsigned col = pos / nz, z0 = (pos - col * nz) & ~1u;  // a run starts at an even component
            f(pos, col, (int)z0);
            pos = col * nz + std::min(nz, z0 + SQ_Z);
        }
    }
};

// False where k_sq takes the set: runs of less than two q-vectors on average,
// so that scattered sets keep k_sq's roundings (those of
// gdb_sq_compute_noalloc), not because runs are slower there: measured, calls
// with k_sq and with runs at 1.6 q-vectors a run, N 20 000 and 250 of them 798
// and 233 us, N 1 000 000 and 600 of them 2425 and 1955 us.  Or a set much
// sparser than its bounding grid (or wide).  The grid is one bit a
// cell and its runs are counted before any item is made, so that a set that
// stays with k_sq costs little: a call of 1000 particles with 1000 scattered
// q-vectors within 24 of the origin took 834 us with all three axes' items
// made on a grid of integers and takes 559, with 3778 of them 1246 and 615.
static bool sq_runs_plan(int nq, const int32_t *nvec, const int kmin[3], const int klen[3], SqRuns &best) {
    const double cells = (double)klen[0] * klen[1] * klen[2];
    if (cells > 64.0 * nq + 65536.0 || cells > 2147483648.0) return false;
    SqGrid g, t;
    size_t nitems = 0;
    for (int run = 2; run >= 0; run--) {
        // (runs along z that are half full are good enough)
        if (nitems && nitems * SQ_Z <= 2 * (size_t)nq) break;
        t.mark(nq, nvec, kmin, klen, run);
        if (2 * t.runs_at_least() > (size_t)nq) continue;
        size_t count = 0;
        t.runs([&](unsigned, unsigned, int) { count++; });
        if (nitems && nitems <= count) continue;
        nitems = count;
        std::swap(g, t);
    }
    if (!nitems || 2 * nitems > (size_t)nq) return false;
    // a q-vector's run is the last one that starts at or before its cell
    std::vector<uint64_t> first(g.bits.size(), 0);
    std::vector<int> below(g.bits.size() + 1, 0);  // runs that start in earlier words
    std::vector<int4> items;
    std::vector<unsigned> start;  // cell of a run's entry 0
    items.reserve(nitems);
    start.reserve(nitems);
    g.runs([&](unsigned pos, unsigned col, int z0) {
        first[pos / 64] |= 1ull << (pos % 64);
        below[pos / 64 + 1]++;
        items.push_back(make_int4((int)(col / (unsigned)g.klen[1]), (int)(col % (unsigned)g.klen[1]), z0, 0));
        start.push_back(col * (unsigned)g.klen[2] + z0);
    });
    for (size_t w = 1; w < below.size(); w++) below[w] += below[w - 1];
    // the lanes of a warp share a run (broadcast loads): items in the order
    // of their run's start
    std::vector<int> place(nitems), at(g.klen[2] + 1, 0);
    for (const int4 &i : items) at[i.z + 1]++;
    for (int z = 0; z < g.klen[2]; z++) at[z + 1] += at[z];
    for (size_t k = 0; k < nitems; k++) place[k] = at[items[k].z]++;
    best.entry.resize(nq);
    for (int q = 0; q < nq; q++) {
        const unsigned c = g.cell[q];
        const int k = below[c / 64] + __builtin_popcountll(first[c / 64] << (63 - c % 64)) - 1;
        best.entry[q] = (int)(c - start[k]) * (int)nitems + place[k];
    }
    best.items.resize(nitems);
    for (size_t k = 0; k < nitems; k++) best.items[place[k]] = items[k];
    for (int d = 0; d < 3; d++) {
        best.axis[d] = g.axis[d];
        best.kmin[d] = g.kmin[d];
        best.klen[d] = g.klen[d];
    }
    // table columns: the run's section starts at an even column and holds
    // whole runs, so that their 16-byte loads are aligned and inside a row
    best.klen[1] += (best.klen[0] + best.klen[1]) & 1;
    int zlen = 0;
    for (const int4 &i : best.items) zlen = std::max(zlen, i.z + SQ_Z);
    best.klen[2] = std::max(best.klen[2] + (best.klen[2] & 1), zlen);
    for (int4 &i : best.items) {
        i.y += best.klen[0];
        i.z += best.klen[0] + best.klen[1];
    }
    return true;
}

// Shared memory of k_sq_runs: two tables and the threads' float64 sums.
static size_t sq_runs_smem(const int klen[3], int threads) {
    return (size_t)2 * SQ_TILE * (klen[0] + klen[1] + klen[2]) * sizeof(float2) +
           (size_t)threads * 2 * SQ_Z * sizeof(double);
}
static cudaError_t launch_sq_runs(cudaStream_t st, SqRunArgs &r, int n) {
    const void *fn = r.ff ? (const void *)k_sq_runs<true> : (const void *)k_sq_runs<false>;
    // as few blocks along the items as SQ_RUN_THREADS allows (every one of
    // them tabulates the particles again), of equal size
    const int nbx = (r.nitems + SQ_RUN_THREADS - 1) / SQ_RUN_THREADS;
    // (at least SQ_TILE threads: they stage the positions)
    const int threads = ((r.nitems + nbx - 1) / nbx + 31) / 32 * 32;
    const size_t smem = sq_runs_smem(r.klen, threads);
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e;
    if ((e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, SQ_RUN_SMEM_MAX)) ||
        (e = cudaGetDevice(&dev)) || (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) ||
        (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem)))
        return e;
    // four waves of blocks (an uneven last wave is an eighth of the time at
    // most), of at least four tiles
    const int slots = std::max(1, sms * std::max(per_sm, 1) * 4 / nbx);
    r.chunk = std::max(4 * SQ_TILE, ((n + slots - 1) / slots + SQ_TILE - 1) / SQ_TILE * SQ_TILE);
    const dim3 grid(nbx, (n + r.chunk - 1) / r.chunk);
    if (r.ff)
        k_sq_runs<true><<<grid, threads, smem, st>>>(r);
    else
        k_sq_runs<false><<<grid, threads, smem, st>>>(r);
    return cudaGetLastError();
}

static int sq_device(gdb_sim *h, cudaStream_t st, const float4 *pos, const int *orig, int n, const float *ff_host,
                     const float *box, int nq, const int32_t *nvec_host, double *re, double *im) {
    if (nq < 1) return GDB_OK;
    SqArgs a;
    a.pos = pos;
    a.orig = orig;
    a.n = n;
    a.nq = nq;
    for (int d = 0; d < 3; d++) {
        int lo = nvec_host[d], hi = nvec_host[d];
        for (int q = 0; q < nq; q++) {
            lo = nvec_host[3 * q + d] < lo ? nvec_host[3 * q + d] : lo;
            hi = nvec_host[3 * q + d] > hi ? nvec_host[3 * q + d] : hi;
        }
        a.kmin[d] = lo;
        a.klen[d] = hi - lo + 1;
        a.invL[d] = 1.0f / box[d];
    }
    const int row = a.klen[0] + a.klen[1] + a.klen[2];
    const size_t smem = (size_t)SQ_TILE * row * sizeof(float2);
    if (smem > SQ_SMEM_MAX) return aset(h, GDB_ERR_ARG, "sq: n_vectors span too wide");
    SqRuns plan;
    const bool runs = sq_runs_plan(nq, nvec_host, a.kmin, a.klen, plan) &&
                      sq_runs_smem(plan.klen, SQ_RUN_THREADS) <= SQ_RUN_SMEM_MAX;
    const size_t nacc = runs ? plan.items.size() * SQ_Z * 2 : (size_t)nq * 2;
    int *dn = nullptr;  // n-vectors, or the runs' items
    float *dff = nullptr;
    double *acc = nullptr;
    const size_t dn_bytes = runs ? plan.items.size() * sizeof(int4) : (size_t)nq * 3 * sizeof(int);
    ACK(timing_begin(h, st));
    ACK(pool_alloc(&dn, dn_bytes, st));
    ACK(pool_alloc(&acc, nacc * sizeof(double), st));
    ACK(cudaMemcpyAsync(dn, runs ? (const void *)plan.items.data() : (const void *)nvec_host, dn_bytes,
                        cudaMemcpyHostToDevice, st));
    ACK(cudaMemsetAsync(acc, 0, nacc * sizeof(double), st));
    double nf = 0.0;
    if (ff_host) {
        ACK(pool_alloc(&dff, (size_t)n * sizeof(float), st));
        ACK(cudaMemcpyAsync(dff, ff_host, (size_t)n * sizeof(float), cudaMemcpyHostToDevice, st));
        for (int i = 0; i < n; i++) nf += ff_host[i];
    } else {
        nf = n;
    }
    a.nvec = dn;
    a.ff = dff;
    a.acc = acc;
    SqRunArgs r;
    if (runs) {
        r.pos = pos;
        r.orig = orig;
        r.ff = dff;
        r.n = n;
        r.nitems = (int)plan.items.size();
        r.items = (const int4 *)dn;
        r.acc = acc;
        for (int d = 0; d < 3; d++) {
            r.axis[d] = plan.axis[d];
            r.kmin[d] = plan.kmin[d];
            r.klen[d] = plan.klen[d];
            r.invL[d] = a.invL[plan.axis[d]];
        }
    }
    if (runs) {
        ACK(launch_sq_runs(st, r, n));
    } else {
        // q-vectors per thread: up to 4, as few blocks along q as that allows,
        // spread evenly over them (2219 q: 3 blocks of 3 x 256)
        const int nbx = (nq + 4 * SQ_THREADS - 1) / (4 * SQ_THREADS);
        const int qpt = (nq + nbx * SQ_THREADS - 1) / (nbx * SQ_THREADS);
        const dim3 grid(nbx, (n + SQ_CHUNK - 1) / SQ_CHUNK);
        const void *fn = nullptr;
        switch (qpt) {
            case 1: fn = a.ff ? (const void *)k_sq<1, true> : (const void *)k_sq<1, false>; break;
            case 2: fn = a.ff ? (const void *)k_sq<2, true> : (const void *)k_sq<2, false>; break;
            case 3: fn = a.ff ? (const void *)k_sq<3, true> : (const void *)k_sq<3, false>; break;
            default: fn = a.ff ? (const void *)k_sq<4, true> : (const void *)k_sq<4, false>; break;
        }
        ACK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, SQ_SMEM_MAX));
        switch (qpt) {
            case 1: launch_sq<1>(grid, smem, st, a); break;
            case 2: launch_sq<2>(grid, smem, st, a); break;
            case 3: launch_sq<3>(grid, smem, st, a); break;
            default: launch_sq<4>(grid, smem, st, a); break;
        }
    }
    ACK(cudaGetLastError());
    std::vector<double> tmp(nacc);
    ACK(timing_end(h, st));
    ACK(cudaMemcpyAsync(tmp.data(), acc, tmp.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
    ACK(cudaFreeAsync(dn, st));
    ACK(cudaFreeAsync(acc, st));
    if (dff) ACK(cudaFreeAsync(dff, st));
    ACK(cudaStreamSynchronize(st));
    timing_store(h);
    const double norm = 1.0 / sqrt(nf);
    for (int q = 0; q < nq; q++) {
        // runs: entry z * nitems + item, its real part at row 2 z of tmp
        const size_t nitems = plan.items.size();
        const size_t e = runs ? (size_t)plan.entry[q] / nitems * 2 * nitems + (size_t)plan.entry[q] % nitems : 2 * (size_t)q;
        re[q] = tmp[e] * norm;
        im[q] = tmp[runs ? e + nitems : e + 1] * norm;
    }
    return GDB_OK;
}

// ---------------------------------------------------------------------------
// S(q) with no device allocation
//
// For callers that cannot let this library call cudaMalloc: applications
// whose own allocator or fixed memory pool owns the GPU's memory, code with
// a hard device-memory budget, and call sites where allocating is not
// allowed while they run.  The caller passes device inputs and outputs; the
// only scratch (the float64 accumulators) is the file-scope array below,
// which every GPU that loads this library holds until the process exits.
// ---------------------------------------------------------------------------
#define GDB_SQ_NOALLOC_MAX_Q 65536  // q-vectors per call
#define GDB_SQ_NOALLOC_MAX_N 48     // largest |n| component (shared table 32 x 291 float2 = 74.5 KB)
#define SQNA_TAIL (2 * GDB_SQ_NOALLOC_MAX_Q)

// [0, 2 nq): (re, im) accumulators; [TAIL]: sum of form factors; [TAIL+1]:
// 1.0 when an n-vector component is outside [-n_max, n_max].  Shared by all
// calls on a device: calls that overlap on the GPU race on it.
static __device__ __align__(256) double g_sq_scratch[SQNA_TAIL + 32];

namespace {

std::mutex g_sq_scratch_mu;
double *g_sq_scratch_addr[256] = {nullptr};

// Device address of g_sq_scratch on the current device, looked up once per
// device (host code cannot use the symbol itself as a device address).
int sq_scratch_address(int dev, double **out) {
    std::lock_guard<std::mutex> lock(g_sq_scratch_mu);
    if (dev < 0 || dev >= 256) return GDB_ERR_ARG;
    if (!g_sq_scratch_addr[dev]) {
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, g_sq_scratch) != cudaSuccess || !p) return GDB_ERR_CUDA;
        g_sq_scratch_addr[dev] = (double *)p;
    }
    *out = g_sq_scratch_addr[dev];
    return GDB_OK;
}

__global__ void k_sqna_clear(double *s, int nq) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < 2 * nq; k += gridDim.x * blockDim.x) s[k] = 0.0;
    if (blockIdx.x == 0 && threadIdx.x < 2) s[SQNA_TAIL + threadIdx.x] = 0.0;
}

__global__ void k_sqna_weight_sum(const float *ff, int n, double *s) {
    __shared__ double sm[32];
    double v = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) v += ff ? ff[i] : 1.0;
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
        double w = threadIdx.x < (blockDim.x >> 5) ? sm[threadIdx.x] : 0.0;
        w = warp_sum(w);
        if (threadIdx.x == 0) atomicAdd(&s[SQNA_TAIL], w);
    }
}

// Same tabulated-phase method as k_sq; positions are the caller's (n, 3)
// float32 array, n-vector components lie in [-nmax, nmax].
__global__ void __launch_bounds__(SQ_THREADS) k_sqna(const float *__restrict__ r, const float *__restrict__ ff, int n,
                                                     const int *__restrict__ nvec, int nq, int nmax, float ilx,
                                                     float ily, float ilz, double *s) {
    extern __shared__ float2 tab[];
    __shared__ float wsh[SQ_TILE];
    const int span = 2 * nmax + 1, row = 3 * span;
    const int q = blockIdx.x * SQ_THREADS + threadIdx.x;
    bool ok = q < nq;
    int nx = 0, ny = 0, nz = 0;
    if (ok) {
        const int a = nvec[3 * q], b = nvec[3 * q + 1], c = nvec[3 * q + 2];
        if (a < -nmax || a > nmax || b < -nmax || b > nmax || c < -nmax || c > nmax) {
            s[SQNA_TAIL + 1] = 1.0;
            ok = false;
        } else {
            nx = a + nmax;
            ny = b + nmax + span;
            nz = c + nmax + 2 * span;
        }
    }
    const float il[3] = {ilx, ily, ilz};
    double sr = 0.0, si = 0.0;
    const int p_begin = blockIdx.y * SQ_CHUNK;
    const int p_end = min(n, p_begin + SQ_CHUNK);
    for (int p0 = p_begin; p0 < p_end; p0 += SQ_TILE) {
        const int np = min(SQ_TILE, p_end - p0);
        __syncthreads();
        for (int e = threadIdx.x; e < np * row; e += SQ_THREADS) {
            const int pl = e / row, col = e % row;
            const int d = col / span, k = col % span - nmax;
            const float x = r[3 * (size_t)(p0 + pl) + d];
            float sn, cs;
            sincospif(2.0f * (float)k * (x * il[d]), &sn, &cs);
            tab[pl * row + col] = make_float2(cs, sn);
        }
        if (threadIdx.x < np) wsh[threadIdx.x] = ff ? ff[p0 + threadIdx.x] : 1.0f;
        __syncthreads();
        if (ok) {
            float tr = 0.f, ti = 0.f;
            for (int pl = 0; pl < np; pl++)
                sq_term(tab[pl * row + nx], tab[pl * row + ny], tab[pl * row + nz], wsh[pl], true, tr, ti);
            sr += tr;
            si += ti;
        }
    }
    if (ok) {
        atomicAdd(&s[2 * q], sr);
        atomicAdd(&s[2 * q + 1], si);
    }
}

__global__ void k_sqna_finish(const double *s, int nq, double *re, double *im) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nq) return;
    const double norm = 1.0 / sqrt(s[SQNA_TAIL]);
    re[q] = s[2 * q] * norm;
    im[q] = s[2 * q + 1] * norm;
}

}  // namespace

extern "C" {

int gdb_sq_compute_noalloc(int n, const float *r_dev, const float *ff_dev, const float box[3], int nq,
                           const int32_t *n_vectors_dev, int n_max, double *rho_re_dev, double *rho_im_dev,
                           void *stream) {
    gdb_sim *h = nullptr;
    if (n < 1 || nq < 1 || !r_dev || !box || !n_vectors_dev || !rho_re_dev || !rho_im_dev)
        return aset(h, GDB_ERR_ARG, "gdb_sq_compute_noalloc: bad arguments");
    if (nq > GDB_SQ_NOALLOC_MAX_Q)
        return aset(h, GDB_ERR_ARG, "gdb_sq_compute_noalloc: more than 65536 q-vectors");
    if (n_max < 0 || n_max > GDB_SQ_NOALLOC_MAX_N)
        return aset(h, GDB_ERR_ARG, "gdb_sq_compute_noalloc: n_max must be in [0, 48]");
    if (!(box[0] > 0.f && box[1] > 0.f && box[2] > 0.f))
        return aset(h, GDB_ERR_ARG, "gdb_sq_compute_noalloc: non-positive box length");
    int dev = 0;
    ACK(cudaGetDevice(&dev));
    double *s = nullptr;
    int rc = sq_scratch_address(dev, &s);
    if (rc) return aset(h, rc, "gdb_sq_compute_noalloc: scratch address lookup failed");
    cudaStream_t st = (cudaStream_t)stream;
    const int span = 2 * n_max + 1;
    const size_t smem = (size_t)SQ_TILE * 3 * span * sizeof(float2);
    constexpr int most = SQ_TILE * 3 * (2 * GDB_SQ_NOALLOC_MAX_N + 1) * (int)sizeof(float2);
    ACK(cudaFuncSetAttribute(k_sqna, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    k_sqna_clear<<<(2 * nq + 255) / 256, 256, 0, st>>>(s, nq);
    k_sqna_weight_sum<<<64, 256, 0, st>>>(ff_dev, n, s);
    dim3 grid((nq + SQ_THREADS - 1) / SQ_THREADS, (n + SQ_CHUNK - 1) / SQ_CHUNK);
    k_sqna<<<grid, SQ_THREADS, smem, st>>>(r_dev, ff_dev, n, n_vectors_dev, nq, n_max, 1.0f / box[0],
                                           1.0f / box[1], 1.0f / box[2], s);
    k_sqna_finish<<<(nq + 255) / 256, 256, 0, st>>>(s, nq, rho_re_dev, rho_im_dev);
    ACK(cudaGetLastError());
    double flag = 0.0;
    ACK(cudaMemcpyAsync(&flag, s + SQNA_TAIL + 1, sizeof(double), cudaMemcpyDeviceToHost, st));
    ACK(cudaStreamSynchronize(st));
    if (flag != 0.0)
        return aset(h, GDB_ERR_ARG, "gdb_sq_compute_noalloc: an n-vector component is outside [-n_max, n_max]");
    return GDB_OK;
}

int gdb_rdf_update(gdb_sim *h, int bins, double r_max, uint64_t *out) {
    if (!h || !out) return aset(h, GDB_ERR_ARG, "gdb_rdf_update: NULL argument");
    if (!gdb_internal_uploaded(h)) return aset(h, GDB_ERR_STATE, "state not uploaded");
    ACK(cudaSetDevice(gdb_internal_dev(h)));
    return rdf_device(h, gdb_internal_stream(h), gdb_internal_pos(h), gdb_internal_n(h), gdb_internal_box(h),
                      gdb_internal_ntypes(h), bins, r_max, out);
}

int gdb_sq_update(gdb_sim *h, int nq, const int32_t *n_vectors, const float *ff, double *rho_re, double *rho_im) {
    if (!h || !n_vectors || !rho_re || !rho_im) return aset(h, GDB_ERR_ARG, "gdb_sq_update: NULL argument");
    if (!gdb_internal_uploaded(h)) return aset(h, GDB_ERR_STATE, "state not uploaded");
    ACK(cudaSetDevice(gdb_internal_dev(h)));
    return sq_device(h, gdb_internal_stream(h), gdb_internal_pos(h), gdb_internal_orig(h), gdb_internal_n(h), ff,
                     gdb_internal_box(h), nq, n_vectors, rho_re, rho_im);
}

int gdb_rdf_compute(int n, const float *r, const int32_t *ptype, const float box[3], int ntypes, int bins,
                    double r_max, uint64_t *out) {
    gdb_sim *h = nullptr;
    if (n < 1 || !r || !box || !out || ntypes < 1) return aset(h, GDB_ERR_ARG, "gdb_rdf_compute: bad arguments");
    if (ptype)
        for (int i = 0; i < n; i++)
            if (ptype[i] < 0 || ptype[i] >= ntypes) return aset(h, GDB_ERR_ARG, "gdb_rdf_compute: type out of range");
    cudaStream_t st;
    ACK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    float *dr = nullptr;
    int *dpt = nullptr, *orig = nullptr;
    float4 *pos = nullptr;
    int rc = GDB_OK;
    do {
        cudaError_t e;
        if ((e = pool_alloc(&dr, (size_t)n * 3 * sizeof(float), st)) ||
            (e = pool_alloc(&pos, (size_t)n * sizeof(float4), st)) ||
            (e = pool_alloc(&orig, (size_t)n * sizeof(int), st)) ||
            (ptype && (e = pool_alloc(&dpt, (size_t)n * sizeof(int), st))) ||
            (e = cudaMemcpyAsync(dr, r, (size_t)n * 3 * sizeof(float), cudaMemcpyHostToDevice, st)) ||
            (ptype && (e = cudaMemcpyAsync(dpt, ptype, (size_t)n * sizeof(int), cudaMemcpyHostToDevice, st)))) {
            rc = aset(h, GDB_ERR_CUDA, "gdb_rdf_compute: staging", e);
            break;
        }
        k_pack_pos<<<(n + 255) / 256, 256, 0, st>>>(n, dr, dpt, pos, orig);
        rc = rdf_device(h, st, pos, n, box, ntypes, bins, r_max, out);
    } while (0);
    if (dr) cudaFreeAsync(dr, st);
    if (pos) cudaFreeAsync(pos, st);
    if (orig) cudaFreeAsync(orig, st);
    if (dpt) cudaFreeAsync(dpt, st);
    cudaStreamSynchronize(st);
    cudaStreamDestroy(st);
    return rc;
}

int gdb_sq_compute(int n, const float *r, const float *ff, const float box[3], int nq, const int32_t *n_vectors,
                   double *rho_re, double *rho_im) {
    gdb_sim *h = nullptr;
    if (n < 1 || !r || !box || !n_vectors || !rho_re || !rho_im) return aset(h, GDB_ERR_ARG, "gdb_sq_compute: bad arguments");
    cudaStream_t st;
    ACK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    float *dr = nullptr;
    int *orig = nullptr;
    float4 *pos = nullptr;
    int rc = GDB_OK;
    do {
        cudaError_t e;
        if ((e = pool_alloc(&dr, (size_t)n * 3 * sizeof(float), st)) ||
            (e = pool_alloc(&pos, (size_t)n * sizeof(float4), st)) ||
            (e = pool_alloc(&orig, (size_t)n * sizeof(int), st)) ||
            (e = cudaMemcpyAsync(dr, r, (size_t)n * 3 * sizeof(float), cudaMemcpyHostToDevice, st))) {
            rc = aset(h, GDB_ERR_CUDA, "gdb_sq_compute: staging", e);
            break;
        }
        k_pack_pos<<<(n + 255) / 256, 256, 0, st>>>(n, dr, nullptr, pos, orig);
        rc = sq_device(h, st, pos, orig, n, ff, box, nq, n_vectors, rho_re, rho_im);
    } while (0);
    if (dr) cudaFreeAsync(dr, st);
    if (pos) cudaFreeAsync(pos, st);
    if (orig) cudaFreeAsync(orig, st);
    cudaStreamSynchronize(st);
    cudaStreamDestroy(st);
    return rc;
}

// Frames of the blocks from first_block on are uploaded in groups of whole
// blocks that fit a staging budget (1 GiB, GDB_DYN_STAGE_BYTES overrides it),
// plus one buffer with the first frame of every such block for the lags
// longer than a block; frame pairs are launched at most 65535 per grid
// (GDB_DYN_PAIR_CHUNK lowers it), the y extent of a CUDA grid.
static size_t env_size(const char *name, size_t dflt) {
    const char *v = getenv(name);
    if (!v || !*v) return dflt;
    const long long x = atoll(v);
    return x > 0 ? (size_t)x : dflt;
}

static cudaError_t dyn_launch(cudaStream_t st, int gx, const float *frames, int n, const int *dpt, int nt,
                              const float *box, const int2 *dpairs, const double *dq, double *dacc, int count,
                              int chunk) {
    for (int off = 0; off < count; off += chunk) {
        const int c = std::min(chunk, count - off);
        k_dynamics<<<dim3(gx, c), DYN_THREADS, 0, st>>>(frames, n, dpt, nt, box[0], box[1], box[2], dpairs + off, dq,
                                                        dacc + (size_t)off * nt * 3);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

int gdb_calc_dynamics(int num_blocks, int conf_per_block, int n, const float *frames, const int32_t *ptype,
                      int ntypes, const float box[3], int first_block, const double *qvalues, int total_times,
                      double *msd, double *m4d, double *fs, int32_t *count) {
    gdb_sim *h = nullptr;
    if (num_blocks < 1 || conf_per_block < 1 || n < 1 || !frames || !ptype || !box || !qvalues || !msd || !m4d ||
        !fs || !count || ntypes < 1)
        return aset(h, GDB_ERR_ARG, "gdb_calc_dynamics: bad arguments");
    if (ntypes > DYN_MAX_TYPES) return aset(h, GDB_ERR_ARG, "gdb_calc_dynamics: more than 8 particle types");
    if (first_block < 0 || first_block >= num_blocks)
        return aset(h, GDB_ERR_ARG, "gdb_calc_dynamics: first_block outside [0, num_blocks)");
    int extra = 0;  // int(log2(num_blocks - first_block)) - 1
    while ((2 << extra) <= num_blocks - first_block) extra++;
    extra -= 1;
    if (extra < 0)  // the reference indexes past its arrays there
        return aset(h, GDB_ERR_ARG, "gdb_calc_dynamics: needs at least two blocks from first_block on");
    if (total_times != conf_per_block - 1 + extra)
        return aset(h, GDB_ERR_ARG, "gdb_calc_dynamics: total_times must be conf_per_block - 1 + log2 term");
    std::vector<int> nper(ntypes, 0);
    for (int i = 0; i < n; i++) {
        if (ptype[i] < 0 || ptype[i] >= ntypes) return aset(h, GDB_ERR_ARG, "gdb_calc_dynamics: type out of range");
        nper[ptype[i]]++;
    }
    const int fb = first_block, nblk = num_blocks - first_block, cpb = conf_per_block;
    const size_t frame_floats = (size_t)2 * n * 3;
    const size_t block_bytes = (size_t)cpb * frame_floats * sizeof(float);
    const int group = (int)std::max<size_t>(1, std::min<size_t>(nblk, env_size("GDB_DYN_STAGE_BYTES", 1ull << 30) /
                                                                       block_bytes));
    const int chunk = (int)std::min<size_t>(65535, env_size("GDB_DYN_PAIR_CHUNK", 65535));
    // frame pairs in the reference's loop order (calc_dynamics.py:50-63),
    // as indices into the staging buffers: within-block lags into the
    // group's buffer, longer lags into the buffer of first frames
    std::vector<int2> pairs;
    std::vector<int> tindex;
    for (int k = 0; k < total_times; k++) count[k] = 0;
    for (int b = fb; b < num_blocks; b++) {
        const int base = ((b - fb) % group) * cpb;
        for (int i = 0; i < cpb - 1; i++) {
            count[i]++;
            pairs.push_back(make_int2(base + i + 1, base));
            tindex.push_back(i);
        }
    }
    const int np_in = (int)pairs.size();
    for (int b = fb; b < num_blocks; b++)
        for (int i = 0; i < extra; i++) {
            const int other = b + (2 << i);
            if (other < num_blocks) {
                count[cpb - 1 + i]++;
                pairs.push_back(make_int2(other - fb, b - fb));
                tindex.push_back(cpb - 1 + i);
            }
        }
    const int np_ = (int)pairs.size();
    for (int k = 0; k < total_times * ntypes; k++) msd[k] = m4d[k] = fs[k] = 0.0;
    cudaStream_t st;
    ACK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    float *dgroup = nullptr, *dfirst = nullptr;
    int *dpt = nullptr;
    int2 *dpairs = nullptr;
    double *dq = nullptr, *dacc = nullptr;
    std::vector<double> acc((size_t)std::max(np_, 1) * ntypes * 3);
    int rc = GDB_OK;
    do {
        cudaError_t e;
        if ((e = pool_alloc(&dgroup, (size_t)group * block_bytes, st)) ||
            (e = pool_alloc(&dfirst, (size_t)nblk * frame_floats * sizeof(float), st)) ||
            (e = pool_alloc(&dpt, (size_t)n * sizeof(int), st)) ||
            (e = pool_alloc(&dpairs, (size_t)std::max(np_, 1) * sizeof(int2), st)) ||
            (e = pool_alloc(&dq, (size_t)ntypes * sizeof(double), st)) ||
            (e = pool_alloc(&dacc, acc.size() * sizeof(double), st)) ||
            (e = cudaMemcpyAsync(dpt, ptype, (size_t)n * sizeof(int), cudaMemcpyHostToDevice, st)) ||
            (e = cudaMemcpyAsync(dpairs, pairs.data(), (size_t)np_ * sizeof(int2), cudaMemcpyHostToDevice, st)) ||
            (e = cudaMemcpyAsync(dq, qvalues, (size_t)ntypes * sizeof(double), cudaMemcpyHostToDevice, st)) ||
            (e = cudaMemsetAsync(dacc, 0, acc.size() * sizeof(double), st))) {
            rc = aset(h, GDB_ERR_CUDA, "gdb_calc_dynamics: staging", e);
            break;
        }
        const int gx = std::min((n + DYN_THREADS - 1) / DYN_THREADS, 64);
        // lags within a block, one group of blocks at a time (stream order
        // keeps a group's kernels ahead of the next group's upload)
        for (int g0 = 0; g0 < nblk && !e; g0 += group) {
            const int gb = std::min(group, nblk - g0);
            const float *src = frames + (size_t)(fb + g0) * cpb * frame_floats;
            if ((e = cudaMemcpyAsync(dgroup, src, (size_t)gb * block_bytes, cudaMemcpyHostToDevice, st))) break;
            for (int b = 0; b < gb && !e; b++) {
                const float *f0 = src + (size_t)b * cpb * frame_floats;
                e = cudaMemcpyAsync(dfirst + (size_t)(g0 + b) * frame_floats, f0, frame_floats * sizeof(float),
                                    cudaMemcpyHostToDevice, st);
            }
            if (e) break;
            const int p0 = g0 * (cpb - 1), pc = gb * (cpb - 1);
            e = dyn_launch(st, gx, dgroup, n, dpt, ntypes, box, dpairs + p0, dq, dacc + (size_t)p0 * ntypes * 3, pc,
                           chunk);
        }
        // lags of whole blocks, between first frames
        if (!e && np_ > np_in)
            e = dyn_launch(st, gx, dfirst, n, dpt, ntypes, box, dpairs + np_in, dq,
                           dacc + (size_t)np_in * ntypes * 3, np_ - np_in, chunk);
        if (e || (e = cudaMemcpyAsync(acc.data(), dacc, acc.size() * sizeof(double), cudaMemcpyDeviceToHost, st)) ||
            (e = cudaStreamSynchronize(st))) {
            rc = aset(h, GDB_ERR_CUDA, "gdb_calc_dynamics: kernel", e);
            break;
        }
        // per pair and type: the means over the type's particles (and, for
        // Fs, components) added at the pair's time index, then / count; a
        // type without particles is NaN, as numpy's mean of an empty array
        for (int p = 0; p < np_; p++)
            for (int t = 0; t < ntypes; t++) {
                if (nper[t] == 0) continue;
                const double *a = &acc[((size_t)p * ntypes + t) * 3];
                const size_t o = (size_t)tindex[p] * ntypes + t;
                msd[o] += a[0] / nper[t];
                m4d[o] += a[1] / nper[t];
                fs[o] += a[2] / (3.0 * nper[t]);
            }
        for (int k = 0; k < total_times; k++)
            for (int t = 0; t < ntypes; t++) {
                const size_t o = (size_t)k * ntypes + t;
                if (nper[t] == 0) {
                    msd[o] = m4d[o] = fs[o] = NAN;
                    continue;
                }
                msd[o] /= count[k];
                m4d[o] /= count[k];
                fs[o] /= count[k];
            }
    } while (0);
    if (dgroup) cudaFreeAsync(dgroup, st);
    if (dfirst) cudaFreeAsync(dfirst, st);
    if (dpt) cudaFreeAsync(dpt, st);
    if (dpairs) cudaFreeAsync(dpairs, st);
    if (dq) cudaFreeAsync(dq, st);
    if (dacc) cudaFreeAsync(dacc, st);
    cudaStreamSynchronize(st);
    cudaStreamDestroy(st);
    return rc;
}

}  // extern "C"
