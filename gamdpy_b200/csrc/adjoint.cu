// adjoint.cu -- gradients of trajectory-averaged observables of an NVE
// leapfrog trajectory with respect to the Lennard-Jones pair parameters
// (sigma_ab, epsilon_ab), by a hand-written discrete adjoint.
//
// Forward (float32 state, float64 reductions), as integrators/NVE.py:78-97
// with the shifted-force LJ of LJ_12_6_sigma_epsilon.py:26-36 and
// apply_shifted_force_cutoff.py:30-37 (s -= s(rc), u += s(rc) rc (r - rc) - u(rc)):
//   f_n     = F(r_n)                       pair sum over the list
//   v_{n+1} = v_n + f_n dt / m
//   r_{n+1} = r_n + v_{n+1} dt             (periodic wrap; derivative identity)
//   U_n, W_n from r_n; K_n = sum m ((v_n + v_{n+1}) / 2)^2 / 2
//   g_b     = soft (Gaussian-kernel) A-A radial distribution on sampled steps
// Observables: time averages <U>, <W>, <K> over n = 0..T-1 and <g_b>.
//
// Backward: reverse sweep over the steps with the cotangents (R, V) of
// (r_{n+1}, v_{n+1}):
//   Vt   = V + dt R + gK dK_n/dv_{n+1}
//   R   <- R + (dt / m) J(r_n)^T Vt + gU dU_n/dr + gW dW_n/dr + sum_b gG_b dg_b/dr
//   V   <- Vt + gK dK_n/dv_n
//   dL/dtheta += (dt / m) (df/dtheta)^T Vt + gU dU_n/dtheta + gW dW_n/dtheta
// J^T Vt is the Hessian-vector product of the pair potential: for each pair
// (s I + s'/r d d^T)(Vt_i - Vt_j).  The states the sweep needs are all kept
// while they fit ADJ_KEEP_BYTES; beyond that the forward keeps checkpoints of
// (r, v) every `checkpoint_every` steps and the backward recomputes each
// segment's states from its checkpoint with the same kernel (bit-identical)
// before sweeping it in reverse, in float64.
//
// Forward and sweep are one cooperative kernel each, one warp per particle
// and one grid barrier per step; every sum over the steps stays with its warp
// until the kernel ends.
//
// Pairs come from a neighbour list (all j within the pair's cut plus a skin of
// 0.5, and, apart, the other type-0 pairs within the RDF kernel's reach plus
// the skin; built N^2 by the warp that uses it, so a rebuild costs no barrier;
// rebuilt when a particle moves more than half the skin); 32 lanes per
// particle, lane L taking its column of the list, the neighbours j = L (mod
// 32) in ascending order.  Every per-lane sum of the forward is then the same
// as a loop over all j (the NbList2 pair set), whatever the list holds beyond
// the cutoff: results do not depend on when the list was built, so recomputed
// segments are bit-identical to the forward.  Every sum has a fixed order, so
// runs are reproducible.  Sized for the small systems this is meant for (N of
// a few thousand; the build is N^2).
#include <cuda_runtime.h>
#include <math.h>
#include <stdarg.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "../../include/gamdb200.h"
#include "gdb_internal.cuh"

using namespace gdb;

namespace {

constexpr int ADJ_MAXT = 4;     // particle types
constexpr int ADJ_MAXB = 128;   // RDF bins
constexpr int ADJ_LANES = 32;   // lanes per particle: a warp
// Most warps per block (72 registers a thread): one block per SM, 4144 particles
// in flight on 148 SMs.  One more takes a second turn every step (50 steps,
// observables and gradient: N 4144 1.90 ms, 4145 2.11, 4200 2.51, 8288 3.01).
constexpr int ADJ_WARPS = 28;
constexpr size_t ADJ_KEEP_BYTES = (size_t)1 << 30;  // states kept instead of checkpoints up to this (GDB_ADJ_KEEP_BYTES)
constexpr int ADJ_NTH = 2 * ADJ_MAXT * ADJ_MAXT;  // d/dsigma, d/depsilon per ordered type pair
constexpr double ADJ_FIX = 4294967296.0;          // fixed-point scale of the RDF kernel sums
constexpr double ADJ_KW = 8.0;                    // kernel support in widths (exp(-32): smooth to 1e-14)

// float32 pair entry, the same arithmetic as the plain kernels' PairEntry
struct Tab32 {
    float c, cu12, cu6, cs12, cs6, uc, sc, sccut, cut, cut2;
};
// float64 parameters and cutoff values for the backward sweep
struct Tab64 {
    double sig2, eps, ieps, eps_sig;  // sigma^2, epsilon, 1 / epsilon, epsilon / sigma
    double cut;
    double s_c;    // s0(rc)
    double dsds_c; // d s0 / d sigma at rc
    double u_c;    // u0(rc)
    double duds_c; // d u0 / d sigma at rc
    float cut2;    // the forward's cutoff test
    float reach2;  // (cut + skin)^2: the list
};

struct Tables {
    int nt;
    Tab32 t32[ADJ_MAXT * ADJ_MAXT];
    Tab64 t64[ADJ_MAXT * ADJ_MAXT];
};

// Grid barrier words, zero at a launch.
struct AdjBar {
    unsigned cnt[3];  // arrivals, by barrier index mod 3
    int abort;
};

struct AdjArgs {
    int n, nt;
    float Lx, Ly, Lz;
    float dt;
    const float *mass;
    int nbins;
    float r_lo, dr, width;  // bin centres r_lo + (b + 1/2) dr
    double step_ratio;      // exp(-dr^2 / width^2)
    // neighbour list: particle i's maxnb entries at nbl + i * maxnb as 32
    // columns of maxnb / 32 rows (row c of column L at c * 32 + L, the
    // neighbours j = L (mod 32)).  From row 0 up, ascending: the pairs within
    // cut_ab + skin at the build; from the last row down: the other type-0
    // pairs within the RDF kernel's reach + skin.  nbc: each column's two
    // counts, the second in the high half.  Rebuilt when a particle moves more
    // than skin/2.
    int *nbl, *nbc;
    int maxnb;
    float far2;     // (RDF reach + skin)^2, 0 without RDF bins
    float any2;     // the largest of the reaches + skin, squared
    float move2;    // (skin / 2 - margin)^2
    float4 *rref;   // positions at the last build
    AdjBar *bar;
    unsigned *status;
};

constexpr float ADJ_SKIN = 0.5f;
constexpr unsigned ADJ_STATUS_OVERFLOW = 1u;
constexpr unsigned ADJ_STATUS_TIMEOUT = 2u;

__device__ __forceinline__ float mic_rint(float d, float L, float iL) { return d - L * rintf(d * iL); }

template <typename T>
__device__ __forceinline__ T wsum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Barrier of the cooperative grid with a flag (a particle of some block has
// moved beyond skin/2).  Arrivals count in the low 20 bits of one of three
// words, flags in the high bits; a block leaves when the count reaches the
// grid.  Block 0 then clears the word of barrier seq + 2: every block has left
// barrier seq - 1, and block 0's next arrival orders the clear before any
// arrival there.  A wait of about a second of SM clock gives up, sets the
// status bit and `abort`; callers return when it fails.
constexpr unsigned ADJ_FLAG_ONE = 1u << 20;
__device__ __forceinline__ bool adj_barrier(const AdjArgs &a, unsigned seq, bool flag, int *any) {
    __shared__ int s_ok;
    const int raised_here = __syncthreads_or(flag);
    if (threadIdx.x == 0) {
        AdjBar *bar = a.bar;
        int ok = *(volatile int *)&bar->abort == 0;
        if (ok) {
            unsigned *cnt = &bar->cnt[seq % 3u];
            const unsigned inc = 1u | (raised_here ? ADJ_FLAG_ONE : 0u);
            unsigned v;
            asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;" : "=r"(v) : "l"(cnt), "r"(inc) : "memory");
            v += inc;
            const long long t0 = clock64();
            int polls = 0;
            while ((v & (ADJ_FLAG_ONE - 1u)) != gridDim.x) {
                if (*(volatile int *)&bar->abort) {
                    ok = 0;
                    break;
                }
                if ((++polls & 63) == 0 && clock64() - t0 > 2000000000LL) {
                    atomicOr(a.status, ADJ_STATUS_TIMEOUT);
                    *(volatile int *)&bar->abort = 1;
                    ok = 0;
                    break;
                }
                if (polls > 64) __nanosleep(32);
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(cnt) : "memory");
            }
            *any = (v >> 20) != 0u;
            if (ok && blockIdx.x == 0) *(volatile unsigned *)&bar->cnt[(seq + 2u) % 3u] = 0u;
        }
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

__device__ __forceinline__ int type_of(float4 p) { return __float_as_int(p.w); }

// The warp's list of particle i at positions pos (AdjArgs::nbl); lane L tests
// j = L, L + 32, ... and writes its own column, which only it reads.  Four
// candidates' loads in flight, the minimum image without the rounding
// instruction (an eighth of an add's rate), and one compare for the candidates
// beyond every reach; the type pair's cutoff only for the others.  With a
// rintf a component and a look at the cutoffs for every candidate the forward
// of N 60 000 took 37.0 ms for 40 steps (20.8 with builds as kernels of their
// own) and takes 17.3; N 4096 0.62 and 0.52.
__device__ __forceinline__ void build_list(const AdjArgs &a, const Tab64 *tab, int nt, const float4 *pos, int i,
                                           float4 pi, int lane) {
    constexpr float RINT = 12582912.0f;  // 1.5 2^23: rint by adding and subtracting it
    const f32x2 mxy = pack2(-pi.x, -pi.y), ilxy = pack2(1.0f / a.Lx, 1.0f / a.Ly), nlxy = pack2(-a.Lx, -a.Ly);
    const float ilz = 1.0f / a.Lz;
    const int n = a.n, rows = a.maxnb / ADJ_LANES, ti = type_of(pi);
    const float any2 = a.any2, far2 = ti == 0 ? a.far2 : 0.f;
    int *col = a.nbl + (size_t)i * a.maxnb + lane;
    int near = 0, far = 0;
    for (int j0 = lane; j0 < n; j0 += 4 * ADJ_LANES) {
        float4 p[4];
#pragma unroll
        for (int q = 0; q < 4; q++) p[q] = pos[min(j0 + q * ADJ_LANES, n - 1)];
        float d2[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            f32x2 dxy = add2(pack2(p[q].x, p[q].y), mxy);
            float dz = p[q].z - pi.z;
            dxy = fma2(add2(fma2(dxy, ilxy, pack2(RINT, RINT)), pack2(-RINT, -RINT)), nlxy, dxy);
            dz = __fmaf_rn(__fsub_rn(__fmaf_rn(dz, ilz, RINT), RINT), -a.Lz, dz);
            float dx, dy;
            unpack2(dxy, dx, dy);
            d2[q] = dx * dx + dy * dy + dz * dz;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int j = j0 + q * ADJ_LANES;
            if (!(d2[q] < any2) || j >= n || j == i) continue;
            const int tj = type_of(p[q]);
            if (d2[q] < tab[ti * nt + tj].reach2) {
                if (near + far < rows) col[near * ADJ_LANES] = j;
                near++;
            } else if (tj == 0 && d2[q] < far2) {
                if (near + far < rows) col[(rows - 1 - far) * ADJ_LANES] = j;
                far++;
            }
        }
    }
    if (near + far > rows) {
        atomicOr(a.status, ADJ_STATUS_OVERFLOW);
        near = min(near, rows);
        far = min(far, rows - near);
    }
    a.nbc[(size_t)i * ADJ_LANES + lane] = near | (far << 16);
    if (lane == 0) a.rref[i] = pi;
}

__device__ __forceinline__ bool moved_far(const AdjArgs &a, float4 p, float4 q) {
    const float ex = mic_rint(p.x - q.x, a.Lx, 1.0f / a.Lx), ey = mic_rint(p.y - q.y, a.Ly, 1.0f / a.Ly),
                ez = mic_rint(p.z - q.z, a.Lz, 1.0f / a.Lz);
    return ex * ex + ey * ey + ez * ez > a.move2;
}

// Gaussian bins around distance r: calls f(b, x, exp(-x^2 / (2 w^2))) for
// every bin b within the kernel's support, x = r - centre_b.  From one bin to
// the next the exponent grows by (2 x dr - dr^2) / (2 w^2): two exponentials
// for the first bin, two products for each further one.  The products' errors
// add up along the bins: against exact values at most 5e-14 of a bin's value
// over 16 bins, 1.6e-13 over 64 and 5e-13 over the 128 that there can be, where
// an exponential each has 4e-15 (the forward then rounds a term to 2^-32, and
// both take r from float32 coordinates).  Bins wider than four widths take one
// exponential each.
template <typename F>
__device__ __forceinline__ void rdf_bins(const AdjArgs &a, double r, F f) {
    const double w = a.width, dr = a.dr, iw2 = 0.5 / (w * w);
    int b0 = (int)floor((r - ADJ_KW * w - a.r_lo) / dr);
    int b1 = (int)floor((r + ADJ_KW * w - a.r_lo) / dr);
    b0 = max(b0, 0);
    b1 = min(b1, a.nbins - 1);
    double x = r - ((double)a.r_lo + (b0 + 0.5) * dr);
    double e = exp(-x * x * iw2);
    if (dr <= 4.0 * w) {
        double g = exp((2.0 * x * dr - dr * dr) * iw2);
        const double k = a.step_ratio;
        for (int b = b0; b <= b1; b++) {
            f(b, x, e);
            x -= dr;
            e *= g;
            g *= k;
        }
    } else {
        for (int b = b0; b <= b1; b++) {
            x = r - ((double)a.r_lo + (b + 0.5) * dr);
            f(b, x, exp(-x * x * iw2));
        }
    }
}

// The states of a run of steps: state k at p + ((k - k0) % mod) * n.
struct States {
    float4 *p, *v;
    int k0, mod;
    __device__ __forceinline__ size_t at(int k, int n) const { return (size_t)((k - k0) % mod) * n; }
};

// Forward: steps [s0, s0 + nsteps) from state s0, one warp per particle.
// acc (observables wanted): float64 sums of U, W, K per block into acc[block][3]
// and, on sampled steps, the A-A kernel sums into gbins (fixed point, integer
// atomics: order-independent).
//
// A step is a serial chain: list chunk, position gathers, warp sums, the new
// position, the grid barrier.  Measured on B200, KA N 4096, 50 steps with 40
// RDF bins sampled every 10: 0.8 ms, and observables and gradient together
// 1.96 ms, against 7.35 ms with eight launches a step (gated N^2 rebuild
// kernels, segments recomputed from checkpoints).
struct ForwardArgs {
    States st;
    int s0, nsteps;
    double *acc;
    unsigned long long *gbins;
    int rdf_every, copies;  // copies of the bins in shared memory, 32 columns each
    float4 *ck_pos, *ck_vel;
    int ckpt;
};
__global__ void __launch_bounds__(ADJ_WARPS * 32, 1) k_adj_forward(AdjArgs a, const __grid_constant__ Tables tab,
                                                                   ForwardArgs f) {
    extern __shared__ unsigned long long s_bins[];  // [copies][nbins][32]
    __shared__ Tab32 s_tab[ADJ_MAXT * ADJ_MAXT];
    __shared__ Tab64 s_tab64[ADJ_MAXT * ADJ_MAXT];
    __shared__ double s_red[ADJ_WARPS][3];
    __shared__ int s_any;
    const int nt = tab.nt;
    for (int t = threadIdx.x; t < nt * nt; t += blockDim.x) {
        s_tab[t] = tab.t32[t];
        s_tab64[t] = tab.t64[t];
    }
    const bool bins = f.gbins != nullptr;
    if (bins)
        for (int b = threadIdx.x; b < f.copies * a.nbins * 32; b += blockDim.x) s_bins[b] = 0ull;
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    const int first = blockIdx.x * wpb + w, nwarps = gridDim.x * wpb;
    const float iLx = 1.0f / a.Lx, iLy = 1.0f / a.Ly, iLz = 1.0f / a.Lz;
    const int rows = a.maxnb / ADJ_LANES;
    double sum_u = 0.0, sum_w = 0.0, sum_k = 0.0;  // lane 0: of the warp's particles, all steps
    for (int s = 0; s < f.nsteps; s++) {
        const int step = f.s0 + s;
        const float4 *pos_in = f.st.p + f.st.at(step, a.n), *vel_in = f.st.v + f.st.at(step, a.n);
        float4 *pos_out = f.st.p + f.st.at(step + 1, a.n), *vel_out = f.st.v + f.st.at(step + 1, a.n);
        const bool rebuild = s == 0 || s_any != 0;
        const bool rdf = bins && step % f.rdf_every == 0;
        bool moved = false;
        for (int i = first; i < a.n; i += nwarps) {
            const float4 pi = pos_in[i];
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            float m = 1.f;
            if (lane == 0) {
                v = vel_in[i];
                m = a.mass[i];
            }
            const int ti = type_of(pi);
            if (rebuild) build_list(a, s_tab64, nt, pos_in, i, pi, lane);
            const Tab32 *row = s_tab + ti * nt;
            const int *lst = a.nbl + (size_t)i * a.maxnb + lane;
            const int both = a.nbc[(size_t)i * ADJ_LANES + lane];
            const int cnt = both & 0xffff;
            float fx = 0.f, fy = 0.f, fz = 0.f, u = 0.f, wv = 0.f;
            // four entries' loads in flight; the sums in ascending j
            for (int c0 = 0; c0 < cnt; c0 += 4) {
                int j[4];
                float4 p[4];
#pragma unroll
                for (int k = 0; k < 4; k++) j[k] = c0 + k < cnt ? lst[(c0 + k) * ADJ_LANES] : i;
#pragma unroll
                for (int k = 0; k < 4; k++) p[k] = pos_in[j[k]];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    if (c0 + k >= cnt) break;
                    const float dx = mic_rint(p[k].x - pi.x, a.Lx, iLx);
                    const float dy = mic_rint(p[k].y - pi.y, a.Ly, iLy);
                    const float dz = mic_rint(p[k].z - pi.z, a.Lz, iLz);
                    const float d2 = dx * dx + dy * dy + dz * dz;
                    const Tab32 &e = row[type_of(p[k])];
                    if (d2 < e.cut2) {
                        const float inv2 = 1.0f / d2;
                        const float x2 = e.c * inv2;
                        const float x6 = x2 * x2 * x2;
                        const float x12 = x6 * x6;
                        const float sp = (e.cs12 * x12 + e.cs6 * x6) * inv2 - e.sc;
                        fx -= dx * sp;
                        fy -= dy * sp;
                        fz -= dz * sp;
                        const float r = sqrtf(d2);
                        u += 0.5f * (e.cu12 * x12 + e.cu6 * x6 - e.uc + e.sccut * (r - e.cut));
                        wv += d2 * sp * (1.0f / 6.0f);
                    }
                }
            }
            if (rdf && ti == 0) {
                const double rg_lo = (double)a.r_lo - ADJ_KW * a.width,
                             rg_hi = (double)a.r_lo + a.nbins * (double)a.dr + ADJ_KW * a.width;
                const double kn = ADJ_FIX / (sqrt(2.0 * M_PI) * (double)a.width);
                unsigned long long *mine = s_bins + (size_t)(w % f.copies) * a.nbins * 32 + lane;
                const int all = cnt + (both >> 16);
                for (int c = 0; c < all; c++) {
                    const int j = lst[(c < cnt ? c : rows - 1 - (c - cnt)) * ADJ_LANES];
                    const float4 p = pos_in[j];
                    if (type_of(p) != 0) continue;
                    const float dx = mic_rint(p.x - pi.x, a.Lx, iLx);
                    const float dy = mic_rint(p.y - pi.y, a.Ly, iLy);
                    const float dz = mic_rint(p.z - pi.z, a.Lz, iLz);
                    const double r = sqrt((double)(dx * dx + dy * dy + dz * dz));
                    if (r > rg_lo && r < rg_hi)
                        rdf_bins(a, r, [&](int b, double, double e) {
                            atomicAdd(&mine[b * 32], (unsigned long long)(kn * e + 0.5));
                        });
                }
                __syncwarp();
            }
            fx = wsum(fx);
            fy = wsum(fy);
            fz = wsum(fz);
            u = wsum(u);
            wv = wsum(wv);
            if (lane == 0) {
                float vv[3] = {v.x, v.y, v.z};
                float r[3] = {pi.x, pi.y, pi.z};
                const float ff[3] = {fx, fy, fz};
                const float L[3] = {a.Lx, a.Ly, a.Lz};
                float k = 0.f;
#pragma unroll
                for (int c = 0; c < 3; c++) {  // integrators/NVE.py:78-97
                    float vm = vv[c];
                    vv[c] += ff[c] / m * a.dt;
                    vm += vv[c];
                    vm *= 0.5f;
                    k += 0.5f * m * vm * vm;
                    r[c] += vv[c] * a.dt;
                    if (r[c] * 2.0f > L[c]) r[c] -= L[c];
                    if (r[c] * 2.0f < -L[c]) r[c] += L[c];
                }
                if (f.ck_pos && step % f.ckpt == 0) {
                    const size_t o = (size_t)(step / f.ckpt) * a.n + i;
                    f.ck_pos[o] = pi;
                    f.ck_vel[o] = v;
                }
                const float4 pn = make_float4(r[0], r[1], r[2], pi.w);
                pos_out[i] = pn;
                vel_out[i] = make_float4(vv[0], vv[1], vv[2], 0.f);
                moved |= moved_far(a, pn, a.rref[i]);
                sum_u += u;
                sum_w += wv;
                sum_k += k;
            }
        }
        if (s + 1 < f.nsteps && !adj_barrier(a, (unsigned)s, moved, &s_any)) return;
    }
    if (!f.acc) return;
    if (lane == 0) {
        s_red[w][0] = sum_u;
        s_red[w][1] = sum_w;
        s_red[w][2] = sum_k;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        double t = 0.0;
        for (int k = 0; k < wpb; k++) t += s_red[k][threadIdx.x];
        f.acc[(size_t)blockIdx.x * 3 + threadIdx.x] = t;
    }
    if (bins)
        for (int b = threadIdx.x; b < a.nbins; b += blockDim.x) {
            unsigned long long t = 0ull;
            for (int c = 0; c < f.copies; c++)
                for (int l = 0; l < 32; l++) t += s_bins[((size_t)c * a.nbins + b) * 32 + l];
            if (t) atomicAdd(&f.gbins[b], t);
        }
}

// Reverse sweep over the steps s0 + len - 1 .. s0, one warp per particle.
// Per step: R += (dt/m) HVP(Vt) + gU dU/dr + gW dW/dr + dG/dr, V = Vt + gK
// dK_n/dv_n, parameter cotangents added to the warp's sums; then, for the step
// before, Vt = V + dt R + gK dK/dv and the kick's cotangent U = (dt / m) Vt,
// which the other particles read after the barrier (double-buffered by step
// parity).  Between the steps of a sweep V holds Vt.
struct SweepArgs {
    States st;
    int s0, len;
    double gU, gW, gK;
    const double *gG;  // 2 grad_g_b norm_b (-1 / w^2) kn by bin, NULL without RDF cotangents
    int rdf_every, window;
    double *R, *V;
    double4 *U;       // 2 n
    // parameter cotangents: the warps' running sums between the segments of a
    // sweep (the same additions in the same order however it is cut), then
    // the blocks' sums of the last one
    double *th_warp;  // [blocks][warps][ADJ_NTH]
    double *th_part;  // [blocks][ADJ_NTH]
    int first_segment, last_segment;
};
// Pairs inside the cutoff wait here until 32 of them are pending, so that
// the float64 derivatives run with every lane busy (a column holds about 1.5
// pairs beyond the cutoff for each inside it, and the columns' lengths differ).
// A warp's ring takes a round's hits beside 31 pending ones.  Measured on
// B200, KA N 4096, 50 steps: the sweep takes 1.0 ms.
constexpr int ADJ_RING = 64;
constexpr size_t ADJ_RING_BYTES = ADJ_RING * sizeof(float4);  // displacement r_j - r_i, and j << 2 | t_j

// LONG: columns may hold more than 64 rows (where they cannot, the test of it
// in every round cost 1.4 % of observables and gradient at KA N 4096).
template <int NT, bool LONG>
__global__ void __launch_bounds__(ADJ_WARPS * 32, 1) k_adj_sweep(AdjArgs a, const __grid_constant__ Tables tab,
                                                                 SweepArgs f) {
    __shared__ Tab64 s_tab[ADJ_MAXT * ADJ_MAXT];
    __shared__ double s_th[ADJ_WARPS][ADJ_NTH];
    __shared__ double s_gG[ADJ_MAXB];
    extern __shared__ float4 s_ring[];  // [warps][ADJ_RING]
    __shared__ int s_any;
    const int nt = tab.nt;
    for (int t = threadIdx.x; t < nt * nt; t += blockDim.x) s_tab[t] = tab.t64[t];
    const int nth = (int)(blockDim.x >> 5) * ADJ_NTH;
    double *th_state = f.th_warp + (size_t)blockIdx.x * nth;
    for (int t = threadIdx.x; t < nth; t += blockDim.x) (&s_th[0][0])[t] = f.first_segment ? 0.0 : th_state[t];
    if (f.gG)
        for (int b = threadIdx.x; b < a.nbins; b += blockDim.x) s_gG[b] = f.gG[b];
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    const int first = blockIdx.x * wpb + w, nwarps = gridDim.x * wpb;
    const float iLx = 1.0f / a.Lx, iLy = 1.0f / a.Ly, iLz = 1.0f / a.Lz;
    const unsigned below = (1u << lane) - 1u;
    const int rows = a.maxnb / ADJ_LANES;
    const double dt = a.dt;
    float4 *ring = s_ring + w * ADJ_RING;
    // lane 0: Vt and U of step s from this particle's V and R after step s + 1
    auto start_step = [&](int s, int i, double (&R)[3], double (&V)[3]) {
        if (f.window > 0 && (s + 1) % f.window == 0) {
            // last step of a window: nothing flows back across its end
#pragma unroll
            for (int c = 0; c < 3; c++) R[c] = V[c] = 0.0;
        }
        const double m = a.mass[i];
        const float4 p = f.st.v[f.st.at(s, a.n) + i], q = f.st.v[f.st.at(s + 1, a.n) + i];
        const double pv[3] = {p.x, p.y, p.z}, qv[3] = {q.x, q.y, q.z};
#pragma unroll
        for (int c = 0; c < 3; c++) V[c] = V[c] + dt * R[c] + f.gK * m * (pv[c] + qv[c]) * 0.25;
        const double k = dt / m;
        f.U[(size_t)(s & 1) * a.n + i] = make_double4(k * V[0], k * V[1], k * V[2], 0.0);
    };
    unsigned seq = 0;
    for (int i = first; i < a.n; i += nwarps)
        if (lane == 0) {
            double R[3], V[3];
#pragma unroll
            for (int c = 0; c < 3; c++) R[c] = f.R[3 * (size_t)i + c], V[c] = f.V[3 * (size_t)i + c];
            start_step(f.s0 + f.len - 1, i, R, V);
#pragma unroll
            for (int c = 0; c < 3; c++) f.R[3 * (size_t)i + c] = R[c], f.V[3 * (size_t)i + c] = V[c];
        }
    if (!adj_barrier(a, seq++, false, &s_any)) return;
    for (int k = f.len - 1; k >= 0; k--) {
        const int s = f.s0 + k;
        const float4 *pos = f.st.p + f.st.at(s, a.n);
        const double4 *U = f.U + (size_t)(s & 1) * a.n;
        const bool rebuild = k == f.len - 1 || s_any != 0;
        const bool rdf = f.gG && f.rdf_every > 0 && s % f.rdf_every == 0;
        bool moved = false;
        for (int i = first; i < a.n; i += nwarps) {
            const float4 pi = pos[i];
            const int ti = type_of(pi);
            if (rebuild) build_list(a, s_tab, nt, pos, i, pi, lane);
            const int *lst = a.nbl + (size_t)i * a.maxnb + lane;
            const int both = a.nbc[(size_t)i * ADJ_LANES + lane];
            const int cnt = both & 0xffff;
            double R[3] = {0, 0, 0}, Vt[3];  // this particle's, on every lane
#pragma unroll
            for (int c = 0; c < 3; c++) Vt[c] = f.V[3 * (size_t)i + c];
            const double4 ui = U[i];
            const double cdt = dt / a.mass[i];
            double acc[3] = {0, 0, 0};  // J^T Vt + gU dU/dr + gW dW/dr + dG/dr
            double th[2 * NT];          // d/dsigma, d/depsilon by neighbour type
#pragma unroll
            for (int t = 0; t < 2 * NT; t++) th[t] = 0.0;
            int head = 0, tail = 0;
            auto drain = [&](int take) {
                __syncwarp();
                if (lane < take) {
                    const float4 en = ring[(head + lane) & (ADJ_RING - 1)];
                    const int code = __float_as_int(en.w), j = code >> 2, tj = code & 3;
                    const double4 uj = U[j];
                    const Tab64 &e = s_tab[ti * nt + tj];
                    // d = r_i - r_j (the forward's difference is r_j - r_i)
                    const double d[3] = {-(double)en.x, -(double)en.y, -(double)en.z};
                    const double r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
                    const double ir = rsqrt(r2), ir2 = ir * ir, r = r2 * ir;
                    const double sr2 = e.sig2 * ir2;
                    const double sr6 = sr2 * sr2 * sr2, sr12 = sr6 * sr6;
                    const double s0 = e.eps * (48.0 * sr12 - 24.0 * sr6) * ir2;
                    const double sp = s0 - e.s_c;
                    const double dsr = e.eps * (-672.0 * sr12 + 192.0 * sr6) * ir2 * ir2;  // s0'(r) / r
                    const double dv[3] = {ui.x - uj.x, ui.y - uj.y, ui.z - uj.z};
                    const double dd = d[0] * dv[0] + d[1] * dv[1] + d[2] * dv[2];
                    // along d: the HVP's second part, gU u'/r, gW (d (r2 s) / dr) / (3 r)
                    const double along = dsr * dd + f.gU * (e.s_c * e.cut * ir - s0) +
                                         f.gW * (2.0 * sp + r2 * dsr) * (1.0 / 3.0);
#pragma unroll
                    for (int c = 0; c < 3; c++) acc[c] += sp * dv[c] + along * d[c];
                    const double vd = d[0] * Vt[0] + d[1] * Vt[1] + d[2] * Vt[2];
                    const double dsde = sp * e.ieps;
                    const double dsds = e.eps_sig * (576.0 * sr12 - 144.0 * sr6) * ir2 - e.dsds_c;
                    const double usf = 4.0 * e.eps * (sr12 - sr6) - e.u_c + e.s_c * e.cut * (r - e.cut);
                    const double dude = usf * e.ieps;
                    const double duds = 4.0 * e.eps_sig * (12.0 * sr12 - 6.0 * sr6) - e.duds_c +
                                        e.dsds_c * e.cut * (r - e.cut);
                    // force term (dt/m) (df_i/dtheta) . Vt_i, f_i = sum_j s d
                    const double ks = cdt * vd + f.gW * r2 * (1.0 / 6.0);
                    const double ts = ks * dsds + f.gU * 0.5 * duds, te = ks * dsde + f.gU * 0.5 * dude;
#pragma unroll
                    for (int t = 0; t < NT; t++)
                        if (t == tj) {
                            th[2 * t] += ts;
                            th[2 * t + 1] += te;
                        }
                }
                head += take;
                __syncwarp();
            };
            // each lane's hits in its column as bits, 64 rows at a time (same
            // float32 displacement and cutoff test as the forward), then round
            // by round every lane's next hit into the ring.  A lane out of hits
            // looks further down its column within the round, so the order of
            // the sums does not depend on what the list holds beyond the
            // cutoff, nor on when it was built
            auto pair = [&](int j, float4 p, float &dx, float &dy, float &dz) {
                dx = mic_rint(p.x - pi.x, a.Lx, iLx);
                dy = mic_rint(p.y - pi.y, a.Ly, iLy);
                dz = mic_rint(p.z - pi.z, a.Lz, iLz);
                return dx * dx + dy * dy + dz * dz;
            };
            unsigned long long hits = 0ull;  // of the rows from base to next
            int base = 0, next = 0;
            auto look = [&] {
                base = next;
                next = min(cnt, base + 64);
                for (int c0 = base; c0 < next; c0 += 4) {
                    int j[4];
                    float4 p[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) j[q] = c0 + q < next ? lst[(c0 + q) * ADJ_LANES] : i;
#pragma unroll
                    for (int q = 0; q < 4; q++) p[q] = pos[j[q]];
                    unsigned bits = 0;
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        float dx, dy, dz;
                        const float d2 = pair(j[q], p[q], dx, dy, dz);
                        if (c0 + q < next && d2 < s_tab[ti * nt + type_of(p[q])].cut2) bits |= 1u << q;
                    }
                    hits |= (unsigned long long)bits << (c0 - base);
                }
            };
            look();
            for (;;) {
                if (LONG)
                    while (hits == 0ull && next < cnt) look();
                const bool hit = hits != 0ull;
                const unsigned m = __ballot_sync(0xffffffffu, hit);
                if (hit) {
                    const int j = lst[(base + __ffsll(hits) - 1) * ADJ_LANES];
                    hits &= hits - 1ull;
                    const float4 p = pos[j];
                    float dx, dy, dz;
                    pair(j, p, dx, dy, dz);
                    ring[(tail + __popc(m & below)) & (ADJ_RING - 1)] =
                        make_float4(dx, dy, dz, __int_as_float((j << 2) | type_of(p)));
                }
                tail += __popc(m);
                // a full round, or after the last hits what is left
                if (tail - head >= 32 || (m == 0u && tail > head))
                    drain(min(32, tail - head));
                else if (m == 0u)
                    break;
            }
            if (rdf && ti == 0) {
                const double rg_lo = (double)a.r_lo - ADJ_KW * a.width,
                             rg_hi = (double)a.r_lo + a.nbins * (double)a.dr + ADJ_KW * a.width;
                // the column's two lists merged: ascending j, wherever the
                // build put a pair
                int near = 0, far = 0;
                const int nfar = both >> 16;
                int jn = near < cnt ? lst[0] : a.n, jf = far < nfar ? lst[(rows - 1) * ADJ_LANES] : a.n;
                while (jn < a.n || jf < a.n) {
                    const int j = min(jn, jf);
                    if (jn < jf) {
                        near++;
                        jn = near < cnt ? lst[near * ADJ_LANES] : a.n;
                    } else {
                        far++;
                        jf = far < nfar ? lst[(rows - 1 - far) * ADJ_LANES] : a.n;
                    }
                    const float4 p = pos[j];
                    if (type_of(p) != 0) continue;
                    float dx, dy, dz;
                    pair(j, p, dx, dy, dz);
                    const double d[3] = {-(double)dx, -(double)dy, -(double)dz};
                    const double r = sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
                    if (r > rg_lo && r < rg_hi) {
                        double g = 0.0;
                        rdf_bins(a, r, [&](int b, double x, double e) { g += s_gG[b] * x * e; });
                        g /= r;
#pragma unroll
                        for (int q = 0; q < 3; q++) acc[q] += g * d[q];
                    }
                }
                __syncwarp();
            }
#pragma unroll
            for (int c = 0; c < 3; c++) acc[c] = wsum(acc[c]);
#pragma unroll
            for (int t = 0; t < NT; t++)
                if (t < nt) {
                    th[2 * t] = wsum(th[2 * t]);
                    th[2 * t + 1] = wsum(th[2 * t + 1]);
                }
            if (lane == 0) {
#pragma unroll
                for (int t = 0; t < NT; t++)
                    if (t < nt) {
                        s_th[w][2 * (ti * nt + t)] += th[2 * t];
                        s_th[w][2 * (ti * nt + t) + 1] += th[2 * t + 1];
                    }
                const double m = a.mass[i];
                const float4 va = f.st.v[f.st.at(s, a.n) + i], vb = f.st.v[f.st.at(s + 1, a.n) + i];
                const double sa[3] = {va.x, va.y, va.z}, sb[3] = {vb.x, vb.y, vb.z};
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    R[c] = f.R[3 * (size_t)i + c] + acc[c];
                    Vt[c] += f.gK * m * (sa[c] + sb[c]) * 0.25;
                }
                if (k > 0) {
                    start_step(s - 1, i, R, Vt);
                    moved |= moved_far(a, f.st.p[f.st.at(s - 1, a.n) + i], a.rref[i]);
                }
#pragma unroll
                for (int c = 0; c < 3; c++) f.R[3 * (size_t)i + c] = R[c], f.V[3 * (size_t)i + c] = Vt[c];
            }
            __syncwarp();
        }
        if (k > 0 && !adj_barrier(a, seq++, moved, &s_any)) return;
    }
    __syncthreads();
    if (!f.last_segment) {
        for (int t = threadIdx.x; t < nth; t += blockDim.x) th_state[t] = (&s_th[0][0])[t];
    } else if (threadIdx.x < ADJ_NTH) {
        double t = 0.0;
        for (int p = 0; p < wpb; p++) t += s_th[p][threadIdx.x];
        f.th_part[(size_t)blockIdx.x * ADJ_NTH + threadIdx.x] = t;
    }
}

__global__ void k_adj_pack(int n, const float *r, const float *v, const int *type, float4 *pos, float4 *vel) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    pos[i] = make_float4(r[3 * i], r[3 * i + 1], r[3 * i + 2], __int_as_float(type[i]));
    vel[i] = make_float4(v[3 * i], v[3 * i + 1], v[3 * i + 2], 0.f);
}

char g_adj_error[512] = "";

}  // namespace

struct gdb_adj {
    int n = 0, nt = 0, dev = 0;
    float box[3] = {0, 0, 0};
    float dt = 0.f;
    int steps = 0, ckpt = 50;
    int nbins = 0, rdf_every = 0;
    int window = 0;  // 0: exact adjoint; W > 0: cotangents cut every W steps
    float r_lo = 0.f, r_hi = 0.f, width = 0.f;
    bool setup = false, forward_done = false;
    Tables tab{};
    int *d_type = nullptr;
    float *d_mass = nullptr;
    bool keep_all = false;                      // every state is kept (d_seg_*), no checkpoints
    float4 *d_pos = nullptr, *d_vel = nullptr;  // two states, the forward's when it keeps checkpoints
    float4 *d_ck_pos = nullptr, *d_ck_vel = nullptr;  // checkpoints
    float4 *d_seg_pos = nullptr, *d_seg_vel = nullptr;  // every state, or one recomputed segment
    int blocks = 0, threads = 0;  // launch shape of the two kernels
    double n_type0 = 0.0;         // particles of type 0
    double *d_acc = nullptr;      // [blocks][3]
    unsigned long long *d_bins = nullptr;
    double *d_R = nullptr, *d_V = nullptr, *d_th = nullptr, *d_gG = nullptr;
    double4 *d_U = nullptr;
    int *d_nbl = nullptr, *d_nbc = nullptr;
    AdjBar *d_bar = nullptr;
    float4 *d_rref = nullptr;
    unsigned *d_status = nullptr;
    int maxnb = 0;
    float rl = 0.f;
    int nsamples = 0;
    std::vector<double> obs;
    cudaStream_t st = nullptr;
    char err[512] = "";
};

namespace {

int aset(gdb_adj *h, int code, const char *fmt, ...) {
    char *dst = h ? h->err : g_adj_error;
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(dst, 512, fmt, ap);
    va_end(ap);
    return code;
}

#define ACK(call)                                                                                          \
    do {                                                                                                   \
        cudaError_t e_ = (call);                                                                           \
        if (e_ != cudaSuccess) {                                                                           \
            (void)cudaGetLastError(); /* reported here, not again by the next launch's check */            \
            return aset(h, GDB_ERR_CUDA, "%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, \
                        __LINE__);                                                                         \
        }                                                                                                  \
    } while (0)

void adj_free(gdb_adj *h) {
    if (!h) return;
    cudaSetDevice(h->dev);
    if (h->st) cudaStreamSynchronize(h->st);
    void *ptrs[] = {h->d_type, h->d_mass, h->d_pos, h->d_vel, h->d_ck_pos, h->d_ck_vel, h->d_seg_pos, h->d_seg_vel,
                    h->d_acc, h->d_bins, h->d_R, h->d_V, h->d_U, h->d_th, h->d_gG, h->d_nbl, h->d_nbc, h->d_bar,
                    h->d_rref, h->d_status};
    for (void *p : ptrs)
        if (p) cudaFreeAsync(p, h->st);
    if (h->st) cudaStreamDestroy(h->st);
}

AdjArgs adj_args(const gdb_adj *h) {
    AdjArgs a;
    a.n = h->n;
    a.nt = h->nt;
    a.Lx = h->box[0];
    a.Ly = h->box[1];
    a.Lz = h->box[2];
    a.dt = h->dt;
    a.mass = h->d_mass;
    a.nbins = h->nbins;
    a.r_lo = h->r_lo;
    a.dr = h->nbins > 0 ? (h->r_hi - h->r_lo) / h->nbins : 1.f;
    a.width = h->width;
    a.nbl = h->d_nbl;
    a.nbc = h->d_nbc;
    a.maxnb = h->maxnb;
    const double ratio = (double)a.dr / (double)a.width;
    a.step_ratio = exp(-ratio * ratio);
    const float far = (float)((double)h->r_hi + ADJ_KW * h->width) + ADJ_SKIN;
    a.far2 = h->nbins > 0 ? far * far : 0.f;
    a.any2 = h->rl * h->rl;
    const float mv = 0.5f * ADJ_SKIN - 0.01f;
    a.move2 = mv * mv;
    a.rref = h->d_rref;
    a.bar = h->d_bar;
    a.status = h->d_status;
    return a;
}

// Shared copies of the RDF bins: at most 8, within 96 KB.
int rdf_copies(const gdb_adj *h) {
    return std::max(1, std::min(8, (int)(96 * 1024 / ((size_t)std::max(h->nbins, 1) * 32 * 8))));
}

template <bool LONG>
const void *sweep_kernel(const gdb_adj *h) {
    return h->nt == 1   ? (const void *)k_adj_sweep<1, LONG>
           : h->nt == 2 ? (const void *)k_adj_sweep<2, LONG>
                        : (const void *)k_adj_sweep<ADJ_MAXT, LONG>;
}
const void *sweep_kernel(const gdb_adj *h) {
    return h->maxnb / ADJ_LANES > 64 ? sweep_kernel<true>(h) : sweep_kernel<false>(h);
}

// One block per SM at most, of as few warps as give every particle one (more
// particles than that are taken in turn).
cudaError_t launch_shape(gdb_adj *h) {
    int sms = 0;
    cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->dev);
    if (e != cudaSuccess) return e;
    const int warps = std::min(ADJ_WARPS, (h->n + sms - 1) / sms);
    h->threads = warps * 32;
    h->blocks = std::min(sms, (h->n + warps - 1) / warps);
    const int most = 96 * 1024 + ADJ_MAXB * 32 * 8;
    if ((e = cudaFuncSetAttribute(k_adj_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, most))) return e;
    for (const void *fn : {sweep_kernel<false>(h), sweep_kernel<true>(h)})
        if ((e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)(ADJ_WARPS * ADJ_RING_BYTES))))
            return e;
    return cudaSuccess;
}

// Zero the barrier words and launch one cooperative kernel.
template <class Args>
int launch(gdb_adj *h, const void *fn, Args f, size_t smem) {
    AdjArgs a = adj_args(h);
    ACK(cudaMemsetAsync(h->d_bar, 0, sizeof(AdjBar), h->st));
    void *args[] = {&a, &h->tab, &f};
    ACK(cudaLaunchCooperativeKernel(fn, dim3(h->blocks), dim3(h->threads), args, smem, h->st));
    return GDB_OK;
}

// Steps [s0, s0 + n) from state s0 of st; observables into d_acc and d_bins
// when wanted.
int run_forward(gdb_adj *h, States st, int s0, int n, bool observe, bool checkpoints) {
    ForwardArgs f{};
    f.st = st;
    f.s0 = s0;
    f.nsteps = n;
    f.acc = observe ? h->d_acc : nullptr;
    f.gbins = observe && h->nbins > 0 && h->rdf_every > 0 ? h->d_bins : nullptr;
    f.rdf_every = h->rdf_every;
    f.copies = rdf_copies(h);
    f.ck_pos = checkpoints ? h->d_ck_pos : nullptr;
    f.ck_vel = h->d_ck_vel;
    f.ckpt = h->ckpt;
    return launch(h, (const void *)k_adj_forward, f,
                  f.gbins ? (size_t)f.copies * h->nbins * 32 * sizeof(unsigned long long) : 0);
}

int check_status(gdb_adj *h, const char *who, unsigned status) {
    if (status & ADJ_STATUS_TIMEOUT)
        return aset(h, GDB_ERR_TIMEOUT, "%s: a grid barrier wait ran out", who);
    if (status & ADJ_STATUS_OVERFLOW)
        return aset(h, GDB_ERR_NBLIST, "%s: a list column outgrew %d entries (reach %.3f)", who,
                    h->maxnb / ADJ_LANES, h->rl);
    return GDB_OK;
}

// List reach (largest cut, or the RDF kernel's reach, plus the skin) and
// capacity (32 columns, each twice its mean count at this density plus 8).
int ensure_list(gdb_adj *h) {
    float reach = 0.f;
    for (int k = 0; k < h->nt * h->nt; k++) reach = std::max(reach, h->tab.t32[k].cut);
    if (h->nbins > 0)
        reach = std::max(reach, (float)((double)h->r_hi + ADJ_KW * h->width));
    h->rl = reach + ADJ_SKIN;
    const double vol = (double)h->box[0] * h->box[1] * h->box[2];
    const double mean = 4.0 / 3.0 * M_PI * (double)h->rl * h->rl * h->rl * h->n / vol;
    // 32 columns of rows entries: a column holds about mean / 32 neighbours
    const int rows = std::min((int)(2.0 * mean / ADJ_LANES) + 8, (h->n + ADJ_LANES - 1) / ADJ_LANES);
    const int want = rows * ADJ_LANES;
    if (want > h->maxnb || !h->d_nbl) {
        if (h->d_nbl) ACK(cudaFreeAsync(h->d_nbl, h->st));
        h->d_nbl = nullptr;
        ACK(gdb::pool_alloc(&h->d_nbl, (size_t)h->n * want * sizeof(int), h->st));
        h->maxnb = want;
    }
    if (!h->d_nbc) {
        ACK(gdb::pool_alloc(&h->d_nbc, (size_t)h->n * ADJ_LANES * sizeof(int), h->st));
        ACK(gdb::pool_alloc(&h->d_rref, h->n * sizeof(float4), h->st));
        ACK(gdb::pool_alloc(&h->d_bar, sizeof(AdjBar), h->st));
        ACK(gdb::pool_alloc(&h->d_status, sizeof(unsigned), h->st));
    }
    ACK(cudaMemsetAsync(h->d_status, 0, sizeof(unsigned), h->st));
    return GDB_OK;
}

void build_tables(gdb_adj *h, const double *params) {
    Tables &T = h->tab;
    T.nt = h->nt;
    for (int k = 0; k < h->nt * h->nt; k++) {
        const double sig = params[3 * k], eps = params[3 * k + 1], cut = params[3 * k + 2];
        Tab32 &e = T.t32[k];
        e.c = (float)(sig * sig);
        e.cu12 = (float)(4.0 * eps);
        e.cu6 = (float)(-4.0 * eps);
        e.cs12 = (float)(48.0 * eps);
        e.cs6 = (float)(-24.0 * eps);
        const double sr6 = pow(sig / cut, 6.0), sr12 = sr6 * sr6;
        const double uc = 4.0 * eps * (sr12 - sr6);
        const double sc = eps * (48.0 * sr12 - 24.0 * sr6) / (cut * cut);
        e.uc = (float)uc;
        e.sc = (float)sc;
        e.sccut = (float)(sc * cut);
        e.cut = (float)cut;
        e.cut2 = (float)cut * (float)cut;
        Tab64 &d = T.t64[k];
        d.sig2 = sig * sig;
        d.eps = eps;
        d.ieps = 1.0 / eps;
        d.eps_sig = eps / sig;
        d.cut = cut;
        d.cut2 = e.cut2;
        d.reach2 = ((float)cut + ADJ_SKIN) * ((float)cut + ADJ_SKIN);
        d.s_c = sc;
        d.dsds_c = eps * (576.0 * sr12 - 144.0 * sr6) / (cut * cut) / sig;
        d.u_c = uc;
        d.duds_c = 4.0 * eps * (12.0 * sr12 - 6.0 * sr6) / sig;
    }
}

}  // namespace

extern "C" {

int gdb_adj_create(int n, int ntypes, int device, gdb_adj **out) {
    gdb_adj *h = nullptr;
    if (!out || n < 2 || ntypes < 1 || ntypes > ADJ_MAXT)
        return aset(nullptr, GDB_ERR_ARG, "gdb_adj_create: bad arguments (n=%d, ntypes=%d, max types %d)", n, ntypes,
                    ADJ_MAXT);
    h = new gdb_adj();
    h->n = n;
    h->nt = ntypes;
    h->dev = device;
    // device memory comes from the library's stream-ordered pool: mapping the
    // kept states anew for every handle took 3.6 ms (N 4096, 51 states)
    cudaError_t e;
    if ((e = cudaSetDevice(device)) != cudaSuccess || (e = cudaStreamCreateWithFlags(&h->st, cudaStreamNonBlocking)) ||
        (e = gdb::pool_alloc(&h->d_type, n * sizeof(int), h->st)) ||
        (e = gdb::pool_alloc(&h->d_mass, n * sizeof(float), h->st)) ||
        (e = launch_shape(h)) || (e = gdb::pool_alloc(&h->d_pos, (size_t)2 * n * sizeof(float4), h->st)) ||
        (e = gdb::pool_alloc(&h->d_vel, (size_t)2 * n * sizeof(float4), h->st)) ||
        (e = gdb::pool_alloc(&h->d_acc, (size_t)h->blocks * 3 * sizeof(double), h->st)) ||
        (e = gdb::pool_alloc(&h->d_bins, ADJ_MAXB * sizeof(unsigned long long), h->st)) ||
        (e = gdb::pool_alloc(&h->d_R, (size_t)n * 3 * sizeof(double), h->st)) ||
        (e = gdb::pool_alloc(&h->d_V, (size_t)n * 3 * sizeof(double), h->st)) ||
        (e = gdb::pool_alloc(&h->d_U, (size_t)2 * n * sizeof(double4), h->st)) ||
        (e = gdb::pool_alloc(&h->d_th, (size_t)h->blocks * (1 + h->threads / 32) * ADJ_NTH * sizeof(double), h->st)) ||
        (e = gdb::pool_alloc(&h->d_gG, ADJ_MAXB * sizeof(double), h->st))) {
        adj_free(h);
        delete h;
        return aset(nullptr, GDB_ERR_CUDA, "gdb_adj_create: %s", cudaGetErrorString(e));
    }
    *out = h;
    return GDB_OK;
}

int gdb_adj_destroy(gdb_adj *h) {
    if (!h) return GDB_OK;
    adj_free(h);
    delete h;
    return GDB_OK;
}

int gdb_adj_setup(gdb_adj *h, const float box[3], const int32_t *ptype, const float *mass, float dt, int steps,
                  int checkpoint_every, int rdf_bins, float rdf_lo, float rdf_hi, float rdf_width, int rdf_every) {
    if (!h || !box || !ptype || !mass || !(dt > 0.f) || steps < 1 || checkpoint_every < 1 || rdf_bins < 0 ||
        rdf_bins > ADJ_MAXB || (rdf_bins > 0 && !(rdf_hi > rdf_lo && rdf_lo >= 0.f && rdf_width > 0.f)))
        return aset(h, GDB_ERR_ARG, "gdb_adj_setup: bad arguments");
    for (int k = 0; k < 3; k++)
        if (!(box[k] > 0.f)) return aset(h, GDB_ERR_ARG, "gdb_adj_setup: box lengths must be positive");
    for (int i = 0; i < h->n; i++) {
        if (ptype[i] < 0 || ptype[i] >= h->nt) return aset(h, GDB_ERR_ARG, "gdb_adj_setup: type out of range");
        if (!(mass[i] > 0.f)) return aset(h, GDB_ERR_ARG, "gdb_adj_setup: masses must be positive");
    }
    ACK(cudaSetDevice(h->dev));
    h->setup = h->forward_done = false;  // until everything below is in place
    memcpy(h->box, box, sizeof(h->box));
    h->dt = dt;
    h->steps = steps;
    h->ckpt = checkpoint_every;
    h->nbins = rdf_bins;
    h->r_lo = rdf_lo;
    h->r_hi = rdf_hi;
    h->width = rdf_width;
    h->rdf_every = rdf_every;
    ACK(cudaMemcpyAsync(h->d_type, ptype, h->n * sizeof(int), cudaMemcpyHostToDevice, h->st));
    ACK(cudaMemcpyAsync(h->d_mass, mass, h->n * sizeof(float), cudaMemcpyHostToDevice, h->st));
    h->n_type0 = (double)std::count(ptype, ptype + h->n, 0);
    for (float4 **p : {&h->d_ck_pos, &h->d_ck_vel, &h->d_seg_pos, &h->d_seg_vel}) {
        if (*p) ACK(cudaFreeAsync(*p, h->st));
        *p = nullptr;
    }
    // every state, or checkpoints and one segment where they would need more
    // than ADJ_KEEP_BYTES (or the memory is not there)
    const size_t all = (size_t)(steps + 1) * h->n * sizeof(float4);
    const char *keep = getenv("GDB_ADJ_KEEP_BYTES");
    h->keep_all = 2 * all <= (keep && *keep ? (size_t)std::max(0LL, atoll(keep)) : ADJ_KEEP_BYTES);
    if (h->keep_all && (gdb::pool_alloc(&h->d_seg_pos, all, h->st) != cudaSuccess ||
                        gdb::pool_alloc(&h->d_seg_vel, all, h->st) != cudaSuccess)) {
        (void)cudaGetLastError();
        if (h->d_seg_pos) cudaFreeAsync(h->d_seg_pos, h->st);
        h->d_seg_pos = h->d_seg_vel = nullptr;
        h->keep_all = false;
    }
    if (!h->keep_all) {
        const int nck = (steps + checkpoint_every - 1) / checkpoint_every;
        ACK(gdb::pool_alloc(&h->d_ck_pos, (size_t)nck * h->n * sizeof(float4), h->st));
        ACK(gdb::pool_alloc(&h->d_ck_vel, (size_t)nck * h->n * sizeof(float4), h->st));
        ACK(gdb::pool_alloc(&h->d_seg_pos, (size_t)(checkpoint_every + 1) * h->n * sizeof(float4), h->st));
        ACK(gdb::pool_alloc(&h->d_seg_vel, (size_t)(checkpoint_every + 1) * h->n * sizeof(float4), h->st));
    }
    ACK(cudaStreamSynchronize(h->st));
    h->setup = true;
    return GDB_OK;
}

int gdb_adj_forward(gdb_adj *h, const double *params, const float *r0, const float *v0, double *obs) {
    if (!h || !params || !r0 || !v0 || !obs) return aset(h, GDB_ERR_ARG, "gdb_adj_forward: bad arguments");
    if (!h->setup) return aset(h, GDB_ERR_STATE, "gdb_adj_forward: call gdb_adj_setup first");
    for (int k = 0; k < h->nt * h->nt; k++) {
        const double sig = params[3 * k], eps = params[3 * k + 1], cut = params[3 * k + 2];
        if (!(sig > 0.0 && eps > 0.0 && cut > 0.0))
            return aset(h, GDB_ERR_ARG, "gdb_adj_forward: sigma, epsilon and cut must be positive");
        if (2.0 * cut >= std::min(std::min(h->box[0], h->box[1]), h->box[2]))
            return aset(h, GDB_ERR_ARG, "gdb_adj_forward: cut must be below half the box");
    }
    ACK(cudaSetDevice(h->dev));
    h->forward_done = false;  // the last forward's tables and states are overwritten from here on
    build_tables(h, params);
    const int n = h->n;
    int rc = ensure_list(h);
    if (rc) return rc;
    float *dr = nullptr, *dv = nullptr;
    ACK(gdb::pool_alloc(&dr, (size_t)n * 3 * sizeof(float), h->st));
    ACK(gdb::pool_alloc(&dv, (size_t)n * 3 * sizeof(float), h->st));
    ACK(cudaMemcpyAsync(dr, r0, (size_t)n * 3 * sizeof(float), cudaMemcpyHostToDevice, h->st));
    ACK(cudaMemcpyAsync(dv, v0, (size_t)n * 3 * sizeof(float), cudaMemcpyHostToDevice, h->st));
    float4 *p0 = h->keep_all ? h->d_seg_pos : h->d_pos, *v0d = h->keep_all ? h->d_seg_vel : h->d_vel;
    k_adj_pack<<<(n + 255) / 256, 256, 0, h->st>>>(n, dr, dv, h->d_type, p0, v0d);
    ACK(cudaGetLastError());
    ACK(cudaFreeAsync(dr, h->st));
    ACK(cudaFreeAsync(dv, h->st));
    ACK(cudaMemsetAsync(h->d_bins, 0, ADJ_MAXB * sizeof(unsigned long long), h->st));
    rc = run_forward(h, States{p0, v0d, 0, h->keep_all ? h->steps + 1 : 2}, 0, h->steps, true, !h->keep_all);
    if (rc) return rc;
    h->nsamples = h->nbins > 0 && h->rdf_every > 0 ? (h->steps + h->rdf_every - 1) / h->rdf_every : 0;
    std::vector<double> acc((size_t)h->blocks * 3);
    std::vector<unsigned long long> bins(ADJ_MAXB);
    ACK(cudaMemcpyAsync(acc.data(), h->d_acc, acc.size() * sizeof(double), cudaMemcpyDeviceToHost, h->st));
    ACK(cudaMemcpyAsync(bins.data(), h->d_bins, ADJ_MAXB * sizeof(unsigned long long), cudaMemcpyDeviceToHost, h->st));
    unsigned status = 0;
    ACK(cudaMemcpyAsync(&status, h->d_status, sizeof(unsigned), cudaMemcpyDeviceToHost, h->st));
    ACK(cudaStreamSynchronize(h->st));
    if ((rc = check_status(h, "gdb_adj_forward", status))) return rc;
    h->obs.assign(3 + h->nbins, 0.0);
    for (int b = 0; b < h->blocks; b++)
        for (int q = 0; q < 3; q++) h->obs[q] += acc[(size_t)b * 3 + q];
    for (int q = 0; q < 3; q++) h->obs[q] /= h->steps;
    if (h->nbins > 0 && h->nsamples > 0) {
        // g_b = sum K / (samples * N_A * rho_A * 4 pi r_b^2)
        const double na = h->n_type0;
        const double vol = (double)h->box[0] * h->box[1] * h->box[2];
        const double dr_ = (double)(h->r_hi - h->r_lo) / h->nbins;
        for (int b = 0; b < h->nbins; b++) {
            const double rb = h->r_lo + (b + 0.5) * dr_;
            const double norm = 1.0 / (h->nsamples * na * (na / vol) * 4.0 * M_PI * rb * rb);
            h->obs[3 + b] = (double)bins[b] / ADJ_FIX * norm;
        }
    }
    memcpy(obs, h->obs.data(), h->obs.size() * sizeof(double));
    h->forward_done = true;
    return GDB_OK;
}

int gdb_adj_backward(gdb_adj *h, const double *grad_obs, double *grad_params) {
    if (!h || !grad_obs || !grad_params) return aset(h, GDB_ERR_ARG, "gdb_adj_backward: bad arguments");
    if (!h->forward_done) return aset(h, GDB_ERR_STATE, "gdb_adj_backward: run gdb_adj_forward first");
    ACK(cudaSetDevice(h->dev));
    const int n = h->n, T = h->steps;
    const double gU = grad_obs[0] / T, gW = grad_obs[1] / T, gK = grad_obs[2] / T;
    // dL/dr contributions of g_b on a sampled step: grad_g_b * norm_b
    std::vector<double> gG(ADJ_MAXB, 0.0);
    bool any_g = false;
    if (h->nbins > 0 && h->nsamples > 0) {
        const double na = h->n_type0;
        const double vol = (double)h->box[0] * h->box[1] * h->box[2];
        const double dr_ = (double)(h->r_hi - h->r_lo) / h->nbins;
        const double w = h->width;
        for (int b = 0; b < h->nbins; b++) {
            const double rb = h->r_lo + (b + 0.5) * dr_;
            const double g = grad_obs[3 + b] / (h->nsamples * na * (na / vol) * 4.0 * M_PI * rb * rb);
            any_g |= g != 0.0;
            gG[b] = g * 2.0 * (-1.0 / (w * w)) / (sqrt(2.0 * M_PI) * w);
        }
        ACK(cudaMemcpyAsync(h->d_gG, gG.data(), ADJ_MAXB * sizeof(double), cudaMemcpyHostToDevice, h->st));
    }
    const int nb = h->blocks;
    ACK(cudaMemsetAsync(h->d_R, 0, (size_t)n * 3 * sizeof(double), h->st));
    ACK(cudaMemsetAsync(h->d_V, 0, (size_t)n * 3 * sizeof(double), h->st));
    SweepArgs f{};
    f.gU = gU;
    f.gW = gW;
    f.gK = gK;
    f.gG = any_g ? h->d_gG : nullptr;
    f.rdf_every = h->rdf_every;
    f.window = h->window;
    f.R = h->d_R;
    f.V = h->d_V;
    f.U = h->d_U;
    f.th_part = h->d_th;
    f.th_warp = h->d_th + (size_t)nb * ADJ_NTH;
    const int seg = h->keep_all ? T : h->ckpt;
    for (int sg = (T + seg - 1) / seg - 1; sg >= 0; sg--) {
        const int s0 = sg * seg, len = std::min(seg, T - s0);
        f.st = States{h->d_seg_pos, h->d_seg_vel, s0, len + 1};
        f.s0 = s0;
        f.len = len;
        f.first_segment = s0 + len == T;
        f.last_segment = sg == 0;
        int rc;
        if (!h->keep_all) {  // recompute the segment's states (bit-identical to the forward)
            const size_t off = (size_t)sg * n;
            ACK(cudaMemcpyAsync(h->d_seg_pos, h->d_ck_pos + off, n * sizeof(float4), cudaMemcpyDeviceToDevice, h->st));
            ACK(cudaMemcpyAsync(h->d_seg_vel, h->d_ck_vel + off, n * sizeof(float4), cudaMemcpyDeviceToDevice, h->st));
            if ((rc = run_forward(h, f.st, s0, len, false, false))) return rc;
        }
        if ((rc = launch(h, sweep_kernel(h), f, h->threads / 32 * ADJ_RING_BYTES))) return rc;
    }
    std::vector<double> th((size_t)nb * ADJ_NTH);
    unsigned status = 0;
    ACK(cudaMemcpyAsync(th.data(), h->d_th, th.size() * sizeof(double), cudaMemcpyDeviceToHost, h->st));
    ACK(cudaMemcpyAsync(&status, h->d_status, sizeof(unsigned), cudaMemcpyDeviceToHost, h->st));
    ACK(cudaStreamSynchronize(h->st));
    if (int rc = check_status(h, "gdb_adj_backward", status)) return rc;
    // fixed-order sum over blocks; a parameter of the unordered pair {a, b}
    // collects the (a, b) and (b, a) entries
    const int nt = h->nt;
    std::vector<double> g(2 * nt * nt, 0.0);
    for (int b = 0; b < nb; b++)
        for (int k = 0; k < 2 * nt * nt; k++) g[k] += th[(size_t)b * ADJ_NTH + k];
    for (int x = 0; x < nt; x++)
        for (int y = 0; y < nt; y++) {
            const int k = x * nt + y, kt = y * nt + x;
            const double gs = x == y ? g[2 * k] : g[2 * k] + g[2 * kt];
            const double ge = x == y ? g[2 * k + 1] : g[2 * k + 1] + g[2 * kt + 1];
            grad_params[3 * k] = gs;
            grad_params[3 * k + 1] = ge;
            grad_params[3 * k + 2] = 0.0;
        }
    return GDB_OK;
}

int gdb_adj_set_window(gdb_adj *h, int window) {
    if (!h || window < 0) return aset(h, GDB_ERR_ARG, "gdb_adj_set_window: bad arguments");
    h->window = window;
    return GDB_OK;
}

int gdb_adj_final_state(gdb_adj *h, float *r, float *v) {
    if (!h || !h->forward_done) return aset(h, GDB_ERR_STATE, "gdb_adj_final_state: no forward run");
    ACK(cudaSetDevice(h->dev));
    const size_t last = (size_t)(h->keep_all ? h->steps : h->steps & 1) * h->n;
    std::vector<float4> p(h->n), q(h->n);
    ACK(cudaMemcpy(p.data(), (h->keep_all ? h->d_seg_pos : h->d_pos) + last, h->n * sizeof(float4), cudaMemcpyDeviceToHost));
    ACK(cudaMemcpy(q.data(), (h->keep_all ? h->d_seg_vel : h->d_vel) + last, h->n * sizeof(float4), cudaMemcpyDeviceToHost));
    for (int i = 0; i < h->n; i++) {
        if (r) {
            r[3 * i] = p[i].x;
            r[3 * i + 1] = p[i].y;
            r[3 * i + 2] = p[i].z;
        }
        if (v) {
            v[3 * i] = q[i].x;
            v[3 * i + 1] = q[i].y;
            v[3 * i + 2] = q[i].z;
        }
    }
    return GDB_OK;
}

int gdb_adj_get_last_error(gdb_adj *h, char *buf, int n) {
    if (!buf || n < 1) return GDB_ERR_ARG;
    snprintf(buf, (size_t)n, "%s", h ? h->err : g_adj_error);
    return GDB_OK;
}

}  // extern "C"
