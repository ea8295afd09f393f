// kernels_expand.cu -- solves whose augmented state evolves by itself.
//
// Without inputs, or with sum-of-sinusoid inputs, nothing has to be sampled:
// with the phases f = [sin th_q ; cos th_q] of every (channel, term) beside
// the scan state, z = [x ; f] obeys z_{k+1} = diag-block map z_k, so over L
// steps from any start
//   x(k + L) = Phi^L x(k) + S_L f(k),        E(L) = [Phi^L | S_L],
//   E(a + b) = Phi^a E(b) + [0 | S_a R_b]    (R_b: rotation by b steps),
// with S_1 the one-step forcing (the reference's BTimesU kernels,
// Kernels/BTimesURK4thOrder.cl:15-37, BTimesUAdamsMoulton.cl:17-38) applied to
// a sin(th + w dt j).  E(2^l) come from squarings, any other length from the
// set bits.  The states entering the blocks of B steps are then a radix-16
// expansion (the exclusive scan's down-sweep with every up-sweep aggregate
// replaced by its closed form S_L f):
//   X_{i d + j} = E(i d B) [X_j ; f_j],   j < d = 16^l, i = 1 .. 15,
// each level one FP64 DMMA product with no sequential step, and the outputs
// of a block are W [X_b ; f_b], W's row (j, o) = C E(j) (+ D's phases).
// Against the sample-window form of the block-response leaf (kernels_br.cu):
// no samples, no aggregates, no carry chain; 2 p (NP + H) flops per step for
// the outputs and 2 NP (NP + H) / B for the states, H = 2 m terms, so the
// blocks can be long (B = 64).  Measured on one B200: RK4 n = 64, m = p = 8,
// 2^20 steps mixed 0.277 ms (samples 0.034, 3xTF32 windows 0.085, carry 0.105,
// state part 0.07) -> 0.086 ms; a free response of 24 states, 10^5 steps
// (FP64) 0.240 ms with the in-block sweeps -> 0.016 ms.
//
// The phases of a block's start are sincos of the argument rounded as the
// oracle rounds it; within a block they advance exactly (by the tables), so
// the result differs from the rounded-argument samples by the rounding of the
// sample times (w ulp(t)): the mixed form's sample planes had the same
// difference.  The FP64 form keeps its samples.
#include "expand.h"

#include "common.h"
#include "device_common.cuh"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace parode {

namespace {

constexpr int kThreads = 256;
constexpr size_t kSmemMax = 220 * 1024;

// Column counts with a kernel (multiples of 8; K steps of 4).
constexpr int kWidths[] = {8, 16, 24, 32, 40, 48, 56, 64, 80, 96, 112, 128, 144, 160};

// Shared row pitch, 8 mod 16 doubles.  A lane reads two consecutive doubles
// (K index 8 c + 2 t + u feeds product 2 c + u): a quarter warp's two rows
// then fall in different bank halves.
__host__ __device__ inline int smem_pitch(int Kc) { return Kc + ((Kc & 8) ? 0 : 8); }

__device__ __forceinline__ void cp_async16(double* dst, const double* src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// ---- tables ------------------------------------------------------------------

// E(2^l), l < pow_levels, by squaring: one cluster of 8 CTAs.  Every CTA holds
// all of Phi^(2^l) (NP x NP) and its own 8-column tiles of S: per level it
// forms its state tile of the square (written into every CTA's next copy
// through distributed shared memory) and its phase tiles, one cluster barrier
// a level.  Set-up only and latency-bound: on one CTA (one SM's FP64 rate)
// a level took 8 us at NP = 64, Kc = 112, 0.16 ms for 20 levels.
constexpr int kSqCtas = 8;

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_barrier()
{
    cluster_arrive();
    cluster_wait();
}

__device__ __forceinline__ void store_remote(double* local, unsigned rank, double v0, double v1)
{
    const unsigned a = (unsigned)__cvta_generic_to_shared(local);
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(a), "r"(rank));
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};\n" ::"r"(r), "d"(v0), "d"(v1) : "memory");
}

__global__ void __cluster_dims__(kSqCtas, 1, 1) __launch_bounds__(kThreads, 1) k_expand_squarings(const ExpandTables t)
{
    extern __shared__ __align__(16) double sm[];
    cluster_arrive();  // waited for before the first store into a peer's shared memory
    const int NP = t.sh.NP, Kc = t.sh.Kc, ld = NP + 4;  // 4 mod 8 doubles: conflict-free fragments
    const int rank = blockIdx.x;
    const int HQ = t.sh.H / 2, n = t.n, m = t.mu, K = t.terms;
    const int htiles = (Kc - NP) / 8, own = (htiles - rank + kSqCtas - 1) / kSqCtas;  // phase tiles rank, rank + 8, ..
    const int maxown = (htiles + kSqCtas - 1) / kSqCtas;
    const int ldS = 8 * maxown + 4;
    double* P[2] = {sm, sm + NP * ld};
    double* S[2] = {P[1] + NP * ld, P[1] + NP * ld + NP * ldS};
    double* sn = S[1] + NP * ldS;  // sin, cos of w dt 2^l of the own phase pairs
    double* cs = sn + 4 * maxown;
    const bool rk4 = t.solver == 0;
    const int Wd = rk4 ? 3 : 5, coff = rk4 ? 0 : 3 * n;
    const double *amp = t.par, *w = t.par + HQ;
    const int steps = rk4 ? 2 : 1;  // samples per step
    for (int e = threadIdx.x; e < NP * NP; e += kThreads) P[0][(e / NP) * ld + e % NP] = t.Phi[e];
    // S_1: window slot s of the step reads sample s, at phase th + w dt s
    for (int e = threadIdx.x; e < NP * 4 * own; e += kThreads) {
        const int r = e / (4 * own), u = e - r * 4 * own;
        const int q = ((u / 4) * kSqCtas + rank) * 4 + u % 4;  // phase pair
        double vs = 0.0, vc = 0.0;
        if (q < HQ && !t.zeroB && r >= coff && r < coff + n)
            for (int sl = 0; sl < Wd; ++sl) {
                double si, co;
                sincos(__dmul_rn(w[q], t.dt) * sl, &si, &co);
                const double b = t.Bbar[(long)(r - coff) * Wd * m + sl * m + q / K] * amp[q];
                vs = fma(b, co, vs);
                vc = fma(b, si, vc);
            }
        S[0][r * ldS + 2 * u] = vs;
        S[0][r * ldS + 2 * u + 1] = vc;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, tq = lane & 3;
    const int MT = NP / 8;
    int cur = 0;
    // every CTA of the cluster runs: its shared memory may be written (the
    // ranks' S_1 take different times, none at all without inputs)
    __syncwarp();
    cluster_wait();
    for (int l = 0;; ++l) {
        for (int u = threadIdx.x; u < 4 * own; u += kThreads) {
            const int q = ((u / 4) * kSqCtas + rank) * 4 + u % 4;
            sincos(q < HQ ? ldexp(__dmul_rn(w[q], t.dt) * steps, l) : 0.0, &sn[u], &cs[u]);
        }
        __syncthreads();
        // own columns of E(2^l)
        double* out = t.E + (long)l * NP * Kc;
        if (rank < MT)
            for (int e = threadIdx.x; e < NP * 8; e += kThreads)
                out[(long)(e >> 3) * Kc + rank * 8 + (e & 7)] = P[cur][(e >> 3) * ld + rank * 8 + (e & 7)];
        for (int e = threadIdx.x; e < NP * 8 * own; e += kThreads) {
            const int r = e / (8 * own), u = e - r * 8 * own;
            out[(long)r * Kc + NP + ((u >> 3) * kSqCtas + rank) * 8 + (u & 7)] = S[cur][r * ldS + u];
        }
        if (l + 1 >= t.sh.pow_levels) break;
        const int nx = cur ^ 1;
        if (warp < MT) {
            const double* a = P[cur] + (warp * 8 + g) * ld + tq;
            const int r = warp * 8 + g;
            for (int tile = rank < MT ? -1 : 0; tile < own; ++tile) {
                const double* b = tile < 0 ? P[cur] + tq * ld + rank * 8 + g : S[cur] + tq * ldS + tile * 8 + g;
                const int lb = tile < 0 ? ld : ldS;
                double part[2][2] = {};
#pragma unroll 4
                for (int k = 0; k < NP / 4; k += 2) {
                    dmma_m8n8k4(part[0][0], part[0][1], a[4 * k], b[4 * k * lb]);
                    dmma_m8n8k4(part[1][0], part[1][1], a[4 * k + 4], b[4 * (k + 1) * lb]);
                }
                double v0 = part[0][0] + part[1][0], v1 = part[0][1] + part[1][1];
                if (tile < 0) {
                    for (unsigned c = 0; c < kSqCtas; ++c) store_remote(P[nx] + r * ld + rank * 8 + 2 * tq, c, v0, v1);
                } else {
                    const int u = tile * 4 + tq;
                    const double s0 = S[cur][r * ldS + 2 * u], s1 = S[cur][r * ldS + 2 * u + 1];
                    S[nx][r * ldS + 2 * u] = v0 + s0 * cs[u] - s1 * sn[u];
                    S[nx][r * ldS + 2 * u + 1] = v1 + s0 * sn[u] + s1 * cs[u];
                }
            }
        }
        // every CTA has written its tile of the next square and is done with this one
        cluster_barrier();
        cur = nx;
    }
    cluster_barrier();  // no CTA leaves while another may still write to it
}

// Table rows from the powers: CTA = 8 rows.  The first rows() rows are W's
// (row (j, o): C E(j), plus D's phases at step j), then the levels' multiples
// (level l, i, r: row r of E(i 16^l B)).  A row vector [c | s] times E(2^b)
// for every set bit b of its length: c <- c Phi^(2^b),
// s <- c S_(2^b) + s R_(2^b).
__global__ void __launch_bounds__(kThreads) k_expand_rows(const ExpandTables t, int out_tiles)
{
    extern __shared__ double sm[];
    const int NP = t.sh.NP, Kc = t.sh.Kc, H = t.sh.H, ld = smem_pitch(Kc), HQ = H / 2;
    const int M = t.sh.rows(), p = t.sh.p;
    double* cur = sm;
    double* nxt = cur + 8 * ld;
    __shared__ long s_len[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, tq = lane & 3;
    const bool outs = (int)blockIdx.x < out_tiles;
    const int steps = t.solver == 0 ? 2 : 1;
    const double *amp = t.par, *w = t.par + HQ;
    double* dst = nullptr;
    int row0 = 0, valid = 8, b0 = 0, nbits = 0;
    if (outs) {
        row0 = blockIdx.x * 8;
        valid = min(8, M - row0);
        dst = t.W + (long)row0 * Kc;
        nbits = t.sh.R;
    } else {
        long tr = ((long)blockIdx.x - out_tiles) * 8;  // row of the level tables
        dst = t.T + tr * Kc;
        int l = 0;
        while (tr >= (long)t.sh.imax[l] * NP) tr -= (long)t.sh.imax[l] * NP, ++l;
        row0 = (int)tr;  // (i - 1) NP + r
        b0 = t.sh.R + 4 * l;
        nbits = 4;
    }
    if (threadIdx.x < 8) {
        const int row = row0 + threadIdx.x;
        s_len[threadIdx.x] = outs ? row / p : row / NP + 1;
    }
    for (int e = threadIdx.x; e < 8 * Kc; e += kThreads) {
        const int r = e / Kc, c = e - r * Kc, row = row0 + r;
        double v = 0.0;
        if (c < NP && r < valid) v = outs ? t.Cext[(long)(row % p) * NP + c] : (row % NP == c ? 1.0 : 0.0);
        cur[r * ld + c] = v;
    }
    __syncthreads();
    for (int b = 0; b < nbits; ++b) {
        bool any = false;
        for (int r = 0; r < 8; ++r) any |= ((s_len[r] >> b) & 1) != 0;
        if (!any) continue;
        const double* E = t.E + (long)(b0 + b) * NP * Kc;
        for (int nt = warp; nt < Kc / 8; nt += kThreads / 32) {
            double part[2][2] = {};
            const double* a = cur + g * ld + tq;
            const double* bb = E + (long)tq * Kc + nt * 8 + g;
#pragma unroll 4
            for (int k = 0; k < NP / 4; ++k)
                dmma_m8n8k4(part[k & 1][0], part[k & 1][1], a[4 * k], bb[(long)4 * k * Kc]);
            double v0 = part[0][0] + part[1][0], v1 = part[0][1] + part[1][1];
            const int c = nt * 8 + 2 * tq, q = (c - NP) / 2;
            const double s0 = cur[g * ld + c], s1 = cur[g * ld + c + 1];
            if (c >= NP && q < HQ) {
                double si, co;
                sincos(ldexp(__dmul_rn(w[q], t.dt) * steps, b0 + b), &si, &co);
                v0 += s0 * co - s1 * si;
                v1 += s0 * si + s1 * co;
            }
            const bool on = ((s_len[g] >> b) & 1) != 0;
            nxt[g * ld + c] = on ? v0 : s0;
            nxt[g * ld + c + 1] = on ? v1 : s1;
        }
        __syncthreads();
        double* x = cur;
        cur = nxt;
        nxt = x;
    }
    for (int e = threadIdx.x; e < valid * Kc; e += kThreads) {
        const int r = e / Kc, c = e - r * Kc;
        double v = cur[r * ld + c];
        if (outs && !t.zeroD && c >= NP && c < NP + H) {
            // D u at step j: RK4 sample 2 j, ABM sample j + 3
            const int row = row0 + r, q = (c - NP) / 2;
            double si, co;
            const long j = row / p;
            sincos(__dmul_rn(w[q], t.dt) * (double)(t.solver == 0 ? 2 * j : j + 3), &si, &co);
            v += t.D[(long)(row % p) * t.mu + q / t.terms] * amp[q] * ((c - NP) & 1 ? si : co);
        }
        dst[e] = v;
    }
}

// ---- one solve ----------------------------------------------------------------

// Phases of every block's first sample (pad columns zero) and X_0.  One
// thread per (block, pair of phase columns): FP64 sincos, ~24 per block.
__global__ void __launch_bounds__(kThreads) k_expand_phases(double* __restrict__ Z, const double* __restrict__ X0,
                                                             const double* __restrict__ par, int NP, int Kc, int HQ,
                                                             double base, double dt, long stride, long nblocks)
{
    grid_dep_trigger();  // the first level may load its table
    const long e = (long)blockIdx.x * kThreads + threadIdx.x;
    if (e < NP) Z[e] = X0[e];
    const int pairs = (Kc - NP) / 2;
    if (pairs == 0 || e >= nblocks * pairs) return;
    const long b = e / pairs;
    const int q = (int)(e - b * pairs);
    double si = 0.0, co = 0.0;
    if (q < HQ) {
        const double ts = sample_time(base, dt, b * stride);
        sincos(__dadd_rn(__dmul_rn(par[HQ + q], ts), par[2 * HQ + q]), &si, &co);
    }
    *reinterpret_cast<double2*>(Z + b * Kc + NP + 2 * q) = make_double2(si, co);
}

// One level: X_{i d + j} = T_i Z_j for j < d, i = blockIdx.y + 1.  A CTA takes
// `tiles` 8-column tiles of j, staged once in shared memory; warp = 8 rows of
// T_i (B fragments in registers, loaded before the wait on the level below).
// Four partial chains: the first levels are latency-bound (a few CTAs), the
// last one FP64-tensor bound.
constexpr int kLevelTiles = 4;

template <int KS>
__global__ void __launch_bounds__(kThreads) k_expand_level(const double* __restrict__ T, double* Z, long d,
                                                            long nblocks, int NP, int tiles)
{
    constexpr int Kc = 4 * KS, ld = Kc + ((Kc & 8) ? 0 : 8);
    __shared__ __align__(16) double Zs[8 * kLevelTiles * ld];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, tq = lane & 3;
    const int MT = NP / 8, groups = (kThreads / 32) / MT;
    const int mt = warp % MT, grp = warp / MT;
    const long i = blockIdx.y + 1;
    double2 eb[KS / 2];
    if (grp < groups) {
        const double* e = T + ((i - 1) * NP + mt * 8 + g) * Kc + 2 * tq;
#pragma unroll
        for (int k = 0; k < KS / 2; ++k) eb[k] = *reinterpret_cast<const double2*>(e + 8 * k);
    }
    grid_dep_wait();     // Z's columns below d
    grid_dep_trigger();  // the next level may load its table
    const long j0 = (long)blockIdx.x * tiles * 8;
    const int cols = (int)max(0L, min((long)tiles * 8, min(d, nblocks - i * d) - j0));
    for (int e = threadIdx.x; e < cols * (Kc / 2); e += kThreads) {
        const int c = e / (Kc / 2), k = 2 * (e - c * (Kc / 2));
        cp_async16(Zs + c * ld + k, Z + (j0 + c) * Kc + k);
    }
    cp_async_wait_all();
    __syncthreads();
    if (grp >= groups) return;
    for (int u = grp; u * 8 < cols; u += groups) {
        const bool ok = u * 8 + g < cols;
        const double* z = Zs + (ok ? u * 8 + g : 0) * ld + 2 * tq;
        double part[4][2] = {};
#pragma unroll
        for (int k = 0; k < KS / 2; ++k) {
            const double2 za = *reinterpret_cast<const double2*>(z + 8 * k);
            dmma_m8n8k4(part[(2 * k) & 3][0], part[(2 * k) & 3][1], za.x, eb[k].x);
            dmma_m8n8k4(part[(2 * k + 1) & 3][0], part[(2 * k + 1) & 3][1], za.y, eb[k].y);
        }
        if (ok) {
            const double v0 = (part[0][0] + part[1][0]) + (part[2][0] + part[3][0]);
            const double v1 = (part[0][1] + part[1][1]) + (part[2][1] + part[3][1]);
            *reinterpret_cast<double2*>(Z + (i * d + j0 + u * 8 + g) * Kc + mt * 8 + 2 * tq) = make_double2(v0, v1);
        }
    }
}

// Outputs: Y[b gs + r] = W[r] . Z[b].  A CTA keeps a slice of W's rows in
// shared memory; a warp takes (tile of 8 CT blocks, part of the slice's rows)
// tasks: the blocks' Z as A fragments in registers, then per 8 rows KS x CT
// m8n8k4 products and direct stores (a block's 8 rows are 64 consecutive
// bytes, two per lane).  FP64-tensor bound: RK4 n = 64, m = p = 8, 2^20 steps
// is 1.88 GFLOP against 67 MB written, 51 us of DMMA; 64 us, the pipe 89 % busy
// while the CTAs run (85 us, 68 %, with 8-byte fragment loads from pitches of
// 4 mod 16 doubles).  Row tiles in equal parts even out the warps of the four
// sub-partitions.
template <int KS>
struct OutCfg {
    static constexpr int CT = KS <= 28 ? 2 : 1;
    static constexpr int threads = KS <= 28 ? 384 : 512;
};

template <int KS>
__global__ void __launch_bounds__(OutCfg<KS>::threads, 1)
    k_expand_out(const double* __restrict__ W, int M, int Ms, int slices, const double* Z, double* Y,
                 long gs, long c0, long c1, long limit, int vec)
{
    extern __shared__ __align__(16) double Ws[];
    constexpr int Kc = 4 * KS, ld = Kc + ((Kc & 8) ? 0 : 8), CT = OutCfg<KS>::CT, kT = OutCfg<KS>::threads;
    const int slice = blockIdx.x % slices, idx = blockIdx.x / slices;
    const int nidx = ((int)gridDim.x - slice + slices - 1) / slices;
    const int m0 = slice * Ms, rows = min(Ms, M - m0), RT = (rows + 7) / 8;
    for (int e = threadIdx.x; e < RT * 8 * (Kc / 2); e += kT) {
        const int r = e / (Kc / 2), c = 2 * (e - r * (Kc / 2));
        if (r < rows) cp_async16(Ws + r * ld + c, W + (long)(m0 + r) * Kc + c);
        else *reinterpret_cast<double2*>(Ws + r * ld + c) = make_double2(0.0, 0.0);
    }
    cp_async_wait_all();
    __syncthreads();
    grid_dep_wait();
    grid_dep_trigger();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, tq = lane & 3;
    const long nt = (c1 - c0 + 8 * CT - 1) / (8 * CT);
    // the slice's row tiles, tile after tile, in equal parts to its CTAs' warps
    const long total = nt * RT, gw = (long)idx * (kT / 32) + warp, nw = (long)nidx * (kT / 32);
    long left = total * (gw + 1) / nw - total * gw / nw, tile = total * gw / nw / RT;
    int r0 = (int)(total * gw / nw - tile * RT);
    for (int r1; left > 0; left -= r1 - r0, r0 = 0, ++tile) {
        r1 = (int)min((long)RT, r0 + left);
        const long b0 = c0 + tile * 8 * CT;
        double2 za[CT][KS / 2];
#pragma unroll
        for (int c = 0; c < CT; ++c) {
            const long b = b0 + 8 * c + g;
            const double* z = Z + (b < c1 ? b : c0) * Kc + 2 * tq;
#pragma unroll
            for (int k = 0; k < KS / 2; ++k) za[c][k] = *reinterpret_cast<const double2*>(z + 8 * k);
        }
        for (int rt = r0; rt < r1; ++rt) {
            double acc[CT][2] = {};
            const double* wr = Ws + (rt * 8 + g) * ld + 2 * tq;
#pragma unroll
            for (int k = 0; k < KS / 2; ++k) {
                const double2 w = *reinterpret_cast<const double2*>(wr + 8 * k);
#pragma unroll
                for (int c = 0; c < CT; ++c) dmma_m8n8k4(acc[c][0], acc[c][1], za[c][k].x, w.x);
#pragma unroll
                for (int c = 0; c < CT; ++c) dmma_m8n8k4(acc[c][0], acc[c][1], za[c][k].y, w.y);
            }
            const int r = m0 + rt * 8 + 2 * tq;
#pragma unroll
            for (int c = 0; c < CT; ++c) {
                const long b = b0 + 8 * c + g, o = b * gs + r;
                if (b >= c1 || r >= M) continue;
                if (vec && o + 1 < limit) {
                    *reinterpret_cast<double2*>(Y + o) = make_double2(acc[c][0], acc[c][1]);
                } else {
                    if (o < limit) Y[o] = acc[c][0];
                    if (r + 1 < M && o + 1 < limit) Y[o + 1] = acc[c][1];
                }
            }
        }
    }
}

// ---- batches -----------------------------------------------------------------
// blockIdx.y = job; the x dimension strides over its elements.

constexpr double kTwoPi = 6.283185307179586476925286766559;

// S_1 into E(1)'s phase columns (pads zero), W's first p rows [Cext | 0], and
// the rotation table.
__global__ void __launch_bounds__(kThreads) k_expand_init_batch(const ExpandJob* __restrict__ jobs)
{
    extern __shared__ double trig[];  // sin, cos of w dt s per (pair, slot)
    const ExpandJob j = jobs[blockIdx.y];
    const int HQ = j.H / 2, pairs = (j.Kc - j.NP) / 2, rk4 = j.solver == 0, Wd = rk4 ? 3 : 5;
    const int coff = rk4 ? 0 : 3 * j.n;
    for (int e = threadIdx.x; e < HQ * Wd; e += kThreads) {
        const int q = e / Wd, sl = e - q * Wd;
        sincos(__dmul_rn(__dmul_rn(kTwoPi, j.freq[q]), j.dt) * sl, &trig[2 * e], &trig[2 * e + 1]);
    }
    __syncthreads();
    const long n0 = (long)j.NP * pairs, n1 = (long)j.p * j.Kc, n2 = (long)j.pow_levels * HQ;
    for (long e = (long)blockIdx.x * kThreads + threadIdx.x; e < n0 + n1 + n2; e += (long)gridDim.x * kThreads) {
        if (e < n0) {
            const int r = (int)(e / pairs), q = (int)(e - (long)r * pairs);
            double vs = 0.0, vc = 0.0;
            if (q < HQ && !j.zeroB && r >= coff && r < coff + j.n)
                for (int sl = 0; sl < Wd; ++sl) {
                    const double b = j.Bbar[(long)(r - coff) * Wd * j.mu + sl * j.mu + q / j.terms] * j.amp[q];
                    vs = fma(b, trig[2 * (q * Wd + sl) + 1], vs);
                    vc = fma(b, trig[2 * (q * Wd + sl)], vc);
                }
            *reinterpret_cast<double2*>(j.E + (long)r * j.Kc + j.NP + 2 * q) = make_double2(vs, vc);
        } else if (e < n0 + n1) {
            const long u = e - n0;
            const int o = (int)(u / j.Kc), c = (int)(u - (long)o * j.Kc);
            j.W[u] = c < j.NP ? j.Cext[(long)o * j.NP + c] : 0.0;
        } else {
            const long u = e - n0 - n1;
            const int l = (int)(u / HQ), q = (int)(u - (long)l * HQ);
            const double step = __dmul_rn(__dmul_rn(kTwoPi, j.freq[q]), j.dt) * (rk4 ? 2 : 1);
            sincos(ldexp(step, l), &j.rot[2 * u], &j.rot[2 * u + 1]);
        }
    }
}

// The rotation parts [0 | S R] of step l, which its GEMMs then add to.
__global__ void __launch_bounds__(kThreads) k_expand_rot_batch(const ExpandJob* __restrict__ jobs, int l)
{
    const ExpandJob j = jobs[blockIdx.y];
    const int half = j.Kc / 2, HQ = j.H / 2;
    const long erows = l + 1 < j.pow_levels ? j.NP : 0, wrows = l < j.R ? ((long)1 << l) * j.p : 0;
    const double* rot = j.rot + (long)l * j.H;
    for (long e = (long)blockIdx.x * kThreads + threadIdx.x; e < (erows + wrows) * half;
         e += (long)gridDim.x * kThreads) {
        const long r = e / half;
        const int c = 2 * (int)(e - r * half), q = (c - j.NP) / 2;
        const double* src = r < erows ? j.E + ((long)l * j.NP + r) * j.Kc : j.W + (r - erows) * j.Kc;
        double* dst = r < erows ? j.E + ((long)(l + 1) * j.NP + r) * j.Kc : j.W + (r - erows + wrows) * j.Kc;
        double2 v = make_double2(0.0, 0.0);
        if (c >= j.NP && q < HQ) {
            const double s0 = src[c], s1 = src[c + 1], si = rot[2 * q], co = rot[2 * q + 1];
            v = make_double2(s0 * co - s1 * si, s0 * si + s1 * co);
        }
        *reinterpret_cast<double2*>(dst + c) = v;
    }
}

// D u of the block's steps into W: step i reads sample 2 i (RK4) or i + 3 (ABM).
__global__ void __launch_bounds__(kThreads) k_expand_feed_batch(const ExpandJob* __restrict__ jobs)
{
    const ExpandJob j = jobs[blockIdx.y];
    if (j.zeroD) return;
    const int HQ = j.H / 2;
    for (long e = (long)blockIdx.x * kThreads + threadIdx.x; e < ((long)HQ << j.R); e += (long)gridDim.x * kThreads) {
        const long i = e / HQ;
        const int q = (int)(e - i * HQ);
        double si, co;
        sincos(__dmul_rn(__dmul_rn(kTwoPi, j.freq[q]), j.dt) * (double)(j.solver == 0 ? 2 * i : i + 3), &si, &co);
        for (int o = 0; o < j.p; ++o) {
            const double d = j.D[(long)o * j.mu + q / j.terms] * j.amp[q];
            double* w = j.W + (i * j.p + o) * j.Kc + j.NP + 2 * q;
            w[0] += d * co;
            w[1] += d * si;
        }
    }
}

__global__ void __launch_bounds__(kThreads) k_expand_phases_batch(const ExpandJob* __restrict__ jobs)
{
    const ExpandJob j = jobs[blockIdx.y];
    const int pairs = (j.Kc - j.NP) / 2, HQ = j.H / 2;
    const long total = j.nblocks * pairs;
    const long e0 = (long)blockIdx.x * kThreads + threadIdx.x, step = (long)gridDim.x * kThreads;
    for (long e = e0; e < j.NP; e += step) j.Z[e] = j.X0[e];
    for (long e = e0; e < total; e += step) {
        const long b = e / pairs;
        const int q = (int)(e - b * pairs);
        double si = 0.0, co = 0.0;
        if (q < HQ) {
            const double ts = sample_time(j.base, j.dt, b * j.stride);
            sincos(__dadd_rn(__dmul_rn(__dmul_rn(kTwoPi, j.freq[q]), ts), j.phi[q]), &si, &co);
        }
        *reinterpret_cast<double2*>(j.Z + b * j.Kc + j.NP + 2 * q) = make_double2(si, co);
    }
}

// dst(g, r) = sum_k P[r][k] src(g, k) (+ acc): CTA = 8 rows x 32 columns g, its four
// warps a quarter of K each (fragments straight from L2, two K values per
// load), the quarters summed in order.  Latency-bound, so a warp has the
// loads of kBatch K chunks in flight before their products.  A level of one
// system with NP = 512, Kc = 608 and up to 32 columns is 64 CTAs instead of 8
// of the 64 x 64 tiles (19 us, mostly padding).
constexpr int kNarrowThreads = 128, kNarrowCols = 32;

template <int CT>
__device__ __forceinline__ void narrow_mma(const double* pr, const double* const (&z)[4], int k0, int k1,
                                           double (&acc)[4][2])
{
    constexpr int kBatch = CT == 1 ? 8 : CT == 2 ? 6 : 4;
    for (int k = k0; k < k1; k += kBatch) {
        double2 e[kBatch], v[kBatch][CT];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int kk = 8 * min(k + u, k1 - 1);  // chunks past the end load the last one and are not used
            e[u] = *reinterpret_cast<const double2*>(pr + kk);
#pragma unroll
            for (int c = 0; c < CT; ++c) v[u][c] = *reinterpret_cast<const double2*>(z[c] + kk);
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u)
#pragma unroll
            for (int c = 0; c < CT; ++c) {
                if (k + u >= k1) continue;
                dmma_m8n8k4(acc[c][0], acc[c][1], v[u][c].x, e[u].x);
                dmma_m8n8k4(acc[c][0], acc[c][1], v[u][c].y, e[u].y);
            }
    }
}

// kSplit: CTA = 8 rows, a quarter of K a warp; else a row tile a warp, its whole
// K.  The first level of a thousand systems (133 MB of powers, 20 us): 79 us in
// 9.7 K split CTAs that each bisected the entries, 60 with find_entry, 46 a row
// tile a warp; later levels of as many bytes 75, 39.
template <bool kSplit>
__global__ void __launch_bounds__(kNarrowThreads) k_expand_narrow(const LevelArgs* __restrict__ args,
                                                                  const long* __restrict__ start, int nent)
{
    __shared__ double2 red[kSplit ? 4 : 1][4][32];
    const long t = blockIdx.x;
    const int lo = find_entry(start, nent, t);
    const LevelArgs& a = args[lo];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, tq = lane & 3;
    const int rows = level_rows(a), rt = kSplit ? rows / 8 : (rows + 31) / 32;
    const long u = t - start[lo], c0 = (u / rt) * kNarrowCols;
    const int r0 = kSplit ? (int)(u % rt) * 8 : (int)(u % rt) * 32 + 8 * warp;
    if (!kSplit && r0 >= rows) return;
    const int cols = (int)min((long)kNarrowCols, a.ncols - c0), ct = (cols + 7) / 8;
    const int n8 = level_k(a) / 8, k0 = kSplit ? n8 * warp / 4 : 0, k1 = kSplit ? n8 * (warp + 1) / 4 : n8;
    const double* pr = a.P + (long)(r0 + g) * a.ldp + 2 * tq;
    const double* z[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) z[c] = a.src + (c0 + (8 * c + g < cols ? 8 * c + g : 0)) * a.src_gs + 2 * tq;
    double acc[4][2] = {};
    switch (ct) {
    case 1: narrow_mma<1>(pr, z, k0, k1, acc); break;
    case 2: narrow_mma<2>(pr, z, k0, k1, acc); break;
    case 3: narrow_mma<3>(pr, z, k0, k1, acc); break;
    default: narrow_mma<4>(pr, z, k0, k1, acc); break;
    }
    auto store = [&](int c, double2 v) {  // column tile c
        if (a.acc) {
            const double2 o = *reinterpret_cast<const double2*>(a.acc + (c0 + 8 * c + g) * a.acc_gs + r0 + 2 * tq);
            v.x += o.x;
            v.y += o.y;
        }
        *reinterpret_cast<double2*>(a.dst + (c0 + 8 * c + g) * a.dst_gs + r0 + 2 * tq) = v;
    };
    if constexpr (kSplit) {
#pragma unroll
        for (int c = 0; c < 4; ++c) red[warp][c][lane] = make_double2(acc[c][0], acc[c][1]);
        __syncthreads();
        if (8 * warp + g < cols) {  // this warp stores column tile `warp`
            double2 v = red[0][warp][lane];
#pragma unroll
            for (int w = 1; w < 4; ++w) {
                v.x += red[w][warp][lane].x;
                v.y += red[w][warp][lane].y;
            }
            store(warp, v);
        }
    } else {
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if (8 * c + g < cols) store(c, make_double2(acc[c][0], acc[c][1]));
    }
}

// x extent of a batched launch: a few CTAs a job, about 2048 in all when the jobs are few.
unsigned batch_x(long max_elems, int njobs)
{
    const long want = std::max<long>(4, (2048 + njobs - 1) / njobs);
    return (unsigned)std::max<long>(1, std::min<long>((max_elems + kThreads - 1) / kThreads, want));
}

template <int KS>
void level_t(const ExpandTables& t, const double* T, double* Z, int imax, long d, cudaStream_t s)
{
    // columns per CTA: one 8-column tile while that leaves CTAs for the whole
    // chip, up to four beyond (the table fragments are loaded once)
    const long tiles = (d + 7) / 8;
    const int ct = (int)std::max<long>(1, std::min<long>(kLevelTiles, tiles * imax / kSmCount));
    dim3 grid((unsigned)((tiles + ct - 1) / ct), (unsigned)imax);
    launch_dependent(k_expand_level<KS>, grid, dim3(kThreads), 0, s, T, Z, d, t.sh.nblocks, t.sh.NP, ct);
}

template <int KS>
void out_t(const ExpandTables& t, const double* Z, double* Y, long c0, long c1, long limit, int sms, cudaStream_t s)
{
    using C = OutCfg<KS>;
    const int M = t.sh.rows(), ld = smem_pitch(t.sh.Kc);
    const int cap = (int)(kSmemMax / (ld * sizeof(double))) / 8, tiles8 = (M + 7) / 8;  // row tiles: of a slice, of W
    const long nt = (c1 - c0 + 8 * C::CT - 1) / (8 * C::CT);
    const int warps = C::threads / 32;
    // Slices of W: cycles to stage one (a CTA draws about 32 bytes a cycle with
    // all SMs reading), to fetch a warp's blocks (500 for each tile it starts)
    // and for its products (three warps share a sub-partition).  A slice
    // as large as fits staged 147 KB for 98 tiles of a free response of 24
    // states, 10^5 steps, and dealt out whole tiles: the solve took 20.6 us,
    // 16.0 in 16 slices; 64 states, 2^20 steps, mixed 116.6, 108.5 in 4 for 3.
    int slices = (tiles8 + cap - 1) / cap;
    double best = 1e300;
    for (int k = slices, end = std::min(tiles8, std::max(slices, std::min(sms, 40))); k <= end; ++k) {
        const int rt = (tiles8 + k - 1) / k;
        const double per = std::ceil((double)nt * rt / ((long)std::max(1, sms / k) * warps));
        const double cost = 2.0 * rt * t.sh.Kc + 500.0 * (per / rt + 1.0) + per * (warps / 4) * 16.0 * C::CT * KS;
        if (cost < best) best = cost, slices = k;
    }
    const int Ms = (tiles8 + slices - 1) / slices * 8;
    slices = (M + Ms - 1) / Ms;
    const size_t smem = (size_t)Ms * ld * sizeof(double);
    PARODE_CUDA(cudaFuncSetAttribute(k_expand_out<KS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax));
    // CTAs: no more than the SMs, each with at least a row tile per warp
    const long ctas = std::max<long>(slices, std::min<long>(sms, nt * tiles8 / warps));
    const long gs = M;
    const int vec = ((reinterpret_cast<uintptr_t>(Y) & 15) == 0 && (gs & 1) == 0) ? 1 : 0;
    launch_dependent(k_expand_out<KS>, dim3((unsigned)ctas), dim3(C::threads), smem, s, t.W, M, Ms, slices, Z, Y, gs, c0,
                     c1, limit, vec);
}

template <class F>
void by_width(int Kc, F&& f)
{
    switch (Kc) {
    case 8: return f(std::integral_constant<int, 2>());
    case 16: return f(std::integral_constant<int, 4>());
    case 24: return f(std::integral_constant<int, 6>());
    case 32: return f(std::integral_constant<int, 8>());
    case 40: return f(std::integral_constant<int, 10>());
    case 48: return f(std::integral_constant<int, 12>());
    case 56: return f(std::integral_constant<int, 14>());
    case 64: return f(std::integral_constant<int, 16>());
    case 80: return f(std::integral_constant<int, 20>());
    case 96: return f(std::integral_constant<int, 24>());
    case 112: return f(std::integral_constant<int, 28>());
    case 128: return f(std::integral_constant<int, 32>());
    case 144: return f(std::integral_constant<int, 36>());
    case 160: return f(std::integral_constant<int, 40>());
    default: throw Error(kInvalidArgument, "expansion: unsupported width");
    }
}

}  // namespace

long ExpandShape::table_rows() const
{
    long r = 0;
    for (int l = 0; l < levels; ++l) r += (long)imax[l] * NP;
    return r;
}

bool expand_shape(int Ns, int mu, int terms, int p, long nScan, int R, ExpandShape* out)
{
    ExpandShape s;
    s.NP = (int)round_up(Ns, 8);
    s.H = 2 * mu * terms;
    if (s.NP > 64 || (long)mu * terms > 256) return false;
    for (int w : kWidths)
        if (w >= s.NP + s.H) {
            s.Kc = w;
            break;
        }
    if (s.Kc == 0) return false;
    s.R = R;
    s.B = 1 << R;
    s.p = p;
    s.nblocks = (nScan + s.B - 1) / s.B;
    s.pow_levels = R;  // W's rows need E(2^0) .. E(2^(R-1))
    long d = 1;
    while (d < s.nblocks) {
        if (s.levels == kExpandMaxLevels) return false;
        const long i = std::min<long>(kExpandRadix - 1, (s.nblocks - 1) / d);
        s.imax[s.levels] = (int)i;
        int bits = 0;
        while ((i >> bits) != 0) ++bits;
        s.pow_levels = R + 4 * s.levels + bits;
        ++s.levels;
        d *= kExpandRadix;
    }
    s.pow_levels = std::max(s.pow_levels, 1);
    *out = s;
    return true;
}

void launch_expand_tables(const ExpandTables& t, cudaStream_t s)
{
    const int maxown = ((t.sh.Kc - t.sh.NP) / 8 + kSqCtas - 1) / kSqCtas;
    size_t smem = (2 * (size_t)t.sh.NP * (t.sh.NP + 4 + 8 * maxown + 4) + 8 * maxown) * sizeof(double);
    PARODE_CUDA(cudaFuncSetAttribute(k_expand_squarings, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax));
    k_expand_squarings<<<kSqCtas, kThreads, smem, s>>>(t);
    PARODE_CUDA(cudaGetLastError());
    const int out_tiles = (t.sh.rows() + 7) / 8;
    const long tiles = out_tiles + t.sh.table_rows() / 8;
    smem = 2 * 8 * (size_t)smem_pitch(t.sh.Kc) * sizeof(double);
    k_expand_rows<<<(unsigned)tiles, kThreads, smem, s>>>(t, out_tiles);
    PARODE_CUDA(cudaGetLastError());
}

int launch_expand_states(const ExpandTables& t, const double* X0, double* Z, double base, long stride, cudaStream_t s)
{
    const long pairs = (t.sh.Kc - t.sh.NP) / 2;
    const long threads = std::max<long>(t.sh.NP, t.sh.nblocks * pairs);
    k_expand_phases<<<(unsigned)((threads + kThreads - 1) / kThreads), kThreads, 0, s>>>(
        Z, X0, t.par, t.sh.NP, t.sh.Kc, t.sh.H / 2, base, t.dt, stride, t.sh.nblocks);
    PARODE_CUDA(cudaGetLastError());
    const double* T = t.T;
    long d = 1;
    for (int l = 0; l < t.sh.levels; ++l, d *= kExpandRadix) {
        by_width(t.sh.Kc, [&](auto ks) { level_t<decltype(ks)::value>(t, T, Z, t.sh.imax[l], d, s); });
        T += (long)t.sh.imax[l] * t.sh.NP * t.sh.Kc;
    }
    return 1 + t.sh.levels;
}

void launch_expand_out(const ExpandTables& t, const double* Z, double* Y, long c0, long c1, long limit, int sms,
                       cudaStream_t s)
{
    if (c1 <= c0) return;
    by_width(t.sh.Kc, [&](auto ks) { out_t<decltype(ks)::value>(t, Z, Y, c0, c1, limit, sms, s); });
}

int expand_log2_block(int NP, int Kc, int p, long nScan, double executions)
{
    int best = 3;
    double best_cost = -1.0;
    for (int R = 3; R <= 7; ++R) {
        const double B = (double)(1 << R);
        if (R > 3 && B / 2 >= (double)nScan) break;
        if (R > 3 && 8.0 * B * p * Kc > 256e6) break;
        const double build = executions > 0 ? 2.0 * B * p * NP * Kc / ((double)nScan * executions) : 0.0;
        const double cost = 2.0 * NP * Kc / B + build;
        if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            best = R;
        }
    }
    return best;
}

void launch_expand_init(const ExpandJob* dJobs, int njobs, int max_hq, long max_elems, cudaStream_t s)
{
    // within the 48 KB that need no limit of the function's own
    static_assert(sizeof(double) * 2 * 5 * kExpandMaxPairs <= 48 * 1024, "trig table");
    const size_t smem = sizeof(double) * 2 * 5 * (size_t)std::max(max_hq, 1);
    k_expand_init_batch<<<dim3(batch_x(max_elems, njobs), (unsigned)njobs), kThreads, smem, s>>>(dJobs);
    PARODE_CUDA(cudaGetLastError());
}

void launch_expand_rot(const ExpandJob* dJobs, int njobs, int l, long max_elems, cudaStream_t s)
{
    k_expand_rot_batch<<<dim3(batch_x(max_elems, njobs), (unsigned)njobs), kThreads, 0, s>>>(dJobs, l);
    PARODE_CUDA(cudaGetLastError());
}

void launch_expand_feed(const ExpandJob* dJobs, int njobs, long max_elems, cudaStream_t s)
{
    k_expand_feed_batch<<<dim3(batch_x(max_elems, njobs), (unsigned)njobs), kThreads, 0, s>>>(dJobs);
    PARODE_CUDA(cudaGetLastError());
}

int expand_power_args(const ExpandJob& j, int l, LevelArgs out[2])
{
    int c = 0;
    const double* El = j.E + (long)l * j.NP * j.Kc;
    LevelArgs a;  // [Phi^(2^l) as rows] x E(2^l), onto the rotation part
    a.P = El;
    a.ldp = j.Kc;
    a.Np = j.NP;
    a.M = j.NP;
    a.K = j.NP;
    a.ncols = j.Kc;
    a.src = El;
    a.src_gs = 1;
    a.src_ks = j.Kc;
    a.acc_gs = a.dst_gs = 1;
    a.acc_is = a.dst_is = j.Kc;
    if (l + 1 < j.pow_levels) {
        a.dst = j.E + (long)(l + 1) * j.NP * j.Kc;
        a.acc = a.dst;
        out[c++] = a;
    }
    if (l < j.R) {
        a.P = j.W;
        a.M = j.p << l;
        a.dst = j.W + ((long)j.p << l) * j.Kc;
        a.acc = a.dst;
        out[c++] = a;
    }
    return c;
}

void launch_expand_phases(const ExpandJob* dJobs, int njobs, long max_elems, cudaStream_t s)
{
    k_expand_phases_batch<<<dim3(batch_x(max_elems, njobs), (unsigned)njobs), kThreads, 0, s>>>(dJobs);
    PARODE_CUDA(cudaGetLastError());
}

LevelArgs expand_level_args(const ExpandJob& j, int l)
{
    const long d = 1L << l;
    LevelArgs a;
    a.P = j.E + (long)(j.R + l) * j.NP * j.Kc;
    a.ldp = j.Kc;
    a.Np = j.NP;
    a.M = j.NP;
    a.K = j.Kc;
    a.ncols = std::min(d, j.nblocks - d);
    a.src = j.Z;
    a.src_gs = j.Kc;
    a.src_ks = 1;
    a.dst = j.Z + d * j.Kc;
    a.dst_gs = j.Kc;
    a.dst_is = 1;
    return a;
}

LevelArgs expand_out_args(const ExpandJob& j, double* Y, long limit)
{
    LevelArgs a;
    a.P = j.W;
    a.ldp = j.Kc;
    a.Np = j.NP;
    a.M = j.p << j.R;
    a.K = j.Kc;
    a.ncols = j.nblocks;
    a.src = j.Z;
    a.src_gs = j.Kc;
    a.src_ks = 1;
    a.dst = Y;
    a.dst_gs = a.M;
    a.dst_is = 1;
    a.dst_limit = limit;
    return a;
}

long expand_narrow_tiles(const LevelArgs& a, bool split)
{
    return (long)(split ? level_rows(a) / 8 : (level_rows(a) + 31) / 32) * ((a.ncols + kNarrowCols - 1) / kNarrowCols);
}

void launch_expand_narrow(const LevelArgs* dArgs, const long* dStart, int nent, long tiles, bool split, cudaStream_t s)
{
    if (tiles <= 0) return;
    if (split) k_expand_narrow<true><<<(unsigned)tiles, kNarrowThreads, 0, s>>>(dArgs, dStart, nent);
    else k_expand_narrow<false><<<(unsigned)tiles, kNarrowThreads, 0, s>>>(dArgs, dStart, nent);
    PARODE_CUDA(cudaGetLastError());
}

}  // namespace parode
