// kernels_general.cu -- the general affine scan: a distinct map per step.
//
// The reference composes a distinct matrix at every tree node of a
// level-by-level scan (Kernels/MMKernelScanUpsweep.cl:13-56,
// Kernels/MVVKernelScanUpsweep.cl:14-50, MVVKernelScanDownsweep.cl:14-50),
// every level a pass over the maps.  Here x_{k+1} = M_k x_k + v_k runs over a
// hierarchy of chunks: the compositions of each chunk's maps (up, M_k .. M_j
// and the matching vectors: the same products, one after another), the same
// on the chunks' maps until few are left, and back down, each chunk's states
// from the state entering it.  The maps are read twice from the caller's
// array (once up, once down) and never copied or padded; a level has 1/16 of
// the maps below it, so nothing else is large.  16 states, 2^16 steps: two
// reads of 134 MB, and 2 NP^3 flop per step for the compositions; 0.49 ms per
// call by levels of pairs, 0.136 ms by chunks (lowest level 33 + 32 us of
// 21 + 21 at the copy rate, the rest the latency of the two upper levels).
// 64 states, 2^15 steps: 0.84 ms, 0.46 of it the DMMA floor; the 3xTF32
// compositions that the mixed form ran at scan dimensions 32 and 64 took
// longer than this, so it runs the FP64 products too.
#include "common.h"
#include "device_common.cuh"
#include "general.h"

#include <algorithm>
#include <type_traits>

namespace parode {

namespace {

// The product Q <- M_k Q of a chunk on the FP64 tensor cores, transposed:
// Q^T <- Q^T M_k^T.  The m8n8k4 result tile of Q^T (rows: Q's columns) then
// already is the next step's A operand, if product 2 c + u of a K chunk of 8
// takes the K indices 8 c + 2 t + u: no shuffle, no shared memory.  The B
// operand of M_k^T with that order is two consecutive elements of a row of
// M_k.  The vector part w <- M_k w + v_k runs on the CUDA cores from the same
// elements (as a ninth row tile with one row in use it cost the products of a
// whole one and left the warps uneven: NP = 64, 2^15 maps, 0.88 ms for level
// 0 alone).
//
// Lane = 4 g + t.  q[mt][nt][u] = Q^T[8 mt + g][8 nt + 2 t + u].  Every kernel
// is launched as a dependent of the one before it.

// NP = 8 or 16: a warp alone per chunk, M_k's fragments straight from global
// memory, kAhead steps in flight (more where the chunks are few and a step's
// load latency is what counts: kDeep chunks and fewer).
constexpr long kDeep = kSmCount * 4;

template <int NP, bool kFull, int kAhead>
__global__ void __launch_bounds__(128) k_scan_up_warp(const double* M, const double* V, int ns, long count, int L,
                                                      long nch, double* Mo, double* Vo)
{
    constexpr int MT = NP / 8;
    grid_dep_wait();  // the maps, from the second level on
    grid_dep_trigger();
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const long c = (long)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (c >= nch) return;
    const long k0 = c * L, k1 = min(count, k0 + L);
    auto el = [&](long k, int r, int col) {
        if (kFull) return M[(k * NP + r) * NP + col];
        return r < ns && col < ns ? M[(k * ns + r) * ns + col] : 0.0;
    };
    auto pair = [&](long k, int r, int col) {
        if (kFull) return *reinterpret_cast<const double2*>(M + (k * NP + r) * NP + col);
        return make_double2(el(k, r, col), el(k, r, col + 1));
    };
    auto vec = [&](long k, int r) { return V && (kFull || r < ns) ? V[k * ns + r] : 0.0; };
    double2 b[kAhead][MT][MT];
    double v[kAhead][MT];  // row 8 nt + g
    auto load = [&](int a, long k) {
#pragma unroll
        for (int nt = 0; nt < MT; ++nt) {
#pragma unroll
            for (int cc = 0; cc < MT; ++cc) b[a][nt][cc] = pair(k, 8 * nt + g, 8 * cc + 2 * t);
            v[a][nt] = vec(k, 8 * nt + g);
        }
    };
    // steps past the end load the last one and are not used
#pragma unroll
    for (int a = 0; a < kAhead; ++a) load(a, min(k0 + 1 + a, k1 - 1));
    double q[MT][MT][2], w[MT][2];  // w[cc][u]: element 8 cc + 2 t + u
#pragma unroll
    for (int nt = 0; nt < MT; ++nt)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) q[mt][nt][u] = el(k0, 8 * nt + 2 * t + u, 8 * mt + g);
            w[nt][u] = vec(k0, 8 * nt + 2 * t + u);
        }
    for (long k = k0 + 1; k < k1; k += kAhead)
#pragma unroll
        for (int a = 0; a < kAhead; ++a) {
            if (k + a >= k1) break;
            double n[MT][MT][2] = {}, y[MT];
#pragma unroll
            for (int nt = 0; nt < MT; ++nt) {
                y[nt] = t == 0 ? v[a][nt] : 0.0;
#pragma unroll
                for (int cc = 0; cc < MT; ++cc)
                    y[nt] = fma(b[a][nt][cc].x, w[cc][0], fma(b[a][nt][cc].y, w[cc][1], y[nt]));
            }
#pragma unroll
            for (int cc = 0; cc < MT; ++cc)
#pragma unroll
                for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                    for (int nt = 0; nt < MT; ++nt) {
                        dmma_m8n8k4(n[mt][nt][0], n[mt][nt][1], q[mt][cc][0], b[a][nt][cc].x);
                        dmma_m8n8k4(n[mt][nt][0], n[mt][nt][1], q[mt][cc][1], b[a][nt][cc].y);
                    }
            load(a, min(k + a + kAhead, k1 - 1));
#pragma unroll
            for (int nt = 0; nt < MT; ++nt) {
                y[nt] += __shfl_xor_sync(0xffffffffu, y[nt], 1);
                y[nt] += __shfl_xor_sync(0xffffffffu, y[nt], 2);
#pragma unroll
                for (int u = 0; u < 2; ++u) w[nt][u] = __shfl_sync(0xffffffffu, y[nt], 4 * (2 * t + u));
            }
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                for (int nt = 0; nt < MT; ++nt) q[mt][nt][0] = n[mt][nt][0], q[mt][nt][1] = n[mt][nt][1];
        }
#pragma unroll
    for (int nt = 0; nt < MT; ++nt)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int r = 8 * nt + 2 * t + u;
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) Mo[(c * NP + r) * NP + 8 * mt + g] = q[mt][nt][u];
            if (g == 0) Vo[c * NP + r] = w[nt][u];
        }
}

// Rows of M x dealt to W warps: eight lanes share a row (two consecutive
// elements each per 16 columns: a warp reads four rows of 128 consecutive
// bytes), row group i of warp w holds rows 4 (w + W i) .. + 3.
template <int NP, int W>
struct RowSplit {
    static constexpr int G = (NP / 4 + W - 1) / W, NI = (NP + 15) / 16;
};

template <int G>
__device__ __forceinline__ void add_lanes(double (&y)[G])
{
#pragma unroll
    for (int o = 1; o < 8; o <<= 1)
#pragma unroll
        for (int i = 0; i < G; ++i) y[i] += __shfl_xor_sync(0xffffffffu, y[i], o);
}

// NP = 24 .. 64: a CTA per chunk, each warp two row tiles of Q^T, M_k staged
// in shared memory by cp.async kStages deep.  FP64-tensor bound from NP = 40
// on (NP = 64: 1024 products a step).
template <int NP>
struct UpCfg {
    static constexpr int MT = NP / 8, warps = (MT + 1) / 2, threads = 32 * warps;
    static constexpr int pitch = NP % 16 == 8 ? NP : NP + 8;  // 8 mod 16 doubles: conflict-free 16-byte fragments
    static constexpr int stages = NP <= 32 ? 3 : 2;
    static constexpr int words = NP * pitch + NP;  // M_k, then v_k
    static constexpr int wlen = (NP + 15) / 16 * 16;
    static constexpr size_t smem = sizeof(double) * (stages * words + 2 * wlen);
};

template <int BYTES>
__device__ __forceinline__ void cp_async(double* dst, const double* src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}

template <int NP, bool kFull>
__global__ void __launch_bounds__(UpCfg<NP>::threads) k_scan_up_cta(const double* M, const double* V, int ns, long count,
                                                                    int L, double* Mo, double* Vo)
{
    using C = UpCfg<NP>;
    using R = RowSplit<NP, C::warps>;
    constexpr int MT = C::MT, ld = C::pitch, kS = C::stages;
    extern __shared__ __align__(16) double sm[];
    double* wb = sm + kS * C::words;  // w, two copies
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int s8 = lane & 7, rr = lane >> 3;
    const long c = blockIdx.x, k0 = c * L, k1 = min(count, k0 + L);
    // the padding (and an absent V) stays zero: the copies write only ns x ns and ns
    if (!kFull || !V)
        for (int e = tid; e < kS * C::words; e += C::threads) sm[e] = 0.0;
    for (int e = tid; e < 2 * C::wlen; e += C::threads) wb[e] = 0.0;
    __syncthreads();
    grid_dep_wait();  // the maps, from the second level on
    grid_dep_trigger();
    auto load = [&](long k, double* s) {
        if (kFull) {
            for (int e = tid; e < NP * (NP / 2); e += C::threads) {
                const int r = e / (NP / 2), col = 2 * (e - r * (NP / 2));
                cp_async<16>(s + r * ld + col, M + (k * NP + r) * NP + col);
            }
        } else {
            for (int e = tid; e < ns * ns; e += C::threads) {
                const int r = e / ns;
                cp_async<8>(s + r * ld + (e - r * ns), M + k * ns * ns + e);
            }
        }
        if (V)
            for (int e = tid; e < ns; e += C::threads) cp_async<8>(s + NP * ld + e, V + k * ns + e);
    };
#pragma unroll
    for (int s = 0; s < kS - 1; ++s) {
        if (k0 + s < k1) load(k0 + s, sm + s * C::words);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    const int m0 = 2 * warp;
    const bool two = m0 + 1 < MT;  // the last warp of an odd count has one row tile
    double q[2][MT][2];
    int cur = 0, slot = 0;
    for (long k = k0; k < k1; ++k) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kS - 2) : "memory");
        __syncthreads();
        {
            const int nx = slot == 0 ? kS - 1 : slot - 1;
            if (k + kS - 1 < k1) load(k + kS - 1, sm + nx * C::words);
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        }
        const double* s = sm + slot * C::words;
        const double* sv = s + NP * ld;
        slot = slot + 1 == kS ? 0 : slot + 1;
        if (k == k0) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int nt = 0; nt < MT; ++nt)
#pragma unroll
                    for (int u = 0; u < 2; ++u)
                        q[i][nt][u] = i == 0 || two ? s[(8 * nt + 2 * t + u) * ld + 8 * (m0 + i) + g] : 0.0;
            for (int e = tid; e < NP; e += C::threads) wb[e] = sv[e];
            continue;
        }
        double n[2][MT][2] = {}, y[R::G];
        // the vector part first: its shuffles run beside the products
#pragma unroll
        for (int i = 0; i < R::G; ++i) y[i] = 0.0;
#pragma unroll
        for (int j = 0; j < R::NI; ++j) {
            const double2 x = *reinterpret_cast<const double2*>(wb + cur * C::wlen + 16 * j + 2 * s8);
#pragma unroll
            for (int i = 0; i < R::G; ++i) {
                const int r = 4 * (warp + C::warps * i) + rr;
                if (r < NP && 16 * j + 2 * s8 < NP) {
                    const double2 m = *reinterpret_cast<const double2*>(s + r * ld + 16 * j + 2 * s8);
                    y[i] = fma(m.x, x.x, fma(m.y, x.y, y[i]));
                }
            }
        }
        add_lanes<R::G>(y);
#pragma unroll
        for (int i = 0; i < R::G; ++i) {
            const int r = 4 * (warp + C::warps * i) + rr;
            if (s8 == 0 && r < NP) wb[(cur ^ 1) * C::wlen + r] = y[i] + sv[r];
        }
        cur ^= 1;
#pragma unroll
        for (int cc = 0; cc < MT; ++cc)
#pragma unroll
            for (int nt = 0; nt < MT; ++nt) {
                const double2 b = *reinterpret_cast<const double2*>(s + (8 * nt + g) * ld + 8 * cc + 2 * t);
                dmma_m8n8k4(n[0][nt][0], n[0][nt][1], q[0][cc][0], b.x);
                if (two) dmma_m8n8k4(n[1][nt][0], n[1][nt][1], q[1][cc][0], b.x);
                dmma_m8n8k4(n[0][nt][0], n[0][nt][1], q[0][cc][1], b.y);
                if (two) dmma_m8n8k4(n[1][nt][0], n[1][nt][1], q[1][cc][1], b.y);
            }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int nt = 0; nt < MT; ++nt) q[i][nt][0] = n[i][nt][0], q[i][nt][1] = n[i][nt][1];
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 2; ++i)
        if (i == 0 || two)
#pragma unroll
            for (int nt = 0; nt < MT; ++nt)
#pragma unroll
                for (int u = 0; u < 2; ++u) Mo[(c * NP + 8 * nt + 2 * t + u) * NP + 8 * (m0 + i) + g] = q[i][nt][u];
    for (int e = tid; e < NP; e += C::threads) Vo[c * NP + e] = wb[cur * C::wlen + e];
}

// States of a chunk from the one entering it: X[k] = x_k, x_{k+1} = M_k x_k +
// v_k.  W warps per chunk, rows dealt as RowSplit; three shuffles add a row up
// and the next state goes through shared memory.  Each step's M and v are
// loaded kAhead steps before its states are stored, so X may be V.  HBM-bound
// at the lowest level (every map is read once), latency-bound above it.
template <int NP>
struct DownCfg {
    static constexpr int warps = (NP + 15) / 16;
    static constexpr int deep = NP <= 16 ? 4 : NP <= 32 ? 2 : 1;  // steps in flight where the chunks are few
    static constexpr int chunks = warps == 1 ? 4 : 1;  // per CTA
    static constexpr int threads = 32 * warps * chunks;
};

template <int NP, bool kFull, int kAhead>
__global__ void __launch_bounds__(DownCfg<NP>::threads) k_scan_down(const double* M, const double* V, int ns, long count,
                                                                    int L, long nchunks, const double* starts, int ss,
                                                                    double* X)
{
    using C = DownCfg<NP>;
    using R = RowSplit<NP, C::warps>;
    __shared__ __align__(16) double xs[C::chunks][2][R::NI * 16];
    const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) % C::warps, ch = (threadIdx.x >> 5) / C::warps;
    const int s = lane & 7, rr = lane >> 3, ct = threadIdx.x - ch * 32 * C::warps;  // thread of the chunk
    grid_dep_wait();  // the states entering the chunks
    grid_dep_trigger();
    const long c = (long)blockIdx.x * C::chunks + ch;
    if (c >= nchunks) return;  // whole warps; with several warps a CTA has one chunk
    auto sync = [&] {
        if (C::warps == 1) __syncwarp();
        else __syncthreads();
    };
    const long k0 = c * L, k1 = min(count, k0 + L);
    double2 m[kAhead][R::G][R::NI];
    double v[kAhead][R::G];
    auto load = [&](int a, long k) {
        if (k + 1 >= k1) return;  // the last map of a chunk belongs to the next chunk's first state
#pragma unroll
        for (int i = 0; i < R::G; ++i) {
            const int r = 4 * (w + C::warps * i) + rr;
            v[a][i] = V && s == 0 && r < ns ? V[k * ns + r] : 0.0;
#pragma unroll
            for (int j = 0; j < R::NI; ++j) {
                const int col = 16 * j + 2 * s;
                double2 x = make_double2(0.0, 0.0);
                if (kFull) {
                    if (r < NP && col < NP) x = *reinterpret_cast<const double2*>(M + (k * NP + r) * NP + col);
                } else if (r < ns) {
                    if (col < ns) x.x = M[(k * ns + r) * ns + col];
                    if (col + 1 < ns) x.y = M[(k * ns + r) * ns + col + 1];
                }
                m[a][i][j] = x;
            }
        }
    };
#pragma unroll
    for (int a = 0; a < kAhead; ++a) load(a, k0 + a);
    for (int e = ct; e < R::NI * 16; e += 32 * C::warps) {
        xs[ch][0][e] = e < min(ns, ss) && starts ? starts[c * ss + e] : 0.0;  // ss < ns: the caller's x0 at a padded level
        xs[ch][1][e] = 0.0;
    }
    sync();
    int cur = 0;
    for (long k = k0; k < k1; k += kAhead)
#pragma unroll
        for (int a = 0; a < kAhead; ++a) {
            if (k + a >= k1) break;
            const double* x = xs[ch][cur];
            if (k + a + 1 < k1) {
                double y[R::G];
#pragma unroll
                for (int i = 0; i < R::G; ++i) y[i] = v[a][i];
#pragma unroll
                for (int j = 0; j < R::NI; ++j) {
                    const double2 xv = *reinterpret_cast<const double2*>(x + 16 * j + 2 * s);
#pragma unroll
                    for (int i = 0; i < R::G; ++i) y[i] = fma(m[a][i][j].x, xv.x, fma(m[a][i][j].y, xv.y, y[i]));
                }
                load(a, k + a + kAhead);
                add_lanes<R::G>(y);
#pragma unroll
                for (int i = 0; i < R::G; ++i) {
                    const int r = 4 * (w + C::warps * i) + rr;
                    if (s == 0 && r < ns) xs[ch][cur ^ 1][r] = y[i];
                }
            }
            for (int e = ct; e < ns; e += 32 * C::warps) X[(k + a) * ns + e] = x[e];
            sync();
            cur ^= 1;
        }
}

// Ms[k] = Phi for k < count (the reference's DistributeA, Kernels/DistributeA.cl:6-13).
__global__ void k_distribute(double* __restrict__ Ms, const double* __restrict__ Phi, int NP, long count)
{
    const long per = (long)NP * NP;
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < count * per; e += (long)gridDim.x * blockDim.x)
        Ms[e] = Phi[e % per];
}

unsigned grid_for(long work, int per, int cap)
{
    return (unsigned)std::max<long>(1, std::min<long>((work + per - 1) / per, cap));
}

template <int NP, bool kFull>
void up_t(const ScanLevel& l, long nch, double* Mo, double* Vo, cudaStream_t s)
{
    if constexpr (NP <= 16) {
        auto* k = nch <= kDeep ? k_scan_up_warp<NP, kFull, NP == 8 ? 6 : 4> : k_scan_up_warp<NP, kFull, 2>;
        launch_dependent(k, dim3((unsigned)((nch + 3) / 4)), dim3(128), 0, s, l.M, l.V, l.ns, l.count, l.L, nch, Mo, Vo);
    } else {
        using C = UpCfg<NP>;
        PARODE_CUDA(cudaFuncSetAttribute(k_scan_up_cta<NP, kFull>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)C::smem));
        launch_dependent(k_scan_up_cta<NP, kFull>, dim3((unsigned)nch), dim3(C::threads), C::smem, s, l.M, l.V, l.ns,
                         l.count, l.L, Mo, Vo);
    }
}

template <int NP, bool kFull>
void down_t(const ScanLevel& l, const double* starts, int ss, cudaStream_t s)
{
    using C = DownCfg<NP>;
    const long nch = (l.count + l.L - 1) / l.L;
    auto* k = nch <= kDeep ? k_scan_down<NP, kFull, C::deep> : k_scan_down<NP, kFull, 1>;
    launch_dependent(k, dim3((unsigned)((nch + C::chunks - 1) / C::chunks)), dim3(C::threads), 0, s, l.M, l.V, l.ns,
                     l.count, l.L, nch, starts, ss, l.X);
}

// kFull: rows of NP doubles on 16-byte boundaries.
bool full(const ScanLevel& l, int NP) { return l.ns == NP && (reinterpret_cast<uintptr_t>(l.M) & 15) == 0; }

template <class F>
void by_dim(int NP, F&& f)
{
    switch (NP) {
    case 8: return f(std::integral_constant<int, 8>());
    case 16: return f(std::integral_constant<int, 16>());
    case 24: return f(std::integral_constant<int, 24>());
    case 32: return f(std::integral_constant<int, 32>());
    case 40: return f(std::integral_constant<int, 40>());
    case 48: return f(std::integral_constant<int, 48>());
    case 56: return f(std::integral_constant<int, 56>());
    case 64: return f(std::integral_constant<int, 64>());
    default: throw Error(kInvalidArgument, "general scan: scan dimension above 64");
    }
}

}  // namespace

int general_padded_dim(int ns)
{
    int NP = 8;
    while (NP < ns) NP <<= 1;
    return NP;
}

void launch_scan_up(const ScanLevel& l, int NP, long nch, double* Mo, double* Vo, cudaStream_t s)
{
    if (nch <= 0) return;
    if (nch > 0x7fffffffL) throw Error(kInvalidArgument, "general scan: too many maps");
    by_dim(NP, [&](auto np) {
        if (full(l, NP)) up_t<decltype(np)::value, true>(l, nch, Mo, Vo, s);
        else up_t<decltype(np)::value, false>(l, nch, Mo, Vo, s);
    });
}

void launch_scan_down(const ScanLevel& l, int NP, const double* starts, int ss, cudaStream_t s)
{
    by_dim(NP, [&](auto np) {
        if (full(l, NP)) down_t<decltype(np)::value, true>(l, starts, ss, s);
        else down_t<decltype(np)::value, false>(l, starts, ss, s);
    });
}

void launch_distribute(double* Ms, const double* Phi, int NP, long count, int sms, cudaStream_t s)
{
    k_distribute<<<grid_for(count * (long)NP * NP, 256, 8 * sms), 256, 0, s>>>(Ms, Phi, NP, count);
    PARODE_CUDA(cudaGetLastError());
}

}  // namespace parode
