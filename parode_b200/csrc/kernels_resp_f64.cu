// kernels_resp_f64.cu -- the FP64 outputs of the block-response leaf
// (kernels_br.cu) for one system: y_b = W_out [window_b ; X_b].
//
// A CTA keeps a slice of 64 rows of W in shared memory for its whole run; a
// warp alone takes tiles of 16 blocks: their windows and states as DMMA A
// fragments straight from global memory (32 columns at a time, the next 32 in
// flight), the slice's eight row tiles as accumulators, results stored two
// rows a lane (a block's 8 rows are 64 consecutive bytes).  No barrier after
// the staging, W's fragments two chunks ahead of their products (0.145 ms
// without that).  Row (j, o) of W_out is zero past the samples that step j
// reads, so a row tile skips the columns past its last row's limit (on average
// half the window).  FP64-tensor bound: the outputs of RK4 n = 64, m = p = 8,
// 2^20 steps are 3.6 GFLOP (97 us) in 0.132 ms, the pipe 79 % busy; 0.203 ms as 64 x 64 tiles over
// the whole of W (5.5 GFLOP), 0.155 as tiles that skip.  The aggregates have no
// zeros and stay with the tiles (82 us against 94).
#include "common.h"
#include "device_common.cuh"
#include "kernels.h"

#include <algorithm>
#include <type_traits>

namespace parode {

namespace {

constexpr int kThreads = 384, kWarps = kThreads / 32;
constexpr int kSliceRows = 64, kRT = kSliceRows / 8, kMaxSlices = 64;
constexpr int kSeg = 32;  // columns per segment
constexpr size_t kSmemMax = 220 * 1024;

struct Args {
    const double* W = nullptr;
    long ldw = 0;
    int M = 0, K1 = 0, K2 = 0;
    const double* U = nullptr;
    long ugs = 0;
    const double* X = nullptr;
    long xgs = 0;
    double* Y = nullptr;
    long gs = 0, limit = 0, nblocks = 0;
    int tri_p = 0, tri_base = 0, tri_step = 0;
    int vec = 0, slices = 0;
    short cta0[kMaxSlices + 1] = {};  // first CTA of each slice
};

// Window columns that rows up to r read, rounded up to 8.
__host__ __device__ inline int window_limit(const Args& a, int r)
{
    const int last = r < a.M ? r : a.M - 1;
    int k = a.K1;
    if (a.tri_p > 0 && a.tri_base + (last / a.tri_p) * a.tri_step < k) k = a.tri_base + (last / a.tri_p) * a.tri_step;
    return (k + 7) & ~7;
}

__host__ __device__ inline int pitch(int cols) { return cols + ((cols & 8) ? 0 : 8); }  // 8 mod 16: conflict-free 16-byte fragments

// Two doubles, or zeros.  Volatile, as the products are: the load stays where
// it is written, a segment ahead of its use.
__device__ __forceinline__ double2 load_pair(const double* p, bool in)
{
    double2 v;
    asm volatile(
        "{\n.reg .pred q;\nsetp.ne.b32 q, %3, 0;\nmov.f64 %0, 0d0000000000000000;\nmov.f64 %1, 0d0000000000000000;\n"
        "@q ld.global.v2.f64 {%0, %1}, [%2];\n}\n"
        : "=&d"(v.x), "=&d"(v.y)
        : "l"(p), "r"((int)in)
        : "memory");
    return v;
}

__device__ __forceinline__ double2 load_shared(unsigned at)
{
    double2 v;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];\n" : "=d"(v.x), "=d"(v.y) : "r"(at) : "memory");
    return v;
}

__global__ void __launch_bounds__(kThreads, 1) k_resp_f64(const __grid_constant__ Args a)
{
    extern __shared__ __align__(16) double Ws[];
    int slice = 0;
    while (slice + 1 < a.slices && (int)blockIdx.x >= a.cta0[slice + 1]) ++slice;
    const int idx = blockIdx.x - a.cta0[slice], nidx = a.cta0[slice + 1] - a.cta0[slice];
    const int m0 = slice * kSliceRows, rows = min(kSliceRows, a.M - m0), nrt = (rows + 7) / 8;
    const int Kw = window_limit(a, m0 + rows - 1), cols = Kw + a.K2, ld = pitch(cols);
    for (int e = threadIdx.x; e < nrt * 8 * (cols / 2); e += kThreads) {
        const int r = e / (cols / 2), c = 2 * (e - r * (cols / 2));
        // window columns up to K1 (even), then the state's
        const bool in = r < rows && (c < a.K1 || c >= Kw);
        const double* src = a.W + (long)(m0 + (in ? r : 0)) * a.ldw + (c < Kw ? (in ? c : 0) : a.K1 + c - Kw);
        const unsigned d = (unsigned)__cvta_generic_to_shared(Ws + r * ld + c);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(in ? 16 : 0) : "memory");
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    grid_dep_wait();  // the samples, the carried states
    grid_dep_trigger();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    __shared__ int lim[kRT];  // window columns of each row tile
    if (threadIdx.x < kRT) lim[threadIdx.x] = (int)threadIdx.x < nrt ? window_limit(a, m0 + threadIdx.x * 8 + 7) : 0;
    __syncthreads();
    const int segs_w = (Kw + kSeg - 1) / kSeg, segs = segs_w + (a.K2 + kSeg - 1) / kSeg;
    // the CTA's tiles of 8 blocks dealt evenly to the warps, taken two at a time
    const long tiles = (a.nblocks + 7) / 8, t0 = tiles * idx / nidx, n = tiles * (idx + 1) / nidx - t0;
    const long w0 = t0 + n * warp / kWarps, w1 = t0 + n * (warp + 1) / kWarps;
    // CT tiles at a time, from `tile` while CT are left below `end`
    auto blocks = [&](long tile, long end, auto ct) {
        constexpr int CT = decltype(ct)::value;
        if (tile + CT > end) return;
        auto load = [&](long at, int s, double2 (&z)[CT][kSeg / 8]) {
            const bool win = s < segs_w;
            const int k0 = (win ? s : s - segs_w) * kSeg + 2 * t, left = (win ? a.K1 : a.K2) - k0;
            const double* base = (win ? a.U : a.X) + k0;
            const long stride = win ? a.ugs : a.xgs;
#pragma unroll
            for (int c = 0; c < CT; ++c) {
                const long b = min((at + c) * 8 + g, a.nblocks - 1);  // past the last block: not stored
#pragma unroll
                for (int q = 0; q < kSeg / 8; ++q) z[c][q] = load_pair(base + b * stride + 8 * q, 8 * q < left);
            }
        };
        double2 z0[CT][kSeg / 8], z1[CT][kSeg / 8];
        load(tile, 0, z0);
        for (; tile + CT <= end; tile += CT) {
        const long b0 = tile * 8;
        double acc[kRT][CT][2] = {};
        auto mma = [&](int rt, int q, double2 w, const double2 (&z)[CT][kSeg / 8]) {
#pragma unroll
            for (int c = 0; c < CT; ++c) dmma_m8n8k4(acc[rt][c][0], acc[rt][c][1], z[c][q].x, w.x);
#pragma unroll
            for (int c = 0; c < CT; ++c) dmma_m8n8k4(acc[rt][c][0], acc[rt][c][1], z[c][q].y, w.y);
        };
        auto products = [&](int s, const double2 (&z)[CT][kSeg / 8]) {
            const bool win = s < segs_w;
            const int k0 = (win ? s : s - segs_w) * kSeg, at = win ? k0 : Kw + k0;
            const int nq = min(kSeg, (win ? Kw : a.K2) - k0) / 8;
            const unsigned w0 = (unsigned)__cvta_generic_to_shared(Ws + g * ld + at + 2 * t), row = 64 * ld;
            int first = 0;  // row tiles before it read none of these columns
            if (win)
                while (first < nrt && k0 >= lim[first]) ++first;
            if (nq == 4) {
                // W's fragments two chunks ahead of their products
                double2 r0 = load_shared(w0 + first * row), r1 = load_shared(w0 + first * row + 64);
#pragma unroll
                for (int rt = 0; rt < kRT; ++rt) {
                    if (rt < first || rt >= nrt) continue;
                    const unsigned w = w0 + rt * row, nx = rt + 1 < nrt ? w + row : w;
                    const double2 r2 = load_shared(w + 128);
                    mma(rt, 0, r0, z);
                    const double2 r3 = load_shared(w + 192);
                    mma(rt, 1, r1, z);
                    r0 = load_shared(nx);
                    mma(rt, 2, r2, z);
                    r1 = load_shared(nx + 64);
                    mma(rt, 3, r3, z);
                }
            } else {
#pragma unroll
                for (int rt = 0; rt < kRT; ++rt) {
                    if (rt < first || rt >= nrt) continue;
#pragma unroll
                    for (int q = 0; q < 3; ++q)
                        if (q < nq) mma(rt, q, load_shared(w0 + rt * row + 64 * q), z);
                }
            }
        };
        for (int s = 0; s < segs; s += 2) {
            if (s + 1 < segs) load(tile, s + 1, z1);
            products(s, z0);
            // the segment after, or the next tile's first
            if (s + 2 < segs) load(tile, s + 2, z0);
            else if (tile + 2 * CT <= end) load(tile + CT, 0, z0);
            if (s + 1 < segs) products(s + 1, z1);
        }
#pragma unroll
        for (int rt = 0; rt < kRT; ++rt) {
            if (rt >= nrt) break;
            const int r = m0 + rt * 8 + 2 * t;
#pragma unroll
            for (int c = 0; c < CT; ++c) {
                const long b = b0 + 8 * c + g, o = b * a.gs + r;
                if (b >= a.nblocks || r >= a.M) continue;
                if (a.vec && o + 1 < a.limit) {
                    *reinterpret_cast<double2*>(a.Y + o) = make_double2(acc[rt][c][0], acc[rt][c][1]);
                } else {
                    if (o < a.limit) a.Y[o] = acc[rt][c][0];
                    if (r + 1 < a.M && o + 1 < a.limit) a.Y[o + 1] = acc[rt][c][1];
                }
            }
        }
        }
    };
    blocks(w0, w1, std::integral_constant<int, 2>());
    blocks(w0 + (w1 - w0) / 2 * 2, w1, std::integral_constant<int, 1>());
}

}  // namespace

bool launch_resp_f64(const LevelArgs& l, int sms, cudaStream_t s)
{
    if (l.ncols <= 0) return true;
    Args a;
    a.W = l.P;
    a.ldw = l.ldp;
    a.M = level_rows(l);
    a.K1 = l.K1 > 0 ? l.K1 : level_k(l);
    a.K2 = level_k(l) - a.K1;
    a.U = l.src;
    a.ugs = l.src_gs;
    a.X = l.src2;
    a.xgs = l.src2_gs;
    a.Y = l.dst;
    a.gs = l.dst_gs;
    a.limit = l.dst_limit >= 0 ? l.dst_limit : (long)1 << 62;
    a.nblocks = l.ncols;
    a.tri_p = l.K1 > 0 ? l.tri_p : 0;
    a.tri_base = l.tri_base;
    a.tri_step = l.tri_step;
    auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    // 16-byte fragments of W, the windows and the states
    if (l.dst_is != 1 || l.src_ks != 1 || (a.K1 & 1) || (a.K2 & 7) || (a.ldw & 1) || (a.ugs & 1) || !aligned(a.W) ||
        !aligned(a.U) || (a.K2 && ((a.xgs & 1) || !aligned(a.X))))
        return false;
    a.vec = aligned(a.Y) && (a.gs & 1) == 0;
    a.slices = (a.M + kSliceRows - 1) / kSliceRows;
    if (a.slices > kMaxSlices || a.slices > sms) return false;
    // CTAs per slice by its products; no more in all than tiles can use
    double cost[kMaxSlices], total = 0.0;
    size_t smem = 0;
    for (int i = 0; i < a.slices; ++i) {
        const int m0 = i * kSliceRows, rows = std::min(kSliceRows, a.M - m0);
        cost[i] = 0.0;
        for (int r = 0; r < rows; r += 8) cost[i] += window_limit(a, m0 + r + 7) + a.K2;
        total += cost[i];
        const int cols = window_limit(a, m0 + rows - 1) + a.K2;
        smem = std::max(smem, sizeof(double) * (size_t)((rows + 7) / 8 * 8) * pitch(cols));
    }
    if (smem > kSmemMax) return false;
    const long tiles = (a.nblocks + 7) / 8;
    const long most = std::max<long>(1, (tiles + kWarps / 4 - 1) / (kWarps / 4));  // a few warps at least per CTA
    int used = 0;
    for (int i = 0; i < a.slices; ++i) {
        a.cta0[i] = (short)used;
        const int left = a.slices - i - 1;
        long n = (long)(sms * cost[i] / total + 0.5);
        n = std::max<long>(1, std::min<long>({n, most, (long)(sms - used - left)}));
        used += (int)n;
    }
    a.cta0[a.slices] = (short)used;
    PARODE_CUDA(cudaFuncSetAttribute(k_resp_f64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax));
    launch_dependent(k_resp_f64, dim3((unsigned)used), dim3(kThreads), smem, s, a);
    return true;
}

}  // namespace parode
