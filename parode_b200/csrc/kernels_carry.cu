// kernels_carry.cu -- exclusive scan of block aggregates for scan dimensions <= 64.
//
// The blocked and block-response leaves leave one aggregate G_b per block of
// B steps; the state entering block b is the exclusive scan
//   X_0 = x0,  X_{b+1} = Q X_b + G_b,  Q = Phi^B,
// which is the reference's Blelloch composition (Kernels/MVVKernelScanUpsweep.cl,
// MVVKernelScanDownsweep.cl) applied to the blocks.  Here it runs as a chunked
// scan: chunks of 16 items, each chunk's aggregate (up), the chunk aggregates
// scanned one level higher with Q^16, and each chunk's items rewritten from its
// carried-in state (down).
//
// A chunk is four runs of four items.  Up: three steps with Q along the runs,
// whose aggregates S_0 .. S_2 are kept in the places of the runs' last items
// (the down pass reads no last item), then a tree with Q^4 and Q^8.  Down: a
// Kogge-Stone scan of [carry, S_0, S_1, S_2] with Q^4 and Q^8 gives the states
// entering the runs, then three steps with Q.  Five dependent steps a pass, two
// chunks filling the eight columns of an NP x 8 tile on the FP64 tensor cores
// (DMMA m8n8k4), one warp per eight rows with the three powers' fragments in
// registers.  A step's products take 512 cycles of an SM at NP = 64 (16 cycles
// per DMMA on each sub-partition), its barrier, shared-memory round trip and
// additions 200 more, and a launch boundary about 2 us: depth and launches bound
// a scan until its tiles fill the chip.  So the top two levels are one launch
// (k_chunk_mid), and level 0 at NP > 32, whose tiles do fill it, takes the form
// with the fewest products (k_chain_up, k_chain_down).  The form depends on the
// level's global index only (k_chunk_mid takes the steps of the launches it
// stands for), so a time-partitioned solve computes the same bits as the whole
// one on the sample windows (the samplers' runs follow the whole horizon too).
//
// The whole scan, against chunks stepped through one item of prefetch ahead with
// depth-4 trees above level 0 and a launch per level and direction: NP = 64,
// 65.5 K blocks 99 -> 73 us, 12.5 K blocks 44 -> 35; NP = 32, 18.8 K blocks
// 44 -> 18; NP = 8, 256 blocks 6.4 -> 4.  At NP = 64 and 65.5 K blocks the two
// level-0 passes take 51 us of it; with the run form they take 78, its powers'
// registers leaving one CTA an SM.
#include "common.h"
#include "device_common.cuh"
#include "kernels.h"

#include <algorithm>

namespace parode {

namespace {

constexpr int kChunk = 16;         // items per chunk: Q^16 = 4 power-table levels up
constexpr int kTile = 2 * kChunk;  // items per tile: two chunks, their eight runs being its columns
constexpr int kLd = 10;            // row pitch (doubles) of the 8-column state: conflict-free B fragments

template <int NP>
struct Tile {
    static constexpr int threads = 4 * NP;  // one warp per 8 rows
    // items one after the other, 4 doubles more after every 8 (conflict-free reads of a run step)
    static constexpr int size = kTile * NP + 16;
    __host__ __device__ static constexpr int at(int item) { return item * NP + (item >> 3) * 4; }
};

struct Lane {
    int g, t, row;
    __device__ Lane()
    {
        const int lane = threadIdx.x & 31;
        g = lane >> 2;
        t = lane & 3;
        row = (threadIdx.x >> 5) * 8 + g;  // this lane's row of the D fragment, columns 2 t and 2 t + 1
    }
};

// A fragments of this warp's rows of a power.  Product 2 c + u takes the K
// values 8 c + 2 t + u, so that a lane reads 16 bytes at a time.
template <int NP>
__device__ __forceinline__ void load_q(const double* __restrict__ Q, const Lane& w, double (&qa)[NP / 4])
{
#pragma unroll
    for (int c = 0; c < NP / 8; ++c) {
        const double2 v = *reinterpret_cast<const double2*>(Q + w.row * NP + 8 * c + 2 * w.t);
        qa[2 * c] = v.x;
        qa[2 * c + 1] = v.y;
    }
}

// Items [32 tile, ..) into buf, zeros past the last; one copy group.
template <int NP>
__device__ __forceinline__ void fetch(const double* items, long count, long tile, double* buf)
{
    const double* src = items + tile * kTile * NP;
    const long left = count - tile * kTile;
#pragma unroll
    for (int q = 0; q < kTile / 8; ++q) {
        const int e = threadIdx.x + q * Tile<NP>::threads, it = e / (NP / 2), c = 2 * (e % (NP / 2));
        const unsigned dst = (unsigned)__cvta_generic_to_shared(buf + Tile<NP>::at(it) + c);
        const bool ok = it < left;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(ok ? src + it * NP + c : items),
                     "r"(ok ? 16 : 0)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void landed() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// acc += Q X[:, col] for this lane's output columns that `use` (bit e: column
// 2 t + e) names; col: this lane's column of X, < 0 a zero one.  The K products
// go to kSplit independent partial sums.
template <int NP>
__device__ __forceinline__ void step(const double* X, const double (&qa)[NP / 4], int col, int use, double (&acc)[2],
                                     const Lane& w)
{
    constexpr int kSplit = NP / 4 < 4 ? NP / 4 : 4;
    double part[kSplit][2] = {};
    const double* x = X + 2 * w.t * kLd + (col < 0 ? 0 : col);
#pragma unroll
    for (int kk = 0; kk < NP / 4; ++kk) {
        const double b = x[(8 * (kk / 2) + kk % 2) * kLd];
        dmma_m8n8k4(part[kk % kSplit][0], part[kk % kSplit][1], qa[kk], col < 0 ? 0.0 : b);
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        double v = acc[e];
#pragma unroll
        for (int q = 0; q < kSplit; ++q) v += part[q][e];
        if (use >> e & 1) acc[e] = v;
    }
}

__device__ __forceinline__ void put(double* X, const double (&v)[2], const Lane& w)
{
    *reinterpret_cast<double2*>(X + w.row * kLd + 2 * w.t) = make_double2(v[0], v[1]);
}

// Item i of the runs of this lane's two columns.
template <int NP>
__device__ __forceinline__ void item(const double* buf, int i, double (&v)[2], const Lane& w)
{
    const double* b = buf + Tile<NP>::at(8 * w.t) + i * NP + w.row;
    v[0] = b[0];
    v[1] = b[4 * NP];
}

// The runs' aggregates, left in acc and X[1].
template <int NP>
__device__ __forceinline__ void runs(const double* buf, const double (&q1)[NP / 4], double (*X)[NP * kLd],
                                     double (&acc)[2], const Lane& w)
{
    item<NP>(buf, 0, acc, w);
    put(X[0], acc, w);
#pragma unroll
    for (int i = 1; i < 4; ++i) {
        __syncthreads();
        item<NP>(buf, i, acc, w);
        step<NP>(X[(i & 1) ^ 1], q1, w.g, 3, acc, w);
        put(X[i & 1], acc, w);
    }
}

// x: [carry, S_0, S_1, S_2] of each chunk -> the states entering its runs.
template <int NP>
__device__ __forceinline__ void enter(const double (&q4)[NP / 4], const double (&q8)[NP / 4], double (*X)[NP * kLd],
                                      double (&x)[2], const Lane& w)
{
    put(X[0], x, w);
    __syncthreads();
    step<NP>(X[0], q4, w.g & 3 ? w.g - 1 : -1, w.t & 1 ? 3 : 2, x, w);
    put(X[1], x, w);
    __syncthreads();
    step<NP>(X[1], q8, w.g & 2 ? w.g - 2 : -1, w.t & 1 ? 3 : 0, x, w);
}

// From the states x entering the runs: out(e, i, x[e]) for the state entering
// item i of run 2 t + e.
template <int NP, class F>
__device__ __forceinline__ void along(const double* buf, const double (&q1)[NP / 4], double (*X)[NP * kLd],
                                      double (&x)[2], const Lane& w, F&& out)
{
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        out(0, i, x[0]);
        out(1, i, x[1]);
        if (i == 3) break;
        put(X[i & 1], x, w);
        __syncthreads();
        item<NP>(buf, i, x, w);
        step<NP>(X[i & 1], q1, w.g, 3, x, w);
    }
}

// The chunks' aggregates from the runs' (X[1]; every thread past a barrier):
// columns 0 and 1, in acc of the lanes t == 0.
template <int NP>
__device__ __forceinline__ void tree(const double (&q4)[NP / 4], const double (&q8)[NP / 4], double (*X)[NP * kLd],
                                     double (&acc)[2], const Lane& w)
{
    // output column p of the first step from runs 2 p, 2 p + 1 (X[1]); of the second from halves 2 p, 2 p + 1 (X[0])
#pragma unroll
    for (int e = 0; e < 2; ++e) acc[e] = w.t < 2 ? X[1][w.row * kLd + 2 * (2 * w.t + e) + 1] : 0.0;
    step<NP>(X[1], q4, w.g < 4 ? 2 * w.g : -1, 3, acc, w);
    if (w.t < 2) put(X[0], acc, w);
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 2; ++e) acc[e] = w.t < 1 ? X[0][w.row * kLd + 2 * e + 1] : 0.0;
    step<NP>(X[0], q8, w.g < 2 ? 2 * w.g : -1, 3, acc, w);
}

// Chunk aggregates, next[c] = sum_{j < 16} Q^(15 - j) items[16 c + j] (items past
// count are zero), and the run aggregates into items.  Q points at the power's
// table level: Q^4 and Q^8 are two and three levels up.
template <int NP>
__global__ void __launch_bounds__(4 * NP) k_chunk_up(double* items, long count, const double* __restrict__ Q,
                                                     double* __restrict__ next)
{
    __shared__ __align__(16) double buf[2][Tile<NP>::size];
    __shared__ __align__(16) double X[2][NP * kLd];
    const Lane w;
    double q1[NP / 4], q4[NP / 4], q8[NP / 4];
    load_q<NP>(Q, w, q1);
    load_q<NP>(Q + 2 * NP * NP, w, q4);
    load_q<NP>(Q + 3 * NP * NP, w, q8);
    grid_dep_wait();     // the items are the previous kernel's
    grid_dep_trigger();  // the next level's CTAs may start loading their powers
    const long tiles = (count + kTile - 1) / kTile, nchunks = (count + kChunk - 1) / kChunk;
    fetch<NP>(items, count, blockIdx.x, buf[0]);
    int cur = 0;
    for (long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        landed();
        __syncthreads();
        if (tile + gridDim.x < tiles) fetch<NP>(items, count, tile + gridDim.x, buf[cur ^ 1]);
        double acc[2];
        runs<NP>(buf[cur], q1, X, acc, w);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int c = 2 * w.t + e;  // chunk c / 4, run c % 4
            const long at = tile * kTile + 4 * c + 3;
            if ((c & 3) < 3 && at < count) items[at * NP + w.row] = acc[e];
        }
        __syncthreads();
        tree<NP>(q4, q8, X, acc, w);
        if (w.t < 1)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                if (2 * tile + e < nchunks) next[(2 * tile + e) * NP + w.row] = acc[e];
        cur ^= 1;
    }
}

// Chunk rewrite: from each chunk's carried-in state x = carries[c], items
// [16 c, 16 c + 16) become the states entering them (x, then Q x + item, ...).
// kTop: the one chunk of a top level, whose run aggregates are formed here.
template <int NP, bool kTop>
__global__ void __launch_bounds__(4 * NP) k_chunk_down(double* items, long count, const double* __restrict__ Q,
                                                       const double* __restrict__ carries)
{
    __shared__ __align__(16) double buf[2][Tile<NP>::size];
    __shared__ __align__(16) double X[2][NP * kLd];
    const Lane w;
    double q1[NP / 4], q4[NP / 4], q8[NP / 4];
    load_q<NP>(Q, w, q1);
    load_q<NP>(Q + 2 * NP * NP, w, q4);
    load_q<NP>(Q + 3 * NP * NP, w, q8);
    grid_dep_wait();     // the carries and items are the previous kernels'
    grid_dep_trigger();  // the next level's CTAs may start loading their powers
    const long tiles = (count + kTile - 1) / kTile, nchunks = (count + kChunk - 1) / kChunk;
    fetch<NP>(items, count, blockIdx.x, buf[0]);
    int cur = 0;
    for (long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        // column c of [carry, S_0, S_1, S_2] per chunk
        double x[2], s[2];
        const long ch = 2 * tile + (w.t >> 1);
        const double carry = !(w.t & 1) && ch < nchunks ? carries[ch * NP + w.row] : 0.0;
        landed();
        __syncthreads();
        if (tile + gridDim.x < tiles) fetch<NP>(items, count, tile + gridDim.x, buf[cur ^ 1]);
        if (kTop) {
            runs<NP>(buf[cur], q1, X, x, w);
            __syncthreads();
#pragma unroll
            for (int e = 0; e < 2; ++e) s[e] = w.t + e > 0 ? X[1][w.row * kLd + 2 * w.t + e - 1] : 0.0;
        } else {
#pragma unroll
            for (int e = 0; e < 2; ++e)
                s[e] = w.t + e > 0 ? buf[cur][Tile<NP>::at(4 * (2 * w.t + e) - 1) + w.row] : 0.0;
        }
        x[0] = w.t & 1 ? s[0] : carry;
        x[1] = s[1];
        enter<NP>(q4, q8, X, x, w);
        const long i0 = tile * kTile + 8 * w.t;  // first items of this lane's two runs: i0, i0 + 4
        along<NP>(buf[cur], q1, X, x, w, [&](int e, int i, double v) {
            if (i0 + 4 * e + i < count) items[(i0 + 4 * e + i) * NP + w.row] = v;
        });
        cur ^= 1;
    }
}

// A level of 17 .. 256 items, the one above it and the way back in one launch of
// one cluster, a CTA per tile: up to the chunk aggregates, which every CTA gets
// through distributed shared memory; the top level (<= 16 items, entered with
// X0) in every CTA; down with the two carries that are the CTA's own.  The same
// steps as the three launches it stands for, without their two launch
// boundaries (about 2 us each).
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

template <int NP>
__global__ void __launch_bounds__(4 * NP) k_chunk_mid(double* items, long count, const double* __restrict__ Q,
                                                      const double* __restrict__ X0)
{
    __shared__ __align__(16) double buf[Tile<NP>::size], top[Tile<NP>::size];
    __shared__ __align__(16) double X[2][NP * kLd];
    __shared__ double mine[2][NP];
    const Lane w;
    const int rank = blockIdx.x, ctas = gridDim.x;
    const double* Qt = Q + 4 * NP * NP;
    double q1[NP / 4], q4[NP / 4], q8[NP / 4];
    load_q<NP>(Q, w, q1);
    load_q<NP>(Q + 2 * NP * NP, w, q4);
    load_q<NP>(Q + 3 * NP * NP, w, q8);
    for (int e = threadIdx.x; e < Tile<NP>::size; e += Tile<NP>::threads) top[e] = 0.0;
    cluster_arrive();    // zeroed before any CTA's aggregates arrive
    grid_dep_wait();     // the items are the previous kernel's
    grid_dep_trigger();  // the next level's CTAs may start loading their powers
    fetch<NP>(items, count, rank, buf);
    landed();
    __syncthreads();
    double acc[2], s[2], x[2];
    runs<NP>(buf, q1, X, acc, w);
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 2; ++e) s[e] = w.t + e > 0 ? X[1][w.row * kLd + 2 * w.t + e - 1] : 0.0;
    tree<NP>(q4, q8, X, acc, w);
    load_q<NP>(Qt, w, q1);
    load_q<NP>(Qt + 2 * NP * NP, w, q4);
    load_q<NP>(Qt + 3 * NP * NP, w, q8);
    const double x0 = X0[w.row];
    cluster_wait();
    if (w.t == 0)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const unsigned at = (unsigned)__cvta_generic_to_shared(top + Tile<NP>::at(2 * rank + e) + w.row);
            for (int c = 0; c < ctas; ++c) {
                unsigned r;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(at), "r"(c));
                asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(r), "d"(acc[e]) : "memory");
            }
        }
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    runs<NP>(top, q1, X, acc, w);
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 2; ++e) x[e] = w.t + e > 0 ? X[1][w.row * kLd + 2 * w.t + e - 1] : 0.0;
    if (w.t == 0) x[0] = x0;
    if (w.t == 2) x[0] = 0.0;
    enter<NP>(q4, q8, X, x, w);
    along<NP>(top, q1, X, x, w, [&](int e, int i, double v) {
        const int c = 4 * (2 * w.t + e) + i - 2 * rank;
        if (c == 0 || c == 1) mine[c][w.row] = v;
    });
    load_q<NP>(Q, w, q1);
    load_q<NP>(Q + 2 * NP * NP, w, q4);
    load_q<NP>(Q + 3 * NP * NP, w, q8);
    __syncthreads();
    x[0] = w.t & 1 ? s[0] : mine[w.t >> 1][w.row];
    x[1] = s[1];
    enter<NP>(q4, q8, X, x, w);
    const long i0 = rank * kTile + 8 * w.t;
    along<NP>(buf, q1, X, x, w, [&](int e, int i, double v) {
        if (i0 + 4 * e + i < count) items[(i0 + 4 * e + i) * NP + w.row] = v;
    });
}

// ---- level 0 at NP > 32 --------------------------------------------------------
// Eight chunks a CTA, stepped through all 16 items: 15 products per eight chunks
// against 20 of the form above (five per two), and one power's registers, so four
// CTAs fit an SM.  The items come through a ring of shared-memory slots filled
// kAhead steps early, as a step is about as long as a trip to L2.  They lie column
// by column, NP + 2 doubles apart (conflict-free reads of a lane's two columns),
// a copy being one 16-byte piece per thread.
constexpr int kCols = 8;
constexpr int kSlots = 8, kAhead = kSlots - 1;

template <int NP>
struct Chain : Lane {
    static constexpr int threads = 4 * NP, pitch = NP + 2, slot = kCols * pitch;
    long c0, count;     // first chunk of the tile; items in all
    const double* src;  // this thread's piece of item 0
    unsigned dst;       // its place in slot 0
    double* ring;

    __device__ Chain(const double* items, long n, long tile, double* r) : count(n), ring(r)
    {
        c0 = tile * kCols;
        const int col = threadIdx.x / (NP / 2), part = threadIdx.x % (NP / 2);
        first = (c0 + col) * kChunk;
        src = items + first * NP + 2 * part;
        dst = (unsigned)__cvta_generic_to_shared(r + col * pitch + 2 * part);
        zero = items;
    }
    // item j of every chunk into its slot (zeros past the last item); one group a call
    __device__ void fetch(int j) const
    {
        const bool ok = j < kChunk && first + j < count;
        if (j < kChunk)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + 8 * slot * (j % kSlots)),
                         "l"(ok ? src + (long)j * NP : zero), "r"(ok ? 16 : 0)
                         : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    __device__ void start() const
    {
#pragma unroll
        for (int j = 0; j < kAhead; ++j) fetch(j);
    }
    // at step j, before its fetch: this thread's pieces of items 0 .. j have landed
    __device__ void landed() const { asm volatile("cp.async.wait_group %0;" ::"n"(kAhead - 1) : "memory"); }
    __device__ void item(int j, double (&v)[2]) const
    {
        const double* q = ring + slot * (j % kSlots) + row;
        v[0] = q[(2 * t) * pitch];
        v[1] = q[(2 * t + 1) * pitch];
    }

private:
    long first;
    const double* zero;
};

// Chunk aggregates of one tile (kCols chunks from c0 = tile * kCols):
// next[c] = sum_{j<16} Q^(15-j) items[16 c + j] (items past count are zero;
// the last chunk's aggregate is never read by the scan).
template <int NP>
__global__ void __launch_bounds__(4 * NP) k_chain_up(const double* __restrict__ items, long count,
                                                     const double* __restrict__ Q, double* __restrict__ next)
{
    __shared__ __align__(16) double Xs[2][NP * kLd];
    __shared__ __align__(16) double ring[kSlots * Chain<NP>::slot];
    const Chain<NP> c(items, count, blockIdx.x, ring);
    double qa[NP / 4];
    load_q<NP>(Q, c, qa);
    grid_dep_wait();  // the items are the previous kernel's
    grid_dep_trigger();  // the next level's CTAs may start loading their powers
    c.start();
    int cur = 0;
    for (int j = 0; j < kChunk; ++j) {
        c.landed();
        __syncthreads();  // item j and the state; slot (j - 1) % kSlots is free
        c.fetch(j + kAhead);
        double acc[2];
        c.item(j, acc);
        if (j > 0) step<NP>(Xs[cur], qa, c.g, 3, acc, c);
        cur ^= 1;
        put(Xs[cur], acc, c);
    }
    __syncthreads();
    const long nchunks = (count + kChunk - 1) / kChunk;
    for (int e = threadIdx.x; e < NP * kCols; e += Chain<NP>::threads) {
        const int col = e / NP, row = e - col * NP;
        if (c.c0 + col < nchunks) next[(c.c0 + col) * NP + row] = Xs[cur][row * kLd + col];
    }
}

// Chunk rewrite of one tile: from the chunk's carried-in state
// x = carries[c], items [16 c, 16 c + 16) become the states entering them (x,
// then Q x + item, ...).  An item has landed in the ring, for every thread,
// before its place in memory is overwritten.
template <int NP>
__global__ void __launch_bounds__(4 * NP) k_chain_down(double* __restrict__ items, long count,
                                                       const double* __restrict__ Q,
                                                       const double* __restrict__ carries)
{
    __shared__ __align__(16) double Xs[2][NP * kLd];
    __shared__ __align__(16) double ring[kSlots * Chain<NP>::slot];
    const Chain<NP> c(items, count, blockIdx.x, ring);
    const long nchunks = (count + kChunk - 1) / kChunk;
    double qa[NP / 4];
    load_q<NP>(Q, c, qa);
    grid_dep_wait();  // the carries and items are the previous kernels'
    grid_dep_trigger();  // the next level's CTAs may start loading their powers
    c.start();
    // slot 0 <- the carried-in state
    double x[2];
    const long i0 = (c.c0 + 2 * c.t) * kChunk;  // items of this lane's two chunks: i0 + e kChunk + j
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const long ch = c.c0 + 2 * c.t + e;
        x[e] = ch < nchunks ? carries[ch * NP + c.row] : 0.0;
    }
    put(Xs[0], x, c);
    int cur = 0;
    for (int j = 0; j < kChunk; ++j) {
        c.landed();
        __syncthreads();  // item j and the state; slot (j - 1) % kSlots is free
        c.fetch(j + kAhead);
#pragma unroll
        for (int e = 0; e < 2; ++e)  // the state entering item j, over the item
            if (i0 + e * kChunk + j < count) items[(i0 + e * kChunk + j) * NP + c.row] = x[e];
        if (j + 1 == kChunk) break;
        c.item(j, x);
        step<NP>(Xs[cur], qa, c.g, 3, x, c);
        cur ^= 1;
        put(Xs[cur], x, c);
    }
}

// ---------------------------------------------------------------------------
// CTAs: a tile each, at most one wave (a CTA keeps its powers for all its tiles).
template <int NP>
unsigned chunk_grid(long count)
{
    constexpr int kPerSm = NP > 32 ? 1 : NP > 16 ? 4 : 8;
    return (unsigned)std::min<long>((count + kTile - 1) / kTile, kSmCount * kPerSm);
}

// Level 0 of a scan (h: the level's global index) steps through whole chunks.
template <int NP>
constexpr bool chained(int h)
{
    return NP > 32 && h == 0;
}

template <int NP>
unsigned chain_grid(long count)
{
    return (unsigned)(((count + kChunk - 1) / kChunk + kCols - 1) / kCols);
}

template <int NP>
int chunk_up_t(double* items, long count, const double* P, int l0, int h0, double* work, int levels, ChunkLevels* L,
               cudaStream_t s)
{
    const long mat = (long)NP * NP;
    L->arr[0] = items;
    L->cnt[0] = count;
    int h = 0;
    double* w = work;
    // levels < 0: up to a level k_chunk_mid or the top takes
    while (levels < 0 ? L->cnt[h] > (chained<NP>(h0 + h) ? kChunk : kChunk * kChunk) : h < levels) {
        if (h + 1 >= 16) throw Error(kInvalidArgument, "chunk carry: too many levels");
        const long cnt = L->cnt[h], nc = (cnt + kChunk - 1) / kChunk;
        const double* Q = P + (long)(l0 + 4 * h) * mat;
        if constexpr (chained<NP>(0)) {
            if (h0 + h == 0) launch_dependent(k_chain_up<NP>, chain_grid<NP>(cnt), Chain<NP>::threads, 0, s, (const double*)L->arr[h], cnt, Q, w);
            else launch_dependent(k_chunk_up<NP>, chunk_grid<NP>(cnt), Tile<NP>::threads, 0, s, L->arr[h], cnt, Q, w);
        } else {
            launch_dependent(k_chunk_up<NP>, chunk_grid<NP>(cnt), Tile<NP>::threads, 0, s, L->arr[h], cnt, Q, w);
        }
        L->arr[h + 1] = w;
        L->cnt[h + 1] = nc;
        w += nc * NP;
        ++h;
    }
    L->h = h;
    return h;
}

template <int NP>
int chunk_down_t(const ChunkLevels& L, const double* P, int l0, int h0, cudaStream_t s)
{
    const long mat = (long)NP * NP;
    for (int k = L.h - 1; k >= 0; --k) {
        const double *Q = P + (long)(l0 + 4 * k) * mat, *carries = L.arr[k + 1];
        if constexpr (chained<NP>(0)) {
            if (h0 + k == 0) {
                launch_dependent(k_chain_down<NP>, chain_grid<NP>(L.cnt[k]), Chain<NP>::threads, 0, s, L.arr[k],
                                 L.cnt[k], Q, carries);
                continue;
            }
        }
        launch_dependent(k_chunk_down<NP, false>, chunk_grid<NP>(L.cnt[k]), Tile<NP>::threads, 0, s, L.arr[k],
                         L.cnt[k], Q, carries);
    }
    return L.h;
}

template <int NP>
void chunk_mid_t(double* items, long count, const double* Q, const double* X0, cudaStream_t s)
{
    unsigned ctas = 1;
    while ((long)ctas * kTile < count) ctas *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = ctas;
    cfg.blockDim = Tile<NP>::threads;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = ctas;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    PARODE_CUDA(cudaLaunchKernelEx(&cfg, k_chunk_mid<NP>, items, count, Q, X0));
}

template <int NP>
int chunk_carry_t(double* items, long count, const double* P, int l0, int h0, const double* X0, double* work,
                  cudaStream_t s)
{
    ChunkLevels L;
    int launches = chunk_up_t<NP>(items, count, P, l0, h0, work, -1, &L, s);
    // the top, entered with X0: one chunk of at most 16 items, or two levels at once
    const double* Q = P + (long)(l0 + 4 * L.h) * NP * NP;
    if (L.cnt[L.h] <= kChunk)
        launch_dependent(k_chunk_down<NP, true>, 1, Tile<NP>::threads, 0, s, L.arr[L.h], L.cnt[L.h], Q, X0);
    else
        chunk_mid_t<NP>(L.arr[L.h], L.cnt[L.h], Q, X0, s);
    return launches + 1 + chunk_down_t<NP>(L, P, l0, h0, s);
}

}  // namespace

int chunk_carry_table_levels(long count) { return 4 * chunk_carry_levels(count) + 4; }

int chunk_carry_levels(long count)
{
    int h = 0;
    while (count > kChunk) {
        count = (count + kChunk - 1) / kChunk;
        ++h;
    }
    return h;
}

long chunk_carry_scratch(long count)
{
    long total = 0;
    while (count > kChunk) {
        count = (count + kChunk - 1) / kChunk;
        total += count;
    }
    return total;
}

#define PARODE_NP_SWITCH(NP, CALL)                                                             \
    switch (NP) {                                                                              \
    case 8: return CALL(8);                                                                    \
    case 16: return CALL(16);                                                                  \
    case 24: return CALL(24);                                                                  \
    case 32: return CALL(32);                                                                  \
    case 40: return CALL(40);                                                                  \
    case 48: return CALL(48);                                                                  \
    case 56: return CALL(56);                                                                  \
    case 64: return CALL(64);                                                                  \
    default: throw Error(kInvalidArgument, "chunk carry: NP must be a multiple of 8 up to 64"); \
    }

int launch_chunk_up(int NP, double* items, long count, const double* P, int l0, double* work, int levels,
                    ChunkLevels* L, cudaStream_t s)
{
#define PARODE_UP(K) chunk_up_t<K>(items, count, P, l0, 0, work, levels, L, s)
    PARODE_NP_SWITCH(NP, PARODE_UP)
#undef PARODE_UP
}

int launch_chunk_down(int NP, const ChunkLevels& L, const double* P, int l0, cudaStream_t s)
{
#define PARODE_DOWN(K) chunk_down_t<K>(L, P, l0, 0, s)
    PARODE_NP_SWITCH(NP, PARODE_DOWN)
#undef PARODE_DOWN
}

int launch_chunk_carry(int NP, double* items, long count, const double* P, int l0, int h0, const double* X0,
                       double* work, cudaStream_t s)
{
    if (count <= 0) return 0;
#define PARODE_CARRY(K) chunk_carry_t<K>(items, count, P, l0, h0, X0, work, s)
    PARODE_NP_SWITCH(NP, PARODE_CARRY)
#undef PARODE_CARRY
}

}  // namespace parode
