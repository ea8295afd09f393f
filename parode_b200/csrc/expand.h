// expand.h -- the radix expansion of a solve whose augmented state is autonomous
// (kernels_expand.cu).
#pragma once

#include <cuda_runtime.h>

#include "kernels.h"

namespace parode {

// Levels of the expansion: level l turns the states entering blocks
// [0, 16^l) into those entering [16^l, min(16^(l+1), blocks)).
constexpr int kExpandRadix = 16;
constexpr int kExpandMaxLevels = 8;

struct ExpandShape {
    int NP = 0;      // scan dimension, a multiple of 8 (<= 64)
    int H = 0;       // phase columns: 2 per (channel, term), 0 without inputs
    int Kc = 0;      // columns of an augmented state: NP + H padded to a supported width
    int R = 0, B = 0, p = 0;
    long nblocks = 0;
    int levels = 0;
    int imax[kExpandMaxLevels] = {};  // multiples of 16^l blocks level l needs
    int pow_levels = 0;               // transition powers E(2^0) .. E(2^(pow_levels - 1))

    __host__ __device__ int rows() const { return B * p; }
    long table_rows() const;  // NP rows per multiple and level
};

// Fills the shape; false when the widths are outside what the kernels take
// (Kc <= 160, one state row slice of the output table in shared memory).
bool expand_shape(int Ns, int mu, int terms, int p, long nScan, int R, ExpandShape* out);

// Everything the table kernels read.  Parameters q = channel * terms + term:
// amp, w = 2 pi f, phi.
struct ExpandTables {
    ExpandShape sh;
    int solver = 0, n = 0, mu = 0, terms = 0;
    int zeroB = 1, zeroD = 1;
    double dt = 0.0;                  // sample spacing (RK4 h / 2, ABM h)
    const double* Phi = nullptr;      // NP x NP
    const double* Bbar = nullptr;     // n x W m
    const double* Cext = nullptr;     // p x NP
    const double* D = nullptr;        // p x m
    const double* par = nullptr;      // amp | w | phi, mu terms each
    double* E = nullptr;              // pow_levels x NP x Kc
    double* T = nullptr;              // table_rows() x Kc
    double* W = nullptr;              // rows() x Kc
};

// The tables (set-up): transition powers by squaring, then the output rows
// and the levels' multiples from them.
void launch_expand_tables(const ExpandTables& t, cudaStream_t s);

// One solve up to the block states: phases of every block and X_0 into Z
// (nblocks x Kc), then the levels.  Sample j of the grid is at base + dt * j;
// block b starts at sample b * stride.  Returns the launches.
int launch_expand_states(const ExpandTables& t, const double* X0, double* Z, double base, long stride, cudaStream_t s);

// Outputs of blocks [c0, c1): Y[b rows + r] = W[r] . Z[b], below `limit`.
void launch_expand_out(const ExpandTables& t, const double* Z, double* Y, long c0, long c1, long limit, int sms,
                       cudaStream_t s);

// ---- batches: any scan dimension, many systems per launch ----------------------
// The same expansion in doublings (radix 2: no table beyond the powers E(2^l),
// which a batch of once-solved systems could not pay for), its products on the
// grouped GEMM launches.  One job per system.
struct ExpandJob {
    int solver = 0, n = 0, mu = 0, terms = 0, p = 0;
    int NP = 0, H = 0, Kc = 0, R = 0;   // Kc = NP + H rounded up to 8
    int pow_levels = 0, zeroB = 1, zeroD = 1;
    long nblocks = 0, stride = 0;       // stride: samples per block
    double base = 0.0, dt = 0.0;        // sample grid
    const double *amp = nullptr, *freq = nullptr, *phi = nullptr;  // the input's, channel-major
    const double *Bbar = nullptr, *Cext = nullptr, *D = nullptr, *X0 = nullptr;
    double* E = nullptr;                // pow_levels x NP x Kc; E(1)'s state columns hold Phi
    double* W = nullptr;                // B p x Kc
    double* Z = nullptr;                // nblocks x Kc
    double* rot = nullptr;              // pow_levels x H: sin, cos of w dt 2^l steps
};

// Channels times terms a batch job may have.
constexpr int kExpandMaxPairs = 512;

// Block length 2^R of a system solved `executions` times, by its FP64 flops
// per step: states 2 NP Kc / B, W's build 2 B p NP Kc spread over the solves
// (outputs 2 p Kc and the powers cost the same for every B).
int expand_log2_block(int NP, int Kc, int p, long nScan, double executions);

// Set-up of all jobs, around the GEMMs of expand_power_args: init (S_1, W's
// first rows, rot); per l the rotation parts of E(2^(l+1)) and of W's rows
// [2^l p, 2^(l+1) p), then the GEMMs onto them; last D's phases into W.
void launch_expand_init(const ExpandJob* dJobs, int njobs, int max_hq, long max_elems, cudaStream_t s);
void launch_expand_rot(const ExpandJob* dJobs, int njobs, int l, long max_elems, cudaStream_t s);
void launch_expand_feed(const ExpandJob* dJobs, int njobs, long max_elems, cudaStream_t s);
// N-contiguous tiled GEMMs of squaring step l (E, then W's doubling): count 0..2.
int expand_power_args(const ExpandJob& j, int l, LevelArgs out[2]);

// Execute: phases of every block and X_0; then per level d = 2^l the GEMM of
// expand_level_args (K-contiguous), and the outputs (expand_out_args).
void launch_expand_phases(const ExpandJob* dJobs, int njobs, long max_elems, cudaStream_t s);
LevelArgs expand_level_args(const ExpandJob& j, int l);
LevelArgs expand_out_args(const ExpandJob& j, double* Y, long limit);

// dst = P src (+ acc, which may be dst) for a few columns (K-contiguous, rows
// and K multiples of 8), where the square tiles would mostly multiply padding.
// A tile is 32 columns and 8 rows, K split over the CTA's warps (split), or 32
// rows, a warp each 8 (launches of many tiles).
long expand_narrow_tiles(const LevelArgs& a, bool split);
void launch_expand_narrow(const LevelArgs* dArgs, const long* dStart, int nent, long tiles, bool split, cudaStream_t s);

}  // namespace parode
