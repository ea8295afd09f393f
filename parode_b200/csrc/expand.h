// expand.h -- the radix expansion of a solve whose augmented state is autonomous
// (kernels_expand.cu).
#pragma once

#include <cuda_runtime.h>

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

}  // namespace parode
