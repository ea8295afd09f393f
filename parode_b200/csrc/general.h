// general.h -- the general affine scan over per-step maps (kernels_general.cu,
// general.cpp).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace parode {

// Padded scan dimension of a plan's general path (8, 16, 32 or 64) and the
// device bytes by which that path judges whether a solve is too large.
int general_padded_dim(int ns);
size_t general_scan_bytes(int ns, long count);

// Ms[k] = Phi (NP x NP) for k < count.
void launch_distribute(double* Ms, const double* Phi, int NP, long count, int sms, cudaStream_t s);

// One level of the chunked scan: count maps M[k] (ns x ns) with V[k] (ns, or
// null), in chunks of L, and the states X[k] (ns) entering them.
struct ScanLevel {
    const double* M = nullptr;
    const double* V = nullptr;
    double* X = nullptr;
    int ns = 0;
    long count = 0;
    int L = 16;
};
// The compositions of the first nch chunks: Mo (NP x NP each) and Vo (NP), NP = ns rounded up to 8.
void launch_scan_up(const ScanLevel& l, int NP, long nch, double* Mo, double* Vo, cudaStream_t s);
// X of every chunk from the states entering the chunks (pitch ss; null: zero).
void launch_scan_down(const ScanLevel& l, int NP, const double* starts, int ss, cudaStream_t s);

// The whole scan on device data: x_0 = x0 (nullptr: 0), x_{k+1} = M_k x_k +
// V_k (V nullptr: 0), X[k] = x_k for k < count; M count x ns x ns, V and X
// count x ns (X over any part of the inputs), row-major FP64.  FP64 in either precision form.
// Scratch from the stream-ordered pool; returns after enqueueing, with the
// number of kernels launched.
int general_scan(const double* M, const double* V, const double* x0, int ns, long count, int precision,
                  double* X, cudaStream_t s);

}  // namespace parode
