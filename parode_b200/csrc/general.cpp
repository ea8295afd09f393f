// general.cpp -- host driver of the general affine scan (general.h).
//
// The reference's scan driver (Sources/GPUFixedStepIterative.cpp:236-398)
// with its matrix products kept, over chunks instead of levels of pairs
// (kernels_general.cu).
#include "general.h"

#include "common.h"
#include "kernels.h"

#include <algorithm>
#include <functional>
#include <vector>

namespace parode {

namespace {

// Maps per chunk of a level: 16, up to 64 while that still leaves 24 chunks per
// SM (a chunk's maps are composed one after another, so short chunks cost
// upper-level work and long ones parallelism).
int chunk_length(long count)
{
    int L = 16;
    while (L < 64 && count / (2 * L) >= kSmCount * 24) L *= 2;
    return L;
}

// The device's stream-ordered pool keeps a scan's scratch mapped for the next
// one (as a plan's buffers): mapped anew, 10 MB cost 0.5 ms a call.
void keep_scratch(size_t bytes)
{
    int dev = 0;
    cudaMemPool_t pool = nullptr;
    PARODE_CUDA(cudaGetDevice(&dev));
    PARODE_CUDA(cudaDeviceGetDefaultMemPool(&pool, dev));
    uint64_t keep = 0, want = 2 * (uint64_t)bytes + ((uint64_t)64 << 20);
    PARODE_CUDA(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    if (keep < want) PARODE_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &want));
}

}  // namespace

size_t general_scan_bytes(int ns, long count)
{
    const long Tp = next_pow2(std::max<long>(count, 1));
    const long NP = general_padded_dim(ns);
    return sizeof(double) * (size_t)(Tp * NP * NP + (Tp + 1) * NP);
}

int general_scan(const double* M, const double* V, const double* x0, int ns, long count, int precision,
                  double* X, cudaStream_t s)
{
    if (!M || !X) throw Error(kInvalidArgument, "general scan: M and X must be device pointers");
    if (ns < 1 || ns > 64) throw Error(kInvalidArgument, "general scan: scan dimension must be in [1, 64]");
    if (count < 1) throw Error(kInvalidArgument, "general scan: count must be >= 1");
    if (precision != kFP64 && precision != kMixed) throw Error(kInvalidArgument, "unknown precision");
    const int NP = (int)round_up(ns, 8);
    int launches = 0;
    // A chunk writes its states while others still read their maps: X over V
    // itself is safe (a step's v is loaded before its state is stored, and by
    // its own chunk only), X over any other part of the inputs goes by way of
    // the scratch.  x0 is read before the first state is written.
    const size_t states = (size_t)count * ns;
    const auto over = [&](const double* p, size_t n) { return p && std::less<>()(p, X + states) && std::less<>()(X, p + n); };
    const bool by_scratch = over(M, states * ns) || (X != V && over(V, states));
    // level 0: the caller's maps; level l + 1: the compositions of level l's
    // chunks (all but the last, whose composition no state needs)
    std::vector<ScanLevel> lev(1);
    lev[0] = ScanLevel{M, V, X, ns, count, chunk_length(count)};
    size_t doubles = 0;
    std::vector<size_t> at;
    while (lev.back().count > lev.back().L) {
        const ScanLevel& b = lev.back();
        ScanLevel u;
        u.ns = NP;
        u.count = (b.count + b.L - 1) / b.L;
        u.L = chunk_length(u.count);
        at.push_back(doubles);
        doubles += (size_t)u.count * NP * (NP + 2);
        lev.push_back(u);
    }
    const size_t x_at = doubles;
    if (by_scratch) doubles += states;
    double* buf = nullptr;
    if (fault_alloc_now()) throw Error(kNotEnoughResources, "general scan: device allocation failed (injected)");
    if (doubles) {
        keep_scratch(sizeof(double) * doubles);
        cudaError_t e = cudaMallocAsync(reinterpret_cast<void**>(&buf), sizeof(double) * doubles, s);
        if (e != cudaSuccess) {
            cudaGetLastError();
            throw Error(kNotEnoughResources, "general scan: device allocation failed");
        }
    }
    if (by_scratch) lev[0].X = buf + x_at;
    try {
        for (size_t l = 1; l < lev.size(); ++l) {
            ScanLevel& u = lev[l];
            double* m = buf + at[l - 1];
            u.M = m;
            u.V = m + (size_t)u.count * NP * NP;
            u.X = m + (size_t)u.count * NP * (NP + 1);
            launch_scan_up(lev[l - 1], NP, u.count - 1, m, m + (size_t)u.count * NP * NP, s);
            ++launches;  // a level above another has at least two maps
        }
        for (size_t l = lev.size(); l-- > 0;) {
            const bool top = l + 1 == lev.size();
            launch_scan_down(lev[l], NP, top ? x0 : lev[l + 1].X, top ? ns : NP, s);
            ++launches;
        }
        if (by_scratch) PARODE_CUDA(cudaMemcpyAsync(X, lev[0].X, sizeof(double) * states, cudaMemcpyDeviceToDevice, s));
    } catch (...) {
        if (buf) cudaFreeAsync(buf, s);
        throw;
    }
    if (buf) PARODE_CUDA(cudaFreeAsync(buf, s));
    return launches;
}

}  // namespace parode
