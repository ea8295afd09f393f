// tuner.h -- measured choice of the block length of a solve's leaf.
//
// The block length B = 2^R trades the work within blocks (the response leaf's
// window GEMMs, the FP64 build of W's tables; growing with B) against the work
// over them (the carry, the expansion's states; shrinking with B).  The engines
// pick R by rules and cost models; ParODE_TuneResponseBlock times the
// candidates on the device for a class of systems instead and stores the
// fastest here, and every plan or batch made afterwards for a system of that
// class uses it.  The leaves are different kernels with different optima, so a
// class names the leaf that was timed.  The table can be saved and loaded per
// GPU (one entry per line).
#pragma once

#include <string>

namespace parode {

// The leaf whose block length an entry is: sample windows (kernels_br.cu), the
// expansion of sinusoid phases in a single plan, and that in doublings (the
// batch engine; kernels_expand.cu).
enum TuneLeaf { kTuneWindows = 0, kTunePhases = 1, kTuneDoublings = 2 };

// A class of systems: solver, padded scan dimension (power of two), input
// and output counts (powers of two), horizon (log2 of the scan steps,
// rounded up), precision form and leaf.
struct TuneClass {
    int solver = 0, np = 0, m = 0, p = 0, tclass = 0, precision = 0, leaf = kTuneWindows;
};

TuneClass tune_class(int solver, int Ns, int m, int p, long nScan, int precision, int leaf);
// The measured log2 block length of the class, or -1 when it was not tuned.
int tuned_log2_block(const TuneClass& c);
void tune_store(const TuneClass& c, int log2B, float ms);
void tune_clear();
// Text form: one line per entry, "gpu solver np m p tclass precision log2B ms
// leaf" (without a leaf: sample windows); load keeps the entries of `gpu` and
// returns how many it read.
std::string tune_dump(const std::string& gpu);
int tune_load_text(const std::string& text, const std::string& gpu);

}  // namespace parode
