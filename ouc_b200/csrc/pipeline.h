// The issuing side of a two-stage copy/multiply pipeline (corrector.cu), apart
// from the instructions so that it also runs on the CPU.
#pragma once
#include <cuda_runtime.h>

namespace ouc {

// Items 0 .. count-1 in order, item k in stage k & 1.  ready(k) waits for the
// item's operands (false: the wait ran out), issue(k) issues its multiplications
// and commits them to the stage, done(stage, parity) waits for the commit that
// completes the stage's phase of that parity.  Returns false when a wait ran
// out, in every case only after the last commit of each stage has been waited
// for: what the multiplications still write may be released afterwards.
template <class Ready, class Issue, class Done>
__host__ __device__ __forceinline__ bool run_items(int count, Ready&& ready, Issue&& issue, Done&& done) {
    int k = 0;
    bool ok = true;
    for (; k < count && (ok = ready(k)); ++k) issue(k);
    for (int q = k > 2 ? k - 2 : 0; q < k; ++q) ok = done(q & 1, (unsigned)(q >> 1) & 1u) && ok;
    return ok;
}

}  // namespace ouc
