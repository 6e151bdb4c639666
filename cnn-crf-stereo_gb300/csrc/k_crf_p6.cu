// k_crf_p6.cu -- the CRF chain passes with 6 labels per lane (see k_crf_chain.cuh).  Compiled with --fmad=false.
#include "k_crf_chain.cuh"

namespace cnncrf {
namespace k {

int crf_pass_p6(const CrfPassArgs &a, bool hpass, int delta, const CrfForm &f, cudaStream_t st)
{
    return launch_pass<6>(a, hpass, delta, f, st);
}

} // namespace k
} // namespace cnncrf
