// k_crf_p12.cu -- the CRF chain passes with 1 and 2 labels per lane (see k_crf_chain.cuh).  Compiled with --fmad=false.
#include "k_crf_chain.cuh"

namespace cnncrf {
namespace k {

int crf_pass_p1(const CrfPassArgs &a, bool hpass, int delta, const CrfForm &f, cudaStream_t st)
{
    return launch_pass<1>(a, hpass, delta, f, st);
}
int crf_pass_p2(const CrfPassArgs &a, bool hpass, int delta, const CrfForm &f, cudaStream_t st)
{
    return launch_pass<2>(a, hpass, delta, f, st);
}

} // namespace k
} // namespace cnncrf
