// FFT ramp filter: transforms of 4096 and 8192 points.
#include "filter_fft.cuh"

namespace gct {

void launch_filter_fft_long(const FilterArgs &a, int L, int num_sms, cudaStream_t s)
{
    if (L == 4096) launch_log2<12>(a, num_sms, s);
    else launch_log2<13>(a, num_sms, s);
}

}  // namespace gct
