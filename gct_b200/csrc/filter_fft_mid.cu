// FFT ramp filter: transforms of 1024 and 2048 points.
#include "filter_fft.cuh"

namespace gct {

void launch_filter_fft_mid(const FilterArgs &a, int L, int num_sms, cudaStream_t s)
{
    if (L == 1024) launch_log2<10>(a, num_sms, s);
    else launch_log2<11>(a, num_sms, s);
}

}  // namespace gct
