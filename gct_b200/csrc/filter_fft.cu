// FFT ramp filter: short transforms, the choice of the length, and the kernels beside it (view maxima and
// scales, redundancy weights).
#include <algorithm>

#include "filter_fft.cuh"

namespace gct {
namespace {

__global__ void view_absmax_kernel(const float *__restrict__ proj, long long pix_per_view,
                                   float *amax)
{
    const int v = blockIdx.y;
    const float *p = proj + static_cast<long long>(v) * pix_per_view;
    float m = 0.f;
    for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < pix_per_view;
         i += static_cast<long long>(gridDim.x) * blockDim.x)
        m = fmaxf(m, fabsf(__ldg(p + i)));
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(reinterpret_cast<int *>(amax + v), __float_as_int(m));
}

__global__ void view_scales_kernel(const float *amax, int nv, float l1, float *vscale, float *vinv)
{
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nv) return;
    const float e = view_exponent(amax[v], l1);
    vscale[v] = exp2f(e);
    vinv[v] = exp2f(-e);
}

// One thread per weight. FP64 steps as in parker_table, each rounded by itself, so that a weight falls
// into the same window; sin() may differ in the last bit. 184 000 weights took the host 2 ms.
__global__ void parker_kernel(const double *__restrict__ gamma, const double *__restrict__ rel, double phi,
                              float constant, int nv, int nc, float *__restrict__ out)
{
    constexpr double kPi = 3.14159265358979323846;
    const long long n = static_cast<long long>(nv) * nc;
    for (long long e = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; e < n;
         e += static_cast<long long>(gridDim.x) * blockDim.x) {
        if (!gamma) {
            out[e] = constant;
            continue;
        }
        const int v = static_cast<int>(e / nc), c = static_cast<int>(e - static_cast<long long>(v) * nc);
        const double b = rel[v], g2 = 2.0 * gamma[c];
        const double t2 = __dadd_rn(__dadd_rn(g2, phi), -kPi), t3 = __dadd_rn(g2, kPi);
        const double p2 = 2.0 * __dadd_rn(phi, -kPi), g4 = 2.0 * g2;
        double w = 0.0;
        if (b >= 0.0 && b <= t2) {
            const double s = sin(__ddiv_rn(__dmul_rn(kPi, b), __dadd_rn(p2, g4)));
            w = __dmul_rn(s, s);
        } else if (b >= t2 && b <= t3) {
            w = 1.0;
        } else if (b >= t3 && b <= phi) {
            const double s = sin(__ddiv_rn(__dmul_rn(kPi, __dadd_rn(phi, -b)), __dadd_rn(p2, -g4)));
            w = __dmul_rn(s, s);
        }
        out[e] = static_cast<float>(w);
    }
}

}  // namespace

void launch_parker(const double *gamma, const double *rel, double phi, float constant, int nv, int nc, float *out,
                   cudaStream_t s)
{
    const long long n = static_cast<long long>(nv) * nc;
    const long long grid = std::min<long long>((n + 255) / 256, 148LL * 16);
    parker_kernel<<<static_cast<unsigned>(grid < 1 ? 1 : grid), 256, 0, s>>>(gamma, rel, phi, constant, nv, nc, out);
}

void launch_filter_fft(const FilterArgs &a, int L, int num_sms, cudaStream_t s)
{
    switch (L) {
        case 256: launch_log2<8>(a, num_sms, s); break;
        case 512: launch_log2<9>(a, num_sms, s); break;
        case 1024:
        case 2048: launch_filter_fft_mid(a, L, num_sms, s); break;
        case 4096:
        case 8192: launch_filter_fft_long(a, L, num_sms, s); break;
        default: break;  // rejected on the host
    }
}

void launch_view_absmax(const float *proj, int nv, long long pix_per_view, float *amax,
                        cudaStream_t s)
{
    long long bx = (pix_per_view + 256 * 8 - 1) / (256 * 8);
    if (bx > 64) bx = 64;
    if (bx < 1) bx = 1;
    view_absmax_kernel<<<dim3(static_cast<unsigned>(bx), nv), 256, 0, s>>>(proj, pix_per_view, amax);
}

void launch_view_scales(const float *amax, int nv, float l1, float *vscale, float *vinv,
                        cudaStream_t s)
{
    view_scales_kernel<<<(nv + 127) / 128, 128, 0, s>>>(amax, nv, l1, vscale, vinv);
}

}  // namespace gct
