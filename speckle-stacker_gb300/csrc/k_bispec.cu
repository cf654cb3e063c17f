// k_bispec.cu -- bispectrum accumulation launches (the kernel is in
// k_bispec.cuh), the Kahan normalise / merge kernels and the bounded-wait
// diagnostic.
#include "k_bispec.cuh"

namespace smip_gpu {

bool bispec_depth_supported(int De) { return De >= 2 && De <= 64 && De % 2 == 0; }

// partial sums of one split-tile part: (8 j x 4 l + 1 edge) float2 per thread, 512 threads
size_t bispec_scratch_bytes(int num_sms) { return (size_t)num_sms * kCtasPerSm * 33 * (512 / kCtasPerSm) * sizeof(float2); }
size_t bispec_tile_counters(int num_sms) { return (size_t)num_sms * kCtasPerSm; }

// The staging variant the stack's tuning chose: four frames per ring stage
// (here), or two (k_bispec_fps2.cu).
cudaError_t launch_bispec_accumulate(const BispecLaunch& L, const Geometry& g, cudaStream_t st)
{
    if (L.nframes <= 0)
        return cudaSuccess;
    if (L.variant == 1)
        return launch_bispec_accumulate_fps2(L, g, st);
    return launch_variant<4>(L, g, st);
}

// ------------------------------------------------ bounded-wait diagnostic
// The failure path every kernel takes when a wait expires, run on purpose:
// block 0 waits (bounded, as the bispectrum kernel's ring does) on an mbarrier
// that nothing arrives on; block 1 polls (bounded, as the phase walk does) a
// global flag that nothing sets.  Both record SMIP_DEV_ERR_TIMEOUT and return;
// no copy is in flight and nothing else waits on them.
__global__ void bounded_wait_probe_kernel(int* err, unsigned long long timeout_ns, const int* never)
{
    __shared__ __align__(8) uint64_t bar;
    if (blockIdx.x == 0) {
        if (threadIdx.x == 0) {
            mbar_init(&bar, 1);
            fence_mbar_init();
        }
        __syncthreads();
        const bool got = mbar_wait_bounded(&bar, 0, timeout_ns);
        if (!__all_sync(0xffffffffu, got) && threadIdx.x == 0)
            record_error(err, SMIP_DEV_ERR_TIMEOUT);
    } else {
        const unsigned long long t0 = globaltimer_ns();
        bool got = false;
        while (!(got = *reinterpret_cast<const volatile int*>(never) != 0) && globaltimer_ns() - t0 <= timeout_ns) {
        }
        if (!got && threadIdx.x == 0)
            record_error(err, SMIP_DEV_ERR_TIMEOUT);
    }
}

cudaError_t launch_bounded_wait_probe(int* err, const int* never, double timeout_s, cudaStream_t st)
{
    bounded_wait_probe_kernel<<<2, 32, 0, st>>>(err, (unsigned long long)(timeout_s * 1e9), never);
    note_launches(1);
    return cudaGetLastError();
}

// ------------------------------------------------------- normalise, merge
// (B - C) / n as FP64 arithmetic and one rounding give it, to the bit, but on the
// FP32 pipes (GB300's FP64 rate bound this kernel: 351 us at 256 x 256, d = 32,
// 1.3 TB/s; now 63 us, 7.1 TB/s of algorithmic bytes).  The difference is an exact float pair, its product
// with 1/n as a float pair is within 2^-45 of FP64's.  Where that leaves the
// rounding open (a value that close to the middle of two floats), and for values
// so small that the pair loses bits, infinities and NaN, the FP64 form decides.
// (a call, so that the compiler does not compute it beside the other form)
__device__ __noinline__ float normalized_f64(float b, float c, double inv_n)
{
    return (float)(((double)b - (double)c) * inv_n);
}
__device__ __forceinline__ float normalized(float b, float c, float ih, float il, double inv_n)
{
    float s, e;
    two_sum(b, -c, s, e);
    const float p = __fmul_rn(s, ih);
    const float q = fmaf(e, ih, fmaf(s, il, fmaf(s, ih, -p))), t = __fmul_rn(fabsf(p), 0x1p-44f);
    const float r = __fadd_rn(p, __fadd_rn(q, -t));
    if (r == __fadd_rn(p, __fadd_rn(q, t)) && fabsf(p) >= 0x1p-80f)
        return r;
    return s == 0.f ? p : normalized_f64(b, c, inv_n);
}

__global__ void __launch_bounds__(256) bispec_normalize_kernel(const float2* __restrict__ B, const float2* __restrict__ C,
                                                               double inv_n, long long count, float2* __restrict__ out)
{
    const float ih = (float)inv_n, il = (float)(inv_n - (double)ih);
    const long long step = (long long)gridDim.x * blockDim.x, pairs = count / 2; // the arrays are 256-byte aligned
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < pairs; i += step) {
        const float4 b = __ldcs(reinterpret_cast<const float4*>(B) + i), c = __ldcs(reinterpret_cast<const float4*>(C) + i);
        float4 o;
        o.x = normalized(b.x, c.x, ih, il, inv_n);
        o.y = normalized(b.y, c.y, ih, il, inv_n);
        o.z = normalized(b.z, c.z, ih, il, inv_n);
        o.w = normalized(b.w, c.w, ih, il, inv_n);
        reinterpret_cast<float4*>(out)[i] = o;
    }
    if ((count & 1) && blockIdx.x == 0 && threadIdx.x == 0) {
        const float2 b = B[count - 1], c = C[count - 1];
        out[count - 1] = make_float2(normalized(b.x, c.x, ih, il, inv_n), normalized(b.y, c.y, ih, il, inv_n));
    }
}

// dst += src, both Kahan pairs: the src sum (b - c) is added with compensation.
__global__ void bispec_merge_kernel(float2* __restrict__ Bd, float2* __restrict__ Cd, const float2* __restrict__ Bs,
                                    const float2* __restrict__ Cs, long long count)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count; i += (long long)gridDim.x * blockDim.x) {
        float2 b = Bd[i], c = Cd[i];
        const float2 sb = Bs[i], sc = Cs[i];
        const float vx = sb.x - sc.x, vy = sb.y - sc.y;
        const float yx = vx - c.x, yy = vy - c.y;
        const float tx = b.x + yx, ty = b.y + yy;
        c.x = (tx - b.x) - yx;
        c.y = (ty - b.y) - yy;
        Bd[i] = make_float2(tx, ty);
        Cd[i] = c;
    }
}

cudaError_t launch_bispec_normalize(const float2* B, const float2* C, double nframes, long long n, float2* out,
                                    cudaStream_t st)
{
    // eight blocks an SM, a few pairs a thread; fewer blocks for a small array
    const long long blocks = (n / 2 + 255) / 256;
    bispec_normalize_kernel<<<(int)(blocks < 1 ? 1 : blocks > 152 * 8 * 4 ? 152 * 8 * 4 : blocks), 256, 0, st>>>(B, C, 1.0 / nframes, n, out);
    note_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_bispec_merge(float2* Bd, float2* Cd, const float2* Bs, const float2* Cs, long long n,
                                cudaStream_t st)
{
    bispec_merge_kernel<<<2048, 256, 0, st>>>(Bd, Cd, Bs, Cs, n); note_launches(1);
    return cudaGetLastError();
}

} // namespace smip_gpu
