// Measurement helper of bench.py (print_scatter_rates), built as its own library (libdtb_bench_probe.so) and not part of
// libdtb.so: the rates at which this GPU makes the push scatter's scattered accesses into J, at J's
// layout (two planes of one float2 a neuron) and with a network's spread of targets.  Nothing in the
// simulator calls it.
#include <cuda_runtime.h>
#include <stdint.h>

namespace {

__device__ __forceinline__ uint32_t hash32(uint32_t x)
{
    x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; x ^= x >> 16;
    return x;
}

constexpr int kInFlight = 4;   // accesses per thread asked for together

// Access i goes to a neuron of the window (a region) that moves over all n with i, or, far_permille
// of 1000 times, to any neuron; the first or second plane as 80 % of the sources are excitatory.
// WHAT 0: float2 reduction; 1: the batch's sectors prefetched into L2 first; 2: a returning 32-bit
// claim and a 16-byte store (one ordered-push record).
template <int WHAT>
__global__ void __launch_bounds__(256) k_probe(float2* J, uint32_t* count, int64_t n, int64_t window, uint32_t far_permille,
                                               int64_t n_ops, uint32_t seed)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n_ops; i0 += stride * kInFlight) {
        float2* at[kInFlight];
        uint32_t cell[kInFlight];
#pragma unroll
        for (int u = 0; u < kInFlight; ++u) {
            const int64_t i = i0 + u * stride;
            at[u] = nullptr;
            if (i >= n_ops) continue;
            const uint32_t h = hash32((uint32_t)i ^ seed), g = hash32(h + 0x9e3779b9u);
            const bool far = g % 1000u < far_permille;
            const int64_t span = far ? n : window;
            const int64_t base = far ? 0 : (int64_t)((double)i / (double)n_ops * (double)(n - window));
            const int64_t t = base + (int64_t)(((uint64_t)h * (uint64_t)span) >> 32);   // < n
            cell[u] = (uint32_t)t;
            at[u] = J + ((g >> 10) % 5u == 0u ? n : 0) + t;
        }
        if (WHAT == 1) {
#pragma unroll
            for (int u = 0; u < kInFlight; ++u)
                if (at[u]) asm volatile("prefetch.global.L2 [%0];" :: "l"(at[u]));
        }
#pragma unroll
        for (int u = 0; u < kInFlight; ++u) {
            if (!at[u]) continue;
            if (WHAT == 2) {
                const uint32_t c = atomicAdd(count + cell[u], 1u);
                __stcg(reinterpret_cast<float4*>(J) + (cell[u] + (c & 1u) < n ? cell[u] + (c & 1u) : cell[u]),
                       make_float4(1.0f, 0.5f, 0.25f, 0.0f));
            } else {
                atomicAdd(at[u], make_float2(1.0f, 0.5f));
            }
        }
    }
}

}  // namespace

// ms_out = milliseconds for n_ops accesses (what: 0, 1, 2 as above) spread over the J of n neurons
// (fastest of 8 launches after 2).  Returns 0, or the CUDA error code.
extern "C" int dtb_bench_scatter_rate(int device, int what, int64_t n, int64_t n_ops, int64_t window, int far_permille,
                                      float* ms_out)
{
    if (!ms_out || what < 0 || what > 2 || n < 1 || n > 0x7fffffffLL || n_ops < 1 || window < 1 || window > n ||
        far_permille < 0 || far_permille > 1000)
        return -1;
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(device);
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    float2* J = nullptr;
    uint32_t* count = nullptr;
    cudaEvent_t a = nullptr, z = nullptr;
    cudaError_t e = cudaMalloc(&J, 2 * sizeof(float2) * (size_t)n);
    if (e == cudaSuccess) e = cudaMalloc(&count, sizeof(uint32_t) * (size_t)n);
    if (e == cudaSuccess) e = cudaMemset(J, 0, 2 * sizeof(float2) * (size_t)n);
    if (e == cudaSuccess) e = cudaMemset(count, 0, sizeof(uint32_t) * (size_t)n);
    if (e == cudaSuccess) e = cudaEventCreate(&a);
    if (e == cudaSuccess) e = cudaEventCreate(&z);
    float best = 0.0f;
    for (int r = 0; r < 10 && e == cudaSuccess; ++r) {
        const uint32_t seed = 12345u + 7919u * (uint32_t)r;   // other targets each time, as another step's
        cudaEventRecord(a);
        if (what == 0) k_probe<0><<<sms * 8, 256>>>(J, count, n, window, (uint32_t)far_permille, n_ops, seed);
        else if (what == 1) k_probe<1><<<sms * 8, 256>>>(J, count, n, window, (uint32_t)far_permille, n_ops, seed);
        else k_probe<2><<<sms * 8, 256>>>(J, count, n, window, (uint32_t)far_permille, n_ops, seed);
        cudaEventRecord(z);
        e = cudaEventSynchronize(z);
        float ms = 0.0f;
        if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, a, z);
        if (r >= 2 && (best == 0.0f || ms < best)) best = ms;
    }
    *ms_out = best;
    if (a) cudaEventDestroy(a);
    if (z) cudaEventDestroy(z);
    cudaFree(J);
    cudaFree(count);
    cudaSetDevice(prev);
    return e == cudaSuccess ? 0 : (int)e;
}
