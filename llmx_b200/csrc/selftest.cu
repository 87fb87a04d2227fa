// Self-tests of what the kernels share: the bounded waits (tc_common.cuh) and the division without a branch (common.cuh).
//
// The bounded waits: a wait that nothing will ever satisfy runs out after the limit it is
// given, records its code in the error word, and the block goes on to its end.
//
// Every wait on an mbarrier in the tensor-core and attention kernels goes through tc::mbar_wait_limit (two seconds
// there).  This kernel makes that path run on purpose and harmlessly: one block initialises a barrier that expects one
// arrival, nobody arrives, and thread 0 waits on it with a limit of the caller's choosing (a millisecond in the
// tests).  Nothing hangs and nothing faults: the wait gives up, `error_word` holds ERR_SELFTEST_WAIT, `out[0]`
// says what the wait returned (1: completed, which would be a fault of the wait; 2: gave up) and the kernel returns.
#include "tc_common.cuh"

namespace {
constexpr int ERR_SELFTEST_WAIT = 105;

__global__ void wait_selftest_kernel(unsigned long long limit_ns, int* error_word, int* out) {
    __shared__ uint64_t bar;
    __shared__ int abort_flag;
    if (threadIdx.x == 0) {
        tc::mbar_init(&bar, 1);
        tc::fence_barrier_init();
        abort_flag = 0;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const bool completed = tc::mbar_wait_limit(&bar, 0, &abort_flag, error_word, ERR_SELFTEST_WAIT, limit_ns);
        out[0] = completed ? 1 : 2;
    }
    __syncthreads();
    // What a kernel's other warps do after a failed wait: every later wait returns at once.
    if (threadIdx.x == 32) out[1] = tc::mbar_wait_limit(&bar, 0, &abort_flag, error_word, ERR_SELFTEST_WAIT, limit_ns) ? 1 : 2;
}

// A warp's wait whose lanes would not agree: the even lanes' barrier has completed, nobody arrives at the odd lanes'.  All
// lanes must come back with the same answer, or the warp-wide instruction after it would wait for lanes that went elsewhere.
__global__ void warp_wait_selftest_kernel(unsigned long long limit_ns, int* error_word, int* out) {
    __shared__ uint64_t bars[2];
    __shared__ int abort_flag;
    if (threadIdx.x == 0) {
        tc::mbar_init(&bars[0], 1);
        tc::mbar_init(&bars[1], 1);
        tc::fence_barrier_init();
        tc::mbar_arrive(&bars[0]);
        abort_flag = 0;
    }
    __syncwarp();
    const bool ok = tc::mbar_wait_warp_limit(&bars[threadIdx.x & 1], 0, &abort_flag, error_word, ERR_SELFTEST_WAIT, limit_ns);
    out[threadIdx.x] = ok ? 1 : 2;
}

__global__ void quotient_selftest_kernel(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ out, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = quotient(a[i], b[i]);
}
}  // namespace

// limit_ns: 1,000 .. 100,000,000 (a tenth of a second at most).  out: two device ints.
LLMX_EXPORT int llmx_wait_selftest(unsigned long long limit_ns, int* error_word, int* out, cudaStream_t stream) {
    if (!error_word || !out || limit_ns < 1000ull || limit_ns > 100000000ull) return LLMX_ERR_BAD_ARGUMENT;
    wait_selftest_kernel<<<1, 64, 0, stream>>>(limit_ns, error_word, out);
    return launch_status();
}

// The same for a warp's wait; out: 32 device ints, what each lane's wait returned.
LLMX_EXPORT int llmx_warp_wait_selftest(unsigned long long limit_ns, int* error_word, int* out, cudaStream_t stream) {
    if (!error_word || !out || limit_ns < 1000ull || limit_ns > 100000000ull) return LLMX_ERR_BAD_ARGUMENT;
    warp_wait_selftest_kernel<<<1, 32, 0, stream>>>(limit_ns, error_word, out);
    return launch_status();
}

// out[i] = a[i] / b[i] for b[i] >= 1 as the kernels divide.
LLMX_EXPORT int llmx_quotient_selftest(const float* a, const float* b, float* out, long long n, cudaStream_t stream) {
    if (!a || !b || !out || n <= 0 || n > (1ll << 32)) return LLMX_ERR_BAD_ARGUMENT;
    quotient_selftest_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(a, b, out, n);
    return launch_status();
}
