// The back projector's wait for a window's copy (bp_fast.cuh) when no copy comes: one warp waits for a barrier that nothing
// completes, gives up after the limit, flags the error word and says so in every lane; with the flag already set it gives
// up sooner, and a barrier that a copy's bytes do complete ends the wait as it should.  Prints "ok <ms> <ms>".
#include <cstdio>

#include "../mbirjax_b200/csrc/bp_fast.cuh"

namespace mbx {
int num_sms() { return 148; }
}  // namespace mbx

using namespace mbx;

// out: [0] lanes whose first wait succeeded, [1] its time in ns, [2], [3] the same of a second wait on the other barrier,
// [4] lanes whose wait for a completed barrier succeeded, [5] failed
__global__ void wait_kernel(long long *out, int *err) {
    __shared__ __align__(16) float bars[8];
    BpfPipe p = bpf_pipe_init(bars);
    for (int b = 0; b < 2; ++b) {
        const unsigned long long t0 = bpf_now_ns();
        const bool ok = bpf_pipe_wait(p, b, err);
        out[2 * b] = __popc(__ballot_sync(0xffffffffu, ok));
        out[2 * b + 1] = (long long)(bpf_now_ns() - t0);
    }
    out[5] = p.failed;
    __syncwarp();
    p = bpf_pipe_init(bars + 4);
    if (threadIdx.x == 0) asm volatile("mbarrier.arrive.shared.b64 _, [%0];" ::"r"(p.bar) : "memory");
    out[4] = __popc(__ballot_sync(0xffffffffu, bpf_pipe_wait(p, 0, err)));
}

int main() {
    long long *out, h[6];
    int *err, e = 0;
    cudaMalloc(&out, sizeof(h));
    cudaMalloc(&err, sizeof(int));
    cudaMemset(err, 0, sizeof(int));
    wait_kernel<<<1, 32>>>(out, err);
    if (cudaMemcpy(h, out, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess ||
        cudaMemcpy(&e, err, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) {
        std::printf("FAIL cuda %s\n", cudaGetErrorString(cudaGetLastError()));
        return 1;
    }
    const bool good = h[0] == 0 && h[2] == 0 && h[4] == 32 && h[5] == 1 && e == MBX_DEVICE_ERROR_INTERNAL &&
                      h[1] >= (long long)BPF_WAIT_NS && h[1] < 2000000000LL && h[3] >= (long long)BPF_WAIT_AGAIN_NS &&
                      h[3] < 1000000000LL;
    std::printf("%s %lld %lld (%lld %lld %lld %lld %d)\n", good ? "ok" : "FAIL", h[1] / 1000000, h[3] / 1000000, h[0], h[2],
                h[4], h[5], e);
    return good ? 0 : 1;
}
