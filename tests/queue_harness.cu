// Two warps of a block on its stage queues (stage_queues.cuh), which pass one
// path to each other: a warp holds it for some 30 us, puts it, and waits until
// the other has taken it (at most 2 ms).  A warp's polls of empty queues end it
// after kPolls in a row: far more than one wait takes, far fewer than all do.
// Prints "<takes of warp 0> <takes of warp 1> <status>", and of a warp that has had
// 2^32 - 1 batches and takes another without a limit "<taken> <batches> <status>".

#include <cstdio>

#include "stage_queues.cuh"

using namespace sky::wave;

constexpr uint32_t kRounds = 400, kPolls = 4000;

__global__ void __launch_bounds__(64) pass_a_path(uint32_t* out, uint32_t* status) {
    __shared__ __align__(16) unsigned char smem[sizeof(Queues) + kQueues * 32u * sizeof(uint16_t)];
    Queues* const q = reinterpret_cast<Queues*>(smem);
    const StageQueues queues(q, 32u, 1u);
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t turn = 0u, idle = 0u, batch = 0u, stage = 0u, count = 0u, id = 0u;
    for (uint32_t tries = 0u; tries < (1u << 20); ++tries) {
        const Taken taken = queues.take<kPolls>(lane, turn, idle, batch, ~0u, status, stage, count, id);
        if (taken == kOutOfWork) break;
        if (taken == kNothing) continue;
        for (int i = 0; i < 30; ++i) __nanosleep(1000);
        __syncwarp();
        if (batch >= kRounds / 2u) {
            if (lane == 0u) atomicSub(&q->live, 1u);
            break;
        }
        queues.put(lane, lane == 0u ? uint32_t(kQTrack) : uint32_t(kQNone), 0u, status);
        for (int i = 0; i < 20000; ++i) {  // until it is taken
            const uint32_t waiting = *reinterpret_cast<volatile uint32_t*>(&q->tail[kQTrack]) -
                                     *reinterpret_cast<volatile uint32_t*>(&q->head[kQTrack]);
            if (__shfl_sync(0xffffffffu, waiting, 0) == 0u) break;
            __nanosleep(100);
            __syncwarp();
        }
    }
    if (lane == 0u) out[threadIdx.x >> 5] = batch;
}

__global__ void __launch_bounds__(32) one_more(uint32_t* out, uint32_t* status) {
    __shared__ __align__(16) unsigned char smem[sizeof(Queues) + kQueues * 32u * sizeof(uint16_t)];
    const StageQueues queues(reinterpret_cast<Queues*>(smem), 32u, 1u);
    __syncthreads();
    uint32_t turn = 0u, idle = 0u, batch = ~0u, stage = 0u, count = 0u, id = 0u;
    const Taken taken =
        queues.take<kMaxIdlePolls, false>(threadIdx.x, turn, idle, batch, 0u, status, stage, count, id);
    if (threadIdx.x == 0u) {
        out[0] = taken == kBatch;
        out[1] = batch;
    }
}

int main() {
    uint32_t *d = nullptr, h[6] = {};
    if (cudaMalloc(&d, sizeof(h)) != cudaSuccess || cudaMemset(d, 0, sizeof(h)) != cudaSuccess) return 1;
    pass_a_path<<<1, 64>>>(d, d + 2);
    one_more<<<1, 32>>>(d + 3, d + 5);
    if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    std::printf("%u %u %u\n%u %u %u\n", h[0], h[1], h[2], h[3], h[4], h[5]);
    return 0;
}
