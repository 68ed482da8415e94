// stage_queues.cuh — the queues of a block's paths by the stage that each needs
// next, for kernels that keep their paths in shared memory (trace_wave.cuh,
// adjoint_wave.cu): a warp takes up to 32 paths of one stage, and puts each
// where it has to go on.  No block barrier, no lock: a take is one
// compare-and-swap on a queue's head, a put one addition to its tail.

#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace sky {
namespace wave {

enum : uint32_t { kQTrack = 0u, kQVertex = 1u, kQContinue = 2u, kQStart = 3u, kQueues = 4u, kQNone = 7u };

// Polls of empty queues (>= 100 ns each) between two batches of a warp before status bit 2.
constexpr uint32_t kIdleBits = 26;
constexpr uint32_t kMaxIdlePolls = (1u << kIdleBits) - 1u;
constexpr uint32_t kMaxSlotPolls = 1u << 24;   // polls of one queue slot before the same

// The stage queues of a block: rings of path numbers with counters of what was
// ever taken (head) and put (tail).  A slot holds kEmpty unless a path number
// is waiting in it.
constexpr uint32_t kEmpty = 0xffffu;
struct Queues {
    uint32_t head[kQueues];
    uint32_t tail[kQueues];
    uint32_t live;   // paths that may still have work
    uint32_t _pad[3];
};

__host__ __device__ inline uint32_t queue_slots(uint32_t paths) {
    uint32_t n = 32u;
    while (n < paths) n <<= 1;
    return n;
}

__host__ __device__ inline size_t align16(size_t v) { return (v + 15u) & ~size_t(15u); }
// Orders a warp's accesses to paths before (after) it puts them into (takes
// them from) a queue.
__device__ __forceinline__ void fence_block() { asm volatile("fence.acq_rel.cta;" ::: "memory"); }

__device__ __forceinline__ float as_f(uint32_t v) { return __uint_as_float(v); }
__device__ __forceinline__ uint32_t as_u(float v) { return __float_as_uint(v); }

// What a take found.
enum Taken : uint32_t { kOutOfWork, kNothing, kBatch };

struct StageQueues {
    Queues* Q;
    volatile uint16_t* slots;
    uint32_t ring;

    // Sets up the queues behind `q`: paths 0 .. used - 1 wait in the start queue.
    // The block's barrier before the first take is the caller's.
    __device__ __forceinline__ StageQueues(Queues* q, uint32_t paths, uint32_t used)
        : Q(q), slots(reinterpret_cast<volatile uint16_t*>(q + 1)), ring(queue_slots(paths)) {
        for (uint32_t i = threadIdx.x; i < kQueues * ring; i += blockDim.x)
            slots[i] = uint16_t(i >= kQStart * ring && i < kQStart * ring + used ? i - kQStart * ring : kEmpty);
        if (threadIdx.x < kQueues) {
            Q->head[threadIdx.x] = 0u;
            Q->tail[threadIdx.x] = threadIdx.x == kQStart ? used : 0u;
        }
        if (threadIdx.x == 0u) Q->live = used;
    }

    // The whole warp: up to 32 paths of one stage (lane i < take has path `id`).
    // `turn` is the stage that the warp prefers, `batch` counts its batches, `idle` its
    // polls of empty queues, under the low bits of the batch count that they came after.
    // `batch_limit`: batches before status bit 2 (kLimited).
    template <uint32_t kMaxPolls = kMaxIdlePolls, bool kLimited = true>
    __device__ __forceinline__ Taken take(uint32_t lane, uint32_t& turn, uint32_t& idle, uint32_t& batch,
                                          uint32_t batch_limit, uint32_t* status, uint32_t& stage, uint32_t& count,
                                          uint32_t& id) const {
        // lanes 0-3 look at one queue each.  A lane's head, read before its tail, goes with
        // its own count: the exchange below fails if the head has moved since, so what it
        // takes has been put there.
        uint32_t h = 0u, waiting = 0u;
        if (lane < kQueues) {
            h = *reinterpret_cast<volatile uint32_t*>(&Q->head[lane]);
            waiting = *reinterpret_cast<volatile uint32_t*>(&Q->tail[lane]) - h;
        }
        // a full batch if there is one, of the warp's last stage rather than of another:
        // warps that stay with a stage keep its code in the instruction caches (fullest
        // queue first: +8 %, stages in turn: +4 %); else the fullest queue
        const uint32_t full = __ballot_sync(0xffffffffu, waiting >= 32u);
        count = 32u;
        if (full) {
            stage = (uint32_t(__ffs(int((full | (full << 4)) >> turn))) - 1u + turn) & 3u;
            turn = stage;
        } else {
            const uint32_t best = __reduce_max_sync(0xffffffffu, (waiting << 2) | (lane & 3u));
            stage = best & 3u;
            count = min(best >> 2, 32u);
        }
        if (count == 0u) {
            // one lane looks for all: the warp leaves together
            if (__shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t*>(&Q->live), 0) == 0u) return kOutOfWork;
            // polls before the last batch don't count, or a launch of many minutes would end here
            // (set back with each batch instead, `idle` costs the LUT case 1.2 %, this 0.9 %)
            if ((idle ^ (batch << kIdleBits)) >> kIdleBits) idle = batch << kIdleBits;
            if ((++idle & kMaxIdlePolls) >= kMaxPolls) {
                if (lane == 0u) atomicOr(status, 2u);
                return kOutOfWork;
            }
            __nanosleep(100);
            __syncwarp();
            return kNothing;
        }
        if (kLimited && batch >= batch_limit) {  // warp-uniform
            if (lane == 0u) atomicOr(status, 2u);
            return kOutOfWork;
        }
        h = __shfl_sync(0xffffffffu, h, stage);
        uint32_t seen = 0u;
        if (lane == 0u) seen = atomicCAS(&Q->head[stage], h, h + count);
        if (__shfl_sync(0xffffffffu, seen, 0) != h) return kNothing;  // another warp was first
        ++batch;
        id = 0u;
        if (lane < count) {
            volatile uint16_t* slot = slots + stage * ring + ((h + lane) & (ring - 1u));
            uint32_t v = *slot, polls = 0u;
            while (v == kEmpty && ++polls < kMaxSlotPolls) v = *slot;  // put, but not yet written
            *slot = uint16_t(kEmpty);
            id = v;
            if (v == kEmpty) {
                atomicOr(status, 2u);
                id = 0u;
            }
        }
        fence_block();
        return kBatch;
    }

    // The whole warp: each lane's path into queue `next` (kQNone: no path).  One lane
    // of those that go to a queue takes room for all of them.
    __device__ __forceinline__ void put(uint32_t lane, uint32_t next, uint32_t id, uint32_t* status) const {
        const uint32_t own = __match_any_sync(0xffffffffu, next);
        const uint32_t first = uint32_t(__ffs(int(own))) - 1u;
        fence_block();
        uint32_t room = 0u;
        if (lane == first && next != kQNone) room = atomicAdd(&Q->tail[next], uint32_t(__popc(own)));
        room = __shfl_sync(0xffffffffu, room, first);
        if (next != kQNone) {
            volatile uint16_t* slot =
                slots + next * ring + ((room + __popc(own & ((1u << lane) - 1u))) & (ring - 1u));
            uint32_t polls = 0u;
            while (*slot != kEmpty && ++polls < kMaxSlotPolls) {}  // its last path is being taken
            if (polls >= kMaxSlotPolls) atomicOr(status, 2u);
            *slot = uint16_t(id);
        }
        __syncwarp();
    }
};

}  // namespace wave
}  // namespace sky
