// Table rows streamed through shared memory, for tables that do not fit beside a block's records (a plan's 801 points
// for every step: 6.4 KB of float intervals a step, megabytes in all).
//
// A block of up to 1024 threads (one an SM) walks its pairs in step: the rows of a stage (a few batches of steps) are
// copied into one half of a ring with cp.async while the block computes on the other half, one barrier a stage. A step
// then waits for a shared-memory read where the table in global memory costs it an L1 lookup of some twenty lines; that
// counts while few warps are there to wait in turn (streams_rows).
#pragma once

#include "fused.cuh"

namespace ob {

// Cells from one row to the next in global memory: whole 16-byte words.
template <typename R>
inline int table_pitch(int n_x) {
    constexpr int per = 16 / static_cast<int>(sizeof(Pair2<R>)) > 0 ? 16 / static_cast<int>(sizeof(Pair2<R>)) : 1;
    return (n_x - 1 + per - 1) / per * per;
}

// The ring for batches of G steps of one name beside `used` bytes of shared memory within `budget`: up to 16 steps a
// stage; false when not even one batch a stage fits, or for rows of a single word (2^32 / chunks must fit 32 bits).
template <typename R>
inline bool plan_row_stream(RowStreamArgs& rs, int n_x, int G, size_t used, size_t budget) {
    rs.pitch = table_pitch<R>(n_x);
    const size_t row = static_cast<size_t>(rs.pitch) * sizeof(Pair2<R>);
    rs.chunks = static_cast<int>(row / 16);
    if (rs.chunks < 2) return false;
    rs.inv = static_cast<unsigned>(((1ull << 32) + rs.chunks - 1) / rs.chunks);
    rs.off = static_cast<int>((used + 15) & ~static_cast<size_t>(15));
    for (rs.batches = std::max(1, 16 / G); rs.batches >= 1; --rs.batches) {
        const size_t rows = static_cast<size_t>(rs.batches) * G;
        const unsigned long long words = static_cast<unsigned long long>(rows) * rs.chunks;
        if (rs.off + 2 * rows * row <= budget && words * rs.chunks < (1ull << 32)) return true;
    }
    return false;
}
inline size_t row_stream_bytes(const RowStreamArgs& rs, int G) {
    return 2 * static_cast<size_t>(rs.batches) * G * rs.chunks * 16;
}

// Whether a launch of n_pairs streams its rows: from kFirst warps an SM, where a block's warps share each row's copy, to
// `most`, from where enough warps hide the lookups and two unsynchronised blocks an SM do better than one in step.
// Kernel times through L1 against streamed, one name, 504 steps of 801-point rows: fused Phoenix 2^14 pairs 140 / 133
// us, 2^15 141 / 124, 2^15.5 144 / 140, 2^16 149 / 157; path engine's columns 2^14 248 / 189, 2^15 252 / 176, 2^16 260 /
// 207, 2^16.5 267 / 235, 2^17 297 / 296; Phoenix script 2^14 277 / 205, 2^15 280 / 215, 2^16 287 / 264, 2^16.5 293 /
// 293. (Two and three names put their legs on two lanes at the sizes where streaming would serve: legs_apart.)
inline bool streams_rows(long long n_pairs, int sms, double most) {
    constexpr double kFirst = 3.4;
    const double warps = static_cast<double>(n_pairs) / (32.0 * sms);
    return warps >= kFirst && warps < most;
}

// One block's ring of one name's rows. Every thread of the block makes the same calls in the same order: first() once, then turn() before
// each batch that opens a stage (opens()).
template <typename R, int G>
struct RowStream {
    const RowStreamArgs& rs;
    const Pair2<R>* tab;
    const NameStep<R>* ns;  // shared memory: row is the first cell of the step's row in tab
    unsigned char* sm;
    int steps, n_batches, cur, row0;

    __device__ __forceinline__ RowStream(const RowStreamArgs& r, const Pair2<R>* t, const NameStep<R>* s,
                                         unsigned char* shared, int S)
        : rs(r), tab(t), ns(s), sm(shared), steps(S), n_batches((S + G - 1) / G), cur(1), row0(0) {}

    __device__ __forceinline__ void issue(int batch, int half) {
        const int s0 = batch * G, rows = min(rs.batches * G, steps - s0), n = rows * rs.chunks;
        const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(sm + rs.off)) +
                             static_cast<uint32_t>(half * rs.batches * G * rs.chunks) * 16u;
        for (int c = threadIdx.x; c < n; c += blockDim.x) {
            const int row = static_cast<int>(__umulhi(static_cast<unsigned>(c), rs.inv));
            const char* src = reinterpret_cast<const char*>(tab + ns[s0 + row].row) + (c - row * rs.chunks) * 16;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + static_cast<uint32_t>(c) * 16u), "l"(src)
                         : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    __device__ __forceinline__ void first() { issue(0, 0); }
    __device__ __forceinline__ bool opens(int batch) const { return batch % rs.batches == 0; }
    // Before batch `batch`, which opens a stage: its rows have arrived in every thread's view and every warp is done
    // with the other half, which takes the next stage's rows (the first stage's, if another pass follows the last).
    __device__ __forceinline__ void turn(int batch, bool more) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        cur ^= 1;
        const int next = batch + rs.batches < n_batches ? batch + rs.batches : more ? 0 : -1;
        if (next >= 0) issue(next, cur ^ 1);
        row0 = (cur * rs.batches * G - batch * G) * rs.pitch;
    }
    // The cell of step i's (1-based) row, from the start of the ring.
    __device__ __forceinline__ int row(int i) const { return row0 + (i - 1) * rs.pitch; }
};

}  // namespace ob
