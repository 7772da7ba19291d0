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

// The ring for batches of G steps of n names beside `used` bytes of shared memory within `budget`: up to 16 steps a
// stage; false when not even one batch a stage fits.
template <typename R>
inline bool plan_row_stream(RowStreamArgs& rs, int n_x, int n, int G, size_t used, size_t budget) {
    rs.pitch = table_pitch<R>(n_x);
    const size_t row = static_cast<size_t>(rs.pitch) * sizeof(Pair2<R>);
    rs.chunks = static_cast<int>(row / 16);
    rs.inv = static_cast<unsigned>(((1ull << 32) + rs.chunks - 1) / rs.chunks);
    rs.off = static_cast<int>((used + 15) & ~static_cast<size_t>(15));
    for (rs.batches = std::max(1, 16 / G); rs.batches >= 1; --rs.batches) {
        const size_t rows = static_cast<size_t>(rs.batches) * G * n;
        const unsigned long long words = static_cast<unsigned long long>(rows) * rs.chunks;
        if (rs.off + 2 * rows * row <= budget && words * rs.chunks < (1ull << 32)) return true;
    }
    return false;
}
inline size_t row_stream_bytes(const RowStreamArgs& rs, int n, int G) {
    return 2 * static_cast<size_t>(rs.batches) * G * n * rs.chunks * 16;
}

// Whether a launch of n_pairs on n names streams its rows. Kernel times, table through L1 against streamed, 504 steps of
// 801-point rows: one name 2^13 pairs 140 / 191 us, 2^14 138 / 133, 2^15 144 / 125, 2^16 194 / 157, 2^17 217 / 219, 2^19
// 767 / 815; three names (756 steps of 40 x 200) 2^13 346 / 351, 2^14 390 / 287, 2^16 800 / 483, 2^17 886 / 772, 2^18
// 1579 / 1521, 801-point rows 2^18 1305 / 1311. Below, a block's few warps share too little of each row's copy; above,
// enough warps hide the lookups, and two unsynchronised blocks an SM do better than one in step.
inline bool streams_rows(int n, long long n_pairs, int sms) {
    const double warps = static_cast<double>(n_pairs) / (32.0 * sms);  // an SM
    return warps >= 3.4 && warps < (n == 1 ? 24.0 : 40.0);
}

// One block's ring. Every thread of the block makes the same calls in the same order: first() once, then turn() before
// each batch that opens a stage (opens()).
template <typename R, int N, int G>
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
        const int s0 = batch * G, rows = min(rs.batches * G, steps - s0) * N, n = rows * rs.chunks;
        const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(sm + rs.off)) +
                             static_cast<uint32_t>(half * rs.batches * G * N * rs.chunks) * 16u;
        for (int c = threadIdx.x; c < n; c += blockDim.x) {
            const int row = static_cast<int>(__umulhi(static_cast<unsigned>(c), rs.inv));
            const char* src = reinterpret_cast<const char*>(tab + ns[s0 * N + row].row) + (c - row * rs.chunks) * 16;
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
        row0 = (cur * rs.batches * G - batch * G) * N * rs.pitch;
    }
    // The cell of step i's (1-based) row of name n, from the start of the ring.
    __device__ __forceinline__ int row(int i, int n) const { return row0 + ((i - 1) * N + n) * rs.pitch; }
};

}  // namespace ob
