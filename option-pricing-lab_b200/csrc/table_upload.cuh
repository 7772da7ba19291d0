// A table of n_rows x n_x doubles as its (y_i, y_i+1 - y_i) intervals in R: into a host array (the staged blobs), or into
// global memory for tables beyond the stage, converted by the host threads straight into the pinned staging (the 801
// points of each of 504 steps, 3.2 MB of intervals: 0.59 ms as one thread's conversion and a pageable copy).
#pragma once

#include "host_copy.cuh"
#include "row_stream.cuh"

namespace ob {

inline size_t table_cells(int n_rows, int n_x) {
    return static_cast<size_t>(n_rows) * static_cast<size_t>(n_x - 1);
}

// Cells [first, first + count) into out, of rows of n_x - 1 intervals padded to `pitch` cells (the padding zero).
template <typename R>
inline void pack_table(const double* table, int n_x, int pitch, size_t first, size_t count, Pair2<R>* out) {
    const size_t w = static_cast<size_t>(n_x - 1), full = static_cast<size_t>(pitch);
    size_t row = first / full, k = first - row * full;
    for (size_t done = 0; done < count; ++row, k = 0) {
        const double* y = table + row * static_cast<size_t>(n_x);
        const size_t end = std::min(full, k + (count - done)), real = std::min(w, end);
        for (; k < real; ++k, ++done) out[done] = {static_cast<R>(y[k]), static_cast<R>(y[k + 1] - y[k])};
        for (; k < end; ++k, ++done) out[done] = {R(0), R(0)};
    }
}

// The table in global memory, its rows table_pitch cells apart, there for the work queued on st from then on.
template <typename R>
inline Pair2<R>* upload_table(DeviceArena& arena, const double* table, int n_rows, int n_x, cudaStream_t st) {
    const int pitch = table_pitch<R>(n_x);
    const size_t cells = static_cast<size_t>(n_rows) * static_cast<size_t>(pitch);
    Pair2<R>* d = arena.alloc<Pair2<R>>(cells);
    const bool staged = staged_upload(reinterpret_cast<char*>(d), cells * sizeof(Pair2<R>),
                                      [&](char* out, size_t at, size_t count) {
                                          pack_table<R>(table, n_x, pitch, at / sizeof(Pair2<R>),
                                                        count / sizeof(Pair2<R>), reinterpret_cast<Pair2<R>*>(out));
                                      });
    if (!staged) {
        std::vector<Pair2<R>> tab(cells);
        pack_table<R>(table, n_x, pitch, 0, cells, tab.data());
        upload_bytes(d, tab.data(), cells * sizeof(Pair2<R>), st);
    }
    return d;
}

}  // namespace ob
