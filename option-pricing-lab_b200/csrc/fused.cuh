// The specialised fused kernel: every name of one kind (Black-Scholes, local vol, Heston by Euler, SLV, or one Heston
// name by QE), N names known at compile time, everything a step reads staged in shared memory.
//
// Per step and name one 16-byte record {lo, inv_dx, log-forward at the step end, table row} (32 bytes in double)
// is read as a warp-wide broadcast; the local-variance table is stored as (y_i, y_i+1) pairs so that an
// interpolation is one 8-byte shared load. Normals are drawn in batches of G steps whose count is a multiple of four,
// so each Philox block fills registers by constant indices; the correlated normal root z is computed once per pair
// and step and used with both signs (the reference's two legs read the same z with opposite signs,
// RC/include/optlab_cuda/paths.hpp:301-329). Each leg's step is the reference's arithmetic up to reassociation:
// x += var (-dt / 2) + sqrt(var) sqrt(dt) z with -dt / 2 and sqrt(dt) precomputed per step, and the table read as
// y + w dy.
#pragma once

#include "model.cuh"

namespace ob {

// org and inv_dx locate x in the step's row: in the cell form (set_cell_row, the fused, script and path kernels) or in
// the form of u = table_u(step, x) (the adjoint): -lo inv_dx in float (u = x inv_dx + org, one multiply-add), lo in
// double (u = (x - lo) inv_dx, the reference's order).
template <typename R>
struct alignas(16) NameStep;
template <>
struct alignas(16) NameStep<float> {
    float org, inv_dx, lf;
    int row;  // first (y_i, y_i+1) pair of the step's table row
};
template <>
struct alignas(16) NameStep<double> {
    double org, inv_dx, lf;
    int row, pad;
};

__host__ __device__ inline float name_step_org(double lo, double inv_dx, float*) {
    return static_cast<float>(-lo * inv_dx);
}
__host__ __device__ inline double name_step_org(double lo, double, double*) { return lo; }
// The origin to store for a row starting at lo with 1 / dx = inv_dx.
template <typename R>
__host__ __device__ inline R name_step_org(double lo, double inv_dx) {
    return name_step_org(lo, inv_dx, static_cast<R*>(nullptr));
}

__device__ __forceinline__ float table_u(float org, float inv_dx, float x) { return fmaf(x, inv_dx, org); }
__device__ __forceinline__ double table_u(double org, double inv_dx, double x) { return (x - org) * inv_dx; }
template <typename R>
__device__ __forceinline__ R table_u(const NameStep<R>& s, R x) {
    return table_u(s.org, s.inv_dx, x);
}

// The cell form of a row, for the kernels that need only a coordinate's interval and weight (the fused, script and
// path kernels; the adjoint keeps table_u's form for its derivative). In float the coordinate is stored divided by
// top, so that its clamp to [0, top] is the saturation of its multiply-add: u / top = sat(x inv_dx / top - lo inv_dx
// / top). In double the row keeps table_u's form.
inline void cell_row(double lo, double inv_dx, float top, float& org, float& inv) {
    org = static_cast<float>(-lo * inv_dx / top), inv = static_cast<float>(inv_dx / top);
}
inline void cell_row(double lo, double inv_dx, double, double& org, double& inv) { org = lo, inv = inv_dx; }
template <typename R>
inline void set_cell_row(NameStep<R>& r, double lo, double inv_dx, R top) {
    cell_row(lo, inv_dx, top, r.org, r.inv_dx);
}

// The interval j = floor(u) and the weight f = u - j of x's coordinate u, clamped to [0, top], in a row of the cell
// form. Float: s = sat(x inv_dx' + org') = u / top; s top + 2^23 rounded toward zero is a float in [2^23, 2^24)
// whose low mantissa bits hold floor(u) exactly (u < 2^23), and f = s top - floor(u) in one more multiply-add (the
// subtraction 2^23 - that float is exact). Four FMA-pipe instructions where the clamp, the conversion to an integer
// and back and the subtraction take six, two of them on the MUFU pipe. Double: the clamp and the conversions.
__device__ __forceinline__ void table_cell(float org, float inv, float top, float x, int& j, float& f) {
    float s;
    asm("fma.rn.ftz.sat.f32 %0, %1, %2, %3;" : "=f"(s) : "f"(x), "f"(inv), "f"(org));
    const float big = __fmaf_rz(s, top, 8388608.0f);
    j = __float_as_int(big) - 0x4B000000;
    f = fmaf(s, top, 8388608.0f - big);
}
__device__ __forceinline__ void table_cell(double org, double inv, double top, double x, int& j, double& f) {
    const double u = fmin(fmax(table_u(org, inv, x), 0.0), top);
    j = static_cast<int>(u);
    f = u - static_cast<double>(j);
}
template <typename R>
__device__ __forceinline__ void table_cell(const NameStep<R>& r, R top, R x, int& j, R& f) {
    table_cell(r.org, r.inv_dx, top, x, j, f);
}

// One leg's log-spot step, x + var (-dt / 2) + sqrt(var) (sqrt(dt) z): in float as two multiply-adds (the drift into
// x, then the diffusion), in double in the reference's grouping (the two terms summed, then added to x).
__device__ __forceinline__ float lv_advance(float x, float var, float hdt, float zd) {
    return fmaf(sqrtf(var), zd, fmaf(var, hdt, x));
}
__device__ __forceinline__ double lv_advance(double x, double var, double hdt, double zd) {
    return x + fma(sqrt(var), zd, var * hdt);
}

// Two floats as one 64-bit register pair, for Blackwell's packed single-precision instructions: one issue slot for two
// multiply-adds, each rounded (and flushed) as the scalar instruction's, so packed and scalar code agree bit for bit.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 fma2_rz(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rz.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// lv_advance of both legs of a pair on the antithetic normal: x0 on sqrt(dt) z, x1 on its negative.
__device__ __forceinline__ void lv_advance_legs(float& x0, float& x1, float var0, float var1, float hdt, float zd) {
    const f32x2 drifted = fma2(pack2(var0, var1), pack2(hdt, hdt), pack2(x0, x1));
    unpack2(fma2(pack2(sqrtf(var0), sqrtf(var1)), pack2(zd, -zd), drifted), x0, x1);
}
__device__ __forceinline__ void lv_advance_legs(double& x0, double& x1, double var0, double var1, double hdt,
                                                double zd) {
    x0 = lv_advance(x0, var0, hdt, zd), x1 = lv_advance(x1, var1, hdt, -zd);
}

// The running extremes of a path: m_min(a, b) and m_max(a, b) in one instruction each. A NaN in b gives NaN, as there;
// a is NaN only once an earlier b was, and a log performance that is NaN once stays NaN.
__device__ __forceinline__ float run_min(float a, float b) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float run_max(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
// run_min over two values in order, one three-input instruction.
__device__ __forceinline__ float run_min(float a, float b, float c) {
    float r;
    asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ double run_min(double a, double b) { return m_min(a, b); }
__device__ __forceinline__ double run_max(double a, double b) { return m_max(a, b); }
__device__ __forceinline__ double run_min(double a, double b, double c) { return m_min(m_min(a, b), c); }

// One table interval: the value at its left point and the increment to the right one, so that an interpolation is
// one multiply-add (y + w dy, the reference's y_i (1 - w) + y_i+1 w up to rounding).
template <typename R>
struct alignas(2 * sizeof(R)) Pair2 {
    R a, b;
};

// An interval of a table left in global memory (too large for the shared-memory stage): one 8- or 16-byte load
// through the read-only data cache.
__device__ __forceinline__ Pair2<float> ldg_pair(const Pair2<float>* p) {
    const float2 v = __ldg(reinterpret_cast<const float2*>(p));
    return {v.x, v.y};
}
__device__ __forceinline__ Pair2<double> ldg_pair(const Pair2<double>* p) {
    const double2 v = __ldg(reinterpret_cast<const double2*>(p));
    return {v.x, v.y};
}

// Where a kernel reads its table: the stage, global memory, or rows streamed through a ring in shared memory.
constexpr int kTabStaged = 0, kTabGlobal = 1, kTabStreamed = 2;

// The local variances of both legs of a pair at x0 and x1 in a step's row of the table: table_cell of each leg and one
// load and multiply-add each. MODE kTabStaged: the table is staged in shared memory, at shared address tab_s; kTabGlobal: in global memory
// (ldg_pair); kTabStreamed: the row is in a ring in the dynamic shared memory sm, tab_s its offset there. Float: the cell's last three
// operations packed, and the interval's address straight from the bits of s top + 2^23, one shift-and-add with the offset
// 2^23's own bits leave (0x4B000000, times 8 modulo 2^32) folded into the row's address. (The staged load has no memory
// clobber: its address depends on the row read after the barrier that follows the staging, and nothing writes the table
// after it. A ring is rewritten, so its loads are plain ones, which no barrier lets pass.)
template <int MODE>
__device__ __forceinline__ void table_vars(const Pair2<float>* tab, const unsigned char* sm, uint32_t tab_s, float org,
                                           float inv, int row, float top, float x0, float x1, float& var0,
                                           float& var1) {
    float s0, s1, b0, b1, f0, f1;
    asm("fma.rn.ftz.sat.f32 %0, %1, %2, %3;" : "=f"(s0) : "f"(x0), "f"(inv), "f"(org));
    asm("fma.rn.ftz.sat.f32 %0, %1, %2, %3;" : "=f"(s1) : "f"(x1), "f"(inv), "f"(org));
    const f32x2 s = pack2(s0, s1), t = pack2(top, top), two23 = pack2(8388608.0f, 8388608.0f);
    const f32x2 big = fma2_rz(s, t, two23);
    unpack2(big, b0, b1);
    unpack2(fma2(s, t, fma2(big, pack2(-1.0f, -1.0f), two23)), f0, f1);  // (2^23 - big is exact)
    const uint32_t i0 = __float_as_uint(b0), i1 = __float_as_uint(b1);
    Pair2<float> y0, y1;
    if (MODE == kTabGlobal) {
        y0 = ldg_pair(tab + row + static_cast<int>(i0 - 0x4B000000u));
        y1 = ldg_pair(tab + row + static_cast<int>(i1 - 0x4B000000u));
    } else {
        const uint32_t base = tab_s + 8u * static_cast<uint32_t>(row) - 8u * 0x4B000000u;
        if (MODE == kTabStaged) {
            asm("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(y0.a), "=f"(y0.b) : "r"(i0 * 8u + base));
            asm("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(y1.a), "=f"(y1.b) : "r"(i1 * 8u + base));
        } else {
            y0 = *reinterpret_cast<const Pair2<float>*>(sm + (i0 * 8u + base));
            y1 = *reinterpret_cast<const Pair2<float>*>(sm + (i1 * 8u + base));
        }
    }
    var0 = fmaf(f0, y0.b, y0.a), var1 = fmaf(f1, y1.b, y1.a);
}
template <int MODE>
__device__ __forceinline__ void table_vars(const Pair2<double>* tab, const unsigned char*, uint32_t, double org, double inv, int row, double top, double x0, double x1,
                                           double& var0, double& var1) {
    static_assert(MODE != kTabStreamed, "rows are streamed in float");
    int j0, j1;
    double f0, f1;
    table_cell(org, inv, top, x0, j0, f0), table_cell(org, inv, top, x1, j1, f1);
    const Pair2<double> y0 = MODE == kTabGlobal ? ldg_pair(tab + row + j0) : tab[row + j0];
    const Pair2<double> y1 = MODE == kTabGlobal ? ldg_pair(tab + row + j1) : tab[row + j1];
    var0 = y0.a + f0 * y0.b, var1 = y1.a + f1 * y1.b;
}
// The shared-memory address of p (0 unless the table is staged there).
template <bool STAGED>
__device__ __forceinline__ uint32_t shared_address(const void* p) {
    return STAGED ? static_cast<uint32_t>(__cvta_generic_to_shared(p)) : 0u;
}

// A record of whole 16-byte words (StepRec, NameStep) read from global memory through the read-only data cache: the
// compiler may then issue the load ahead of the kernel's stores and reductions, which a plain load could alias.
template <typename T>
__device__ __forceinline__ T ldg_rec(const T* p) {
    static_assert(sizeof(T) % 16 == 0 && alignof(T) >= 16, "a record of whole 16-byte words");
    T out;
    const int4* src = reinterpret_cast<const int4*>(p);
    int4* dst = reinterpret_cast<int4*>(&out);
#pragma unroll
    for (int k = 0; k < static_cast<int>(sizeof(T) / 16); ++k) dst[k] = __ldg(src + k);
    return out;
}

// A block's copy of the staged blob (whole 16-byte words): every thread's copies are in flight together (cp.async),
// where a loop of loads and stores waits for each few: 64 threads bring 81 KB in about 2 us instead of 10. The copy is complete
// after the caller's next barrier.
__device__ __forceinline__ void stage_blob(unsigned char* sm, const unsigned char* blob, int bytes) {
    const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(sm));
    for (int t = static_cast<int>(threadIdx.x) * 16; t < bytes; t += static_cast<int>(blockDim.x) * 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + static_cast<uint32_t>(t)), "l"(blob + t)
                     : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Per step: -dt / 2, sqrt(dt), dt, and the index of the observation taken at the step's end (negative: none; in an
// autocall minus the number of steps to the next observation).
template <typename R>
struct alignas(16) StepRec {
    R hdt, sdt, dt;
    int obs;
};

// A ring of streamed rows (row_stream.cuh).
struct RowStreamArgs {
    int batches;  // batches of steps a stage
    int pitch;    // intervals from one row to the next, a whole number of 16-byte words
    int chunks;   // 16-byte words a row
    unsigned inv; // 2^32 / chunks, rounded up: c / chunks = c inv >> 32 for the c of a stage
    int off;      // the ring's offset in shared memory (two stages)
};

// Byte offsets inside the staged blob.
struct FusedOffsets {
    int step,  // StepRec a step; Heston QE: the observation of each step alone (an autocall's)
        name_step, root, hes, table2, ln_trig, obs_disc, leg_type, leg_strike, leg_barrier, ln_level;
    int mix_den, low_root;  // local correlation: per step sigma sqrt(max(t0, 1/12)); the aligned low root
    int qe_tables;          // Heston QE in double: Qe64Tables
};

template <typename R>
struct FusedArgs {
    FusedOffsets off;
    const unsigned char* blob;
    int smem_blob;
    int smem_acc;  // the warps' sums, after the blob and the ring
    int n_steps, n_obs, n_out, n_legs, n_x, same;
    R top;  // n_x - 1 - 1e-4, the clamp of the table interpolation
    QeConsts<R> qe;
    R spot0;
    double discount;
    int has_coupon, memory, ki_daily;
    R ln_cb, ln_ki;
    double coupon, put_strike;
    const Pair2<R>* tab;  // the table in global memory (kTabGlobal, kTabStreamed), else unused
    RowStreamArgs rs;     // kTabStreamed
    // local correlation (kernels with MIX): w0 + level, down, up, sign, cos, sin of the mixer (paths.hpp:219-237)
    R mix_base, mix_down, mix_up, mix_sign, mix_cos, mix_sin;
};

}  // namespace ob
