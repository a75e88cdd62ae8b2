// Device pieces of the plain Euler step shared by the streaming kernels (kernels_plain.cu) and the
// resident one (kernels_resident.cu): barriers and bulk copies, a work unit's contraction and a
// row's terms and update. Both run them on the same work table, so their steps agree bit for bit.
#pragma once

#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "dtb_internal.h"

namespace dtb {

// ------------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ unsigned long long globaltimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void mbar_init(uint32_t bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Waits for the phase with the given parity; gives up after kWaitLimitNs or when another
// role of the block raised the abort flag.
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = globaltimer();
    while (true) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
        if (globaltimer() - t0 > kWaitLimitNs) return false;
    }
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
        "l"(src), "r"(bytes), "r"(bar)
        : "memory");
}
template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Julia's min on Float64 with -0.0 ordered below +0.0 (NaN is mapped to Inf before).
__device__ __forceinline__ double jl_min(double a, double b) {
    if (a < b) return a;
    if (b < a) return b;
    return signbit(a) ? a : b;
}
__device__ __forceinline__ double nan_to_inf(double x) { return isnan(x) ? CUDART_INF : x; }

// Julia `x * b::Bool` = ifelse(b, x, copysign(0, x)).
template <typename T>
__device__ __forceinline__ T jl_mul_bool(T x, bool b) {
    return b ? x : copysign(T(0), x);
}

// ------------------------------------------------------------------ one work unit of the gain
struct SpOff {
    int n;
    int off[DTB_MAX_SPECIES + 1];   // unpadded
    int offp[DTB_MAX_SPECIES + 1];  // padded (multiples of 8)
};

// 16 bytes of G as FP64 values.
template <typename T>
struct Vec;
template <>
struct Vec<float> {
    using type = float4;
    static constexpr int n = 4;
    __device__ __forceinline__ static void unpack(const float4& g, double (&v)[4]) {
        v[0] = g.x;
        v[1] = g.y;
        v[2] = g.z;
        v[3] = g.w;
    }
};
template <>
struct Vec<double> {
    using type = double2;
    static constexpr int n = 2;
    __device__ __forceinline__ static void unpack(const double2& g, double (&v)[2]) {
        v[0] = g.x;
        v[1] = g.y;
    }
};

constexpr int kGainThreads = (kGainConsumerWarps + 1) * 32;
constexpr int kGainConsumers = kGainConsumerWarps * 32;

__host__ __device__ constexpr int round_up_int(int x, int m) { return (x + m - 1) / m * m; }
__host__ __device__ constexpr int pow2_ceil(int x) { return x <= 1 ? 1 : 2 * pow2_ceil((x + 1) / 2); }

// Staged states: in the state type for one cell, FP64 for several (one conversion per state and
// block, not one per b-row).
template <typename T, int C>
struct StagedT {
    using type = double;
};
template <typename T>
struct StagedT<T, 1> {
    using type = T;
};

// Sums of N values over the warp's 32 lanes: halving exchanges while several values are left,
// then a butterfly. Lane l of the result holds value l >> (5 - log2 N). Every value is summed by
// the same tree (lane distances 16, 8, 4, 2, 1), so its bits do not depend on N.
template <int N>
__device__ __forceinline__ double warp_sum_n(double (&v)[N], int lane) {
    int o = 16;
#pragma unroll
    for (int n = N; n > 1; n /= 2, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < N / 2; ++i) {
            if (i < n / 2) {
                const double send = up ? v[i] : v[i + n / 2];
                const double keep = up ? v[i + n / 2] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
        }
    }
#pragma unroll
    for (; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    return v[0];
}

// Thread `tid`'s share of one work unit: the 16-byte columns cv, cv + w, .. (KV of them, w threads
// to a b-row) of the unit's b-rows r0, r0 + dr, ..
struct UnitMap {
    int nvr, w, dr, r0, cv;
    bool on;
};
template <typename T, int KV>
__device__ __forceinline__ UnitMap unit_map(int n2p, int tid) {
    UnitMap m;
    m.nvr = n2p / Vec<T>::n;
    m.w = (m.nvr + KV - 1) / KV;
    m.dr = kGainConsumers / m.w;
    m.r0 = tid / m.w;
    m.cv = tid - m.r0 * m.w;
    m.on = m.r0 < m.dr;
    return m;
}

// A thread's contraction of a work unit, FP64 throughout (the unit is read once for all C cells).
// With three or four columns per thread (few cells) the thread keeps its columns' f2 in x and forms
//   acc += f1[b] (g . x) per b-row,
// so a unit costs no f2 reads of its own while the next one has the same columns; with fewer
// columns (many cells) it accumulates y += f1[b] g per column and dots with f2 once per unit, which
// holds one value per column and cell instead of one plus one per cell.
template <typename T, int C, int KV>
struct UnitSum {
    static constexpr bool kDotRows = KV >= 3;
    using V = Vec<T>;
    using S = typename StagedT<T, C>::type;
    using vec_t = typename V::type;
    double v[KV][C][V::n];  // x or y
    double acc[C];

    // f2: the unit's input-2 states (cell c's are c * f_len further)
    __device__ __forceinline__ void load_x(const UnitMap& m, const S* f2, int f_len) {
#pragma unroll
        for (int k = 0; k < KV; ++k) {
            const bool in = m.on && (k == 0 || m.cv + k * m.w < m.nvr);
            const S* p = f2 + (m.cv + k * m.w) * V::n;
#pragma unroll
            for (int c = 0; c < C; ++c)
#pragma unroll
                for (int e = 0; e < V::n; ++e) v[k][c][e] = in ? (double)p[c * f_len + e] : 0.0;
        }
    }
    __device__ __forceinline__ void begin() {
#pragma unroll
        for (int c = 0; c < C; ++c) acc[c] = 0.0;
        if constexpr (!kDotRows) {
#pragma unroll
            for (int k = 0; k < KV; ++k)
#pragma unroll
                for (int c = 0; c < C; ++c)
#pragma unroll
                    for (int e = 0; e < V::n; ++e) v[k][c][e] = 0.0;
        }
    }
    // The thread's b-rows among the `rows` of `tile`, in order; r: its next b-row, counted from the
    // tile's first, on return from the next tile's.
    __device__ __forceinline__ void tile(const UnitMap& m, const unsigned char* tile, int rows, int& r, const S* f1,
                                         int f_len) {
        if (!m.on) return;
        const vec_t* tv = reinterpret_cast<const vec_t*>(tile) + r * m.nvr + m.cv;
        constexpr int kUnroll = KV * C * V::n <= 8 ? 2 : 1;
#pragma unroll kUnroll
        for (; r < rows; r += m.dr, tv += m.dr * m.nvr) {
            double g[KV][V::n];
#pragma unroll
            for (int k = 0; k < KV; ++k) {
                if constexpr (kDotRows) {  // columns past the row's end take no part
#pragma unroll
                    for (int e = 0; e < V::n; ++e) g[k][e] = 0.0;
                    if (k == 0 || m.cv + k * m.w < m.nvr) V::unpack(tv[k * m.w], g[k]);
                } else {  // such a column repeats the last one; its sum is not used
                    V::unpack(tv[k == 0 ? 0 : min(k * m.w, m.nvr - 1 - m.cv)], g[k]);
                }
            }
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const double x1 = (double)f1[c * f_len + r];
                if constexpr (kDotRows) {
                    double d[2] = {0.0, 0.0};  // two chains: columns 0, 1 and the others
#pragma unroll
                    for (int k = 0; k < KV; ++k)
#pragma unroll
                        for (int e = 0; e < V::n; ++e) d[k / 2] = fma(g[k][e], v[k][c][e], d[k / 2]);
                    acc[c] = fma(x1, d[0] + d[1], acc[c]);
                } else {
#pragma unroll
                    for (int k = 0; k < KV; ++k)
#pragma unroll
                        for (int e = 0; e < V::n; ++e) v[k][c][e] = fma(x1, g[k][e], v[k][c][e]);
                }
            }
        }
        r -= rows;
    }
    // acc complete (f2 as for load_x)
    __device__ __forceinline__ void finish(const UnitMap& m, const S* f2, int f_len) {
        if constexpr (!kDotRows) {
            if (!m.on) return;
#pragma unroll
            for (int k = 0; k < KV; ++k) {
                if (k == 0 || m.cv + k * m.w < m.nvr) {
                    const S* p = f2 + (m.cv + k * m.w) * V::n;
#pragma unroll
                    for (int c = 0; c < C; ++c)
#pragma unroll
                        for (int e = 0; e < V::n; ++e) acc[c] = fma((double)p[c * f_len + e], v[k][c][e], acc[c]);
                }
            }
        }
    }
};

// The cells of a pass, padded per species ([cell][state]: the lanes of a warp read consecutive
// states of one cell); zeros in the padding and for cells past the last.
template <typename T, int C>
__device__ __forceinline__ void stage_f(typename StagedT<T, C>::type* f_s, const T* __restrict__ f, const SpOff& so,
                                        int f_len, int n_mom, const int* cell_list, int cell0, int n_cells, int tid,
                                        int n_threads) {
    for (int i = tid; i < f_len; i += n_threads) {
        int s = 0;
        while (s + 1 < so.n && i >= so.offp[s + 1]) ++s;
        const int j = i - so.offp[s];
        const bool in = j < so.off[s + 1] - so.off[s];
#pragma unroll
        for (int c = 0; c < C; ++c) {
            T v = T(0);
            if (in && cell0 + c < n_cells) {
                const int cell = cell_list ? cell_list[cell0 + c] : cell0 + c;
                v = f[(size_t)cell * n_mom + so.off[s] + j];
            }
            f_s[c * f_len + i] = v;
        }
    }
}

// ------------------------------------------------------------------ one row of the step
// The pieces of a row's step, shared by the kernels that run it so that they agree bit for bit.

// Flux, emission and loss sums of state row i (row a of species s in its cell) over one warp.
// f_at(k): the step's input state k in FP64.
template <typename T, typename FAt>
__device__ __forceinline__ void row_terms(const RowOps<T>& ops, int i, int cell, int a, int s, bool bin_here, int lane,
                                          const FAt& f_at, double& flux, double& emi, double& loss) {
    flux = emi = loss = 0.0;
    // (a) banded flux row: ELL slots of width ell_w, 128-bit loads of 4 slots per lane
    {
        const T* vrow = ops.ell_val + (size_t)i * ops.ell_w;
        const int* crow = ops.ell_col + (size_t)i * ops.ell_w;
#pragma unroll 1
        for (int k = lane * 4; k < ops.ell_w; k += 128) {
            const int4 c4 = __ldg(reinterpret_cast<const int4*>(crow + k));
            T v0, v1, v2, v3;
            if constexpr (sizeof(T) == 4) {
                const float4 v4 = __ldg(reinterpret_cast<const float4*>(vrow + k));
                v0 = v4.x; v1 = v4.y; v2 = v4.z; v3 = v4.w;
            } else {
                const double2 va = __ldg(reinterpret_cast<const double2*>(vrow + k));
                const double2 vb = __ldg(reinterpret_cast<const double2*>(vrow + k + 2));
                v0 = va.x; v1 = va.y; v2 = vb.x; v3 = vb.y;
            }
            // padding slots carry column -1: only stored entries take part, like a CSC product
            if (c4.x >= 0) flux = fma((double)v0, f_at(c4.x), flux);
            if (c4.y >= 0) flux = fma((double)v1, f_at(c4.y), flux);
            if (c4.z >= 0) flux = fma((double)v2, f_at(c4.z), flux);
            if (c4.w >= 0) flux = fma((double)v3, f_at(c4.w), flux);
        }
    }
    // (c) emission row pieces
    if (ops.has_emi) {
#pragma unroll 1
        for (int p = __ldg(ops.emi_rptr + i), e = __ldg(ops.emi_rptr + i + 1); p < e; ++p) {
            const int pc = __ldg(ops.emi_piece + p);
            const T* row = ops.emi_data + __ldg(ops.emi_data_off + pc) +
                           (size_t)(i - __ldg(ops.emi_row0 + pc)) * __ldg(ops.emi_ld + pc);
            const int c0 = __ldg(ops.emi_col0 + pc), nc = __ldg(ops.emi_ncols + pc);
            for (int c = lane; c < nc; c += 32) emi = fma((double)__ldg(row + c), f_at(c0 + c), emi);
        }
    }
    // loss bilinear term
    if (bin_here) {
        const int la = a - ops.sp_off[s];
#pragma unroll 1
        for (int b = ops.loss_ptr[s]; b < ops.loss_ptr[s + 1]; ++b) {
            const T* row = ops.loss_data + __ldg(ops.loss_data_off + b) + (size_t)la * __ldg(ops.loss_ld + b);
            const int c0 = cell * ops.n_mom + __ldg(ops.loss_col_off + b), nc = __ldg(ops.loss_ncols + b);
            for (int c = lane; c < nc; c += 32) loss = fma((double)__ldg(row + c), f_at(c0 + c), loss);
        }
    }
    double v[4] = {flux, emi, loss, 0.0};
    const double sum = warp_sum_n<4>(v, lane);  // lanes 8 j .. 8 j + 7 hold sum j
    flux = __shfl_sync(0xffffffffu, sum, 0);
    emi = __shfl_sync(0xffffffffu, sum, 8);
    loss = __shfl_sync(0xffffffffu, sum, 16);
}

// A row's gain: the sums of its (at most three) segments of units, in order (RowOps::cuts).
__device__ __forceinline__ double row_gain(double a, double b, double c) { return a + b + c; }

// The gain from partials lo .. hi - 1, in unit order within the segments, eight loads in flight
// (from L2: other blocks wrote them).
__device__ __forceinline__ double sum_partials(const double* pr, int lo, int2 cut, int hi) {
    double a = 0.0, b = 0.0, c = 0.0;
    for (int u = lo; u < hi; u += 8) {
        double v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = u + k < hi ? __ldcg(pr + u + k) : 0.0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (u + k < min(cut.x, hi)) a += v[k];
            else if (u + k < min(cut.y, hi)) b += v[k];
            else if (u + k < hi) c += v[k];
        }
    }
    return row_gain(a, b, c);
}

// df of a row before and after its scaling (SteppingMethods.jl:31-46).
template <typename T>
__device__ __forceinline__ T row_df(const RowOps<T>& ops, bool bin_here, T fa, T iap, T volc, double flux, double emi,
                                    double loss, double gain, double dt_scale, T& dbin) {
    dbin = bin_here ? (T)((double)volc * fma(-(double)fa, loss, gain)) : T(0);
    T df = -(T)flux;
    if (ops.has_emi) df = df + (T)emi;
    if (ops.has_bin) df = df + dbin;
    return (T)((double)df * ((double)iap * dt_scale));
}
// :97-101, arithmetic in Float64 like Julia's promotion, one rounding at the store
template <typename T>
__device__ __forceinline__ T row_update(const RowOps<T>& ops, T fa, T df, T injv, double dt_scale) {
    T fn = (T)((double)fa + fma((double)injv, dt_scale, (double)df));
    fn = jl_mul_bool(fn, fn >= (T)ops.thr);
    return jl_mul_bool(fn, fn != (T)CUDART_INF);
}
// The row's space update (SteppingMethods.jl:165-237): f_Space clamped at 1f-20, then the
// injection, the clamp with the sign factor of :235 and the Inf fix of :237.
template <typename T>
__device__ __forceinline__ T row_space_update(const RowOps<T>& ops, T fm, double xf, T iap, T injv, double dt_scale,
                                              T& dsp) {
    dsp = (T)((double)(-(T)xf * iap) * dt_scale);
    T fs = fm + dsp;
    fs = jl_mul_bool(fs, fs >= (T)ops.thr_space);
    T v = (T)fma((double)injv, dt_scale, (double)fs);
    const T sg = isnan(v) ? v : (v > T(0) ? T(1) : (v < T(0) ? T(-1) : v));
    v = jl_mul_bool(v, v >= (T)ops.thr_space) * sg;
    return jl_mul_bool(v, v != (T)CUDART_INF);
}
// Field k of a block record from its rows in order: fields 0-3 are minima, 4-5 sums.
__device__ __forceinline__ double rec_join(int k, double r, double v) { return k < 4 ? jl_min(r, v) : r + v; }

}  // namespace dtb
