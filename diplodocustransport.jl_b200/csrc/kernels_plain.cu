// Kernels of the plain (single-instance) explicit Euler step, FP64 or FP32.
//
// One step is two launches,
//   gain_stream  - streams the gain blocks G[a][b][c] from HBM through a bulk-copy (TMA)
//                  pipeline in shared memory and contracts each tile against f_b, then each
//                  work unit (a row and a range of b) against f_c, for up to eight space cells
//                  per read of G; writes one FP64 partial per unit and cell.
//   euler_rows   - one warp per state row: banded flux row (ELL, 128-bit loads), emission
//                  row pieces, loss bilinear term, sum of the row's gain partials, then the
//                  Euler update and clamp of SteppingMethods.jl:46-101; each block writes a
//                  record of its rows' CFL diagnostics.
// and, once per sequence of steps (a graph of them, or the steps run outside one),
//   step_diag    - one block per step reduces the step's block records (SteppingMethods.jl:48-94)
//                  and advances the step counter, off the steps' critical path.
// The state is double-buffered (f_in -> f_out) because a row reads other rows' f.
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include <algorithm>

#include "dtb_internal.h"
#include "pdl.cuh"
#include "plain_step.cuh"

namespace dtb {

// ------------------------------------------------------------------ gain_stream
// Ring of the units in flight in a block (records and warp sums). A tile is copied once every
// consumer warp has released the tile kGainStages before it, and a unit has at least one tile: when
// a unit's record is written, or its warp sums are, every warp is past the unit kGainStages + 1
// before it, so that many slots never alias one still read.
constexpr int kRedRing = kGainStages + 1;

// What the consumers need of a work unit: 16 bytes, so that the ring takes no more shared memory
// than it leaves to the longest state vectors (20,800 FP64 states). The loop bounds stay 32 bits
// wide: with 16-bit ones the compiler unrolls the b-rows further, at 3 to 10 % of a step.
struct GainRec {
    unsigned short b_off, c_off;
    int nb, n2p, tile_b;
};
static_assert(sizeof(GainRec) == 16, "GainRec layout");

int gain_stream_smem_bytes(int elem_size, int f_smem_len, int cells) {
    return kGainStages * kGainTileBytes + round_up_int(f_smem_len * cells * (cells == 1 ? elem_size : 8), 16) +
           2 * kGainStages * 8 + kRedRing * 8 + kRedRing * (int)sizeof(GainRec) +
           kRedRing * kGainConsumerWarps * cells * 8 + 8;
}

// One block streams work units through a ring of 16 KB tiles for up to C space cells at once
// (grid y: groups of C cells), so G crosses HBM once per group and not once per cell. Bound: HBM
// with one cell (2 x 1024 states in FP32: 7.1 TB/s); with eight FP64 cells the
// shared-memory reads and the work per 16 KB tile (4.8 TB/s of G on 2 x 256 states). At most 96
// registers: two CTAs of nine warps per SM.
template <typename T, int C, int KV>
__global__ void __launch_bounds__(kGainThreads, 2) gain_stream_kernel(const T* __restrict__ G,
                                                                   const GainUnit* __restrict__ units,
                                                                   int n_units, const T* __restrict__ f,
                                                                   int n_mom, SpOff so, int f_len,
                                                                   double* __restrict__ partial, int* err,
                                                                   const int* __restrict__ cell_list, int n_cells) {
    constexpr int kTileElems = kGainTileBytes / sizeof(T);
    constexpr int kMaxVec = KV * kGainConsumers;

    extern __shared__ __align__(128) unsigned char smem[];
    using S = typename StagedT<T, C>::type;
    S* f_s = reinterpret_cast<S*>(smem + kGainStages * kGainTileBytes);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + kGainStages * kGainTileBytes +
                                                 round_up_int(f_len * C * (int)sizeof(S), 16));
    uint64_t* empty = full + kGainStages;
    uint64_t* unit_bar = empty + kGainStages;
    GainRec* unit_s = reinterpret_cast<GainRec*>(unit_bar + kRedRing);  // by unit slot
    double* red = reinterpret_cast<double*>(unit_s + kRedRing);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(red + kRedRing * kGainConsumerWarps * C);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cell0 = blockIdx.y * C;

    if (tid == 0) {
        for (int s = 0; s < kGainStages; ++s) {
            mbar_init(smem_u32(&full[s]), 1);
            mbar_init(smem_u32(&empty[s]), kGainConsumerWarps);
        }
        for (int s = 0; s < kRedRing; ++s) mbar_init(smem_u32(&unit_bar[s]), kGainConsumerWarps);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();  // barriers initialised; the producer may stream G before f is ready
    const auto bad = [](const GainUnit& U) {
        return U.nb <= 0 || U.tile_b <= 0 || U.n2p <= 0 || U.tile_b * U.n2p > kTileElems ||
               U.n2p / Vec<T>::n > kMaxVec || (unsigned)U.b_off > 65535u || (unsigned)U.c_off > 65535u;
    };

    if (warp == kGainConsumerWarps) {
        // ---------------- producer: one thread issues the bulk copies
        if (lane == 0) {
            uint32_t it = 0;
            int slot = 0;  // the unit's place in the ring
            bool ok = true;
            GainUnit N{};
            if ((int)blockIdx.x < n_units) N = units[blockIdx.x];
            for (int u = blockIdx.x; u < n_units && ok; u += gridDim.x, slot = slot + 1 == kRedRing ? 0 : slot + 1) {
                const GainUnit U = N;
                if (u + (int)gridDim.x < n_units) N = units[u + gridDim.x];  // in flight beside this unit
                if (bad(U)) {
                    atomicOr(err, KERR_BAD_UNIT);
                    *abort_flag = 1;
                    ok = false;
                    break;
                }
                const int nt = (U.nb + U.tile_b - 1) / U.tile_b;
                for (int t = 0; t < nt; ++t, ++it) {
                    const int st = it % kGainStages;
                    const uint32_t ph = (it / kGainStages) & 1u;
                    if (!mbar_wait_bounded(smem_u32(&empty[st]), ph ^ 1u, abort_flag)) {
                        if (!*abort_flag) atomicOr(err, KERR_TIMEOUT_EMPTY);
                        *abort_flag = 1;
                        ok = false;
                        break;
                    }
                    // the record reaches the consumers with the unit's first tile
                    if (t == 0)
                        unit_s[slot] = {(unsigned short)U.b_off, (unsigned short)U.c_off, U.nb, U.n2p, U.tile_b};
                    const int rows = min(U.tile_b, U.nb - t * U.tile_b);
                    const uint32_t bytes = (uint32_t)rows * (uint32_t)U.n2p * (uint32_t)sizeof(T);
                    mbar_arrive_expect_tx(smem_u32(&full[st]), bytes);
                    bulk_g2s(smem_u32(smem + (size_t)st * kGainTileBytes), G + U.g_off + (long long)t * U.tile_b * U.n2p,
                             bytes, smem_u32(&full[st]));
                }
            }
            // Wait for this block's own copies before the block may exit.
            const uint32_t first = it > (uint32_t)kGainStages ? it - kGainStages : 0u;
            volatile int never = 0;
            for (uint32_t k = first; k < it; ++k) {
                if (!mbar_wait_bounded(smem_u32(&full[k % kGainStages]), (k / kGainStages) & 1u, &never))
                    atomicOr(err, KERR_TIMEOUT_DRAIN);
            }
        }
        return;
    }

    // ---------------- consumers: 8 warps
    // f is the previous step's output and the previous step still reads the partials this
    // kernel writes: wait for it (the G tiles already stream in meanwhile)
    pdl_wait();
    if (tid == 0) pdl_trigger();
    stage_f<T, C>(f_s, f, so, f_len, n_mom, cell_list, cell0, n_cells, tid, kGainConsumers);
    asm volatile("bar.sync 1, %0;" ::"n"(kGainConsumers) : "memory");  // the consumer warps only
    uint32_t it = 0;
    int slot = 0;  // the unit's place in the ring, and the parity of its phase there
    uint32_t unit_ph = 0;
    UnitSum<T, C, KV> sum;
    int c_off = -1, n2p = 0;  // the columns in sum's x
    for (int u = blockIdx.x; u < n_units; u += gridDim.x) {
        const GainRec* U = &unit_s[slot];  // valid from the unit's first tile on
        UnitMap m{};
        const S* f1 = f_s;
        sum.begin();
        int left = 1, tile_b = 0, r = 0;  // b-rows left (at least one tile), the thread's next b-row
        for (; left > 0; left -= tile_b, f1 += tile_b, ++it) {
            const int st = it % kGainStages;
            const uint32_t ph = (it / kGainStages) & 1u;
            if (!mbar_wait_bounded(smem_u32(&full[st]), ph, abort_flag)) {
                if (!*abort_flag) atomicOr(err, KERR_TIMEOUT_FULL);
                *abort_flag = 1;
                return;
            }
            if (tile_b == 0) {
                m = unit_map<T, KV>(U->n2p, tid);
                r = m.r0;
                if (sum.kDotRows && (U->c_off != c_off || U->n2p != n2p)) {
                    c_off = U->c_off;
                    n2p = U->n2p;
                    sum.load_x(m, f_s + c_off, f_len);
                }
                f1 += U->b_off;
                left = U->nb;
                tile_b = U->tile_b;
            }
            sum.tile(m, smem + (size_t)st * kGainTileBytes, min(tile_b, left), r, f1, f_len);
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&empty[st]));
        }
        sum.finish(m, f_s + U->c_off, f_len);
        double part[pow2_ceil(C)];
#pragma unroll
        for (int c = 0; c < pow2_ceil(C); ++c) part[c] = c < C ? sum.acc[c < C ? c : 0] : 0.0;
        const double acc = warp_sum_n<pow2_ceil(C)>(part, lane);
        constexpr int kLanes = 32 / pow2_ceil(C);  // lanes per cell of the warp's sums
        if (lane % kLanes == 0 && lane / kLanes < C) red[(slot * kGainConsumerWarps + warp) * C + lane / kLanes] = acc;
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&unit_bar[slot]));
        if (warp == 0) {
            if (!mbar_wait_bounded(smem_u32(&unit_bar[slot]), unit_ph, abort_flag)) {
                if (!*abort_flag) atomicOr(err, KERR_TIMEOUT_FULL);
                *abort_flag = 1;
                return;
            }
            if (lane < C && cell0 + lane < n_cells) {
                double s = 0.0;
#pragma unroll
                for (int w = 0; w < kGainConsumerWarps; ++w) s += red[(slot * kGainConsumerWarps + w) * C + lane];
                const int cell = cell_list ? cell_list[cell0 + lane] : cell0 + lane;
                partial[(size_t)cell * n_units + u] = s;
            }
        }
        if (++slot == kRedRing) {
            slot = 0;
            unit_ph ^= 1u;
        }
    }
}

namespace {

template <typename T>
using GainKernel = void (*)(const T*, const GainUnit*, int, const T*, int, SpOff, int, double*, int*, const int*, int);

// The instance of a pass (gain_pass picks only these): at most 32 FP64 accumulators per thread.
template <typename T, int KV, int C>
GainKernel<T> gain_kernel_upto(int cells) {
    if constexpr (C > 1) {
        if (cells < C) return gain_kernel_upto<T, KV, C - 1>(cells);
    }
    return gain_stream_kernel<T, C, KV>;
}
template <typename T>
GainKernel<T> gain_kernel(const GainPass& p) {
    constexpr int n = Vec<T>::n;
    if (p.kv == 1) return gain_kernel_upto<T, 1, sizeof(T) == 8 ? 2 : 8>(p.cells);
    if (p.kv == 2) return gain_kernel_upto<T, 2, 32 / (2 * n)>(p.cells);
    if constexpr (sizeof(T) == 8)
        return gain_kernel_upto<T, 4, 4>(p.cells);
    else
        return p.kv == 3 ? gain_stream_kernel<T, 1, 3> : gain_stream_kernel<T, 1, 4>;
}

template <typename T>
int pass_blocks_per_sm(const GainPass& p, int f_smem_len) {
    int n = 0;
    const int smem = gain_stream_smem_bytes(sizeof(T), f_smem_len, p.cells);
    const auto k = gain_kernel<T>(p);
    if (smem > kGainSmemLimit || allow_gain_smem(k) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, kGainThreads, smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

}  // namespace

// Cells that share one read of G: as many as fit a thread's accumulators (32 FP64 values, 8 cells
// at most) and the staged states a CTA's shared memory, split evenly over the passes they take
// (the least padding). G is the traffic: eight cells of a 2 x 256-state FP64 grid (268 MB of G)
// take 61 us per step in one pass and 321 us in eight. Four columns per thread spill at the most
// cells: with FP32 a pass takes one cell then (b-rows of 2,056 states, two cells: 86 us per step in
// two passes, 144 in one), with FP64 three, or just four where the threads' last column is nearly
// full (b-rows of 1,032 / 1,600 / 2,000 states: four cells in two passes 41 / 85 / 122 us, in one
// 75 / 87 / 110; eight in three passes 76 / 138 / 194, in two 127 / 167 / 212).
// 16-byte columns per thread: what covers the longest b-row with 256 threads, and with three or more
// FP64 cells at least two, since every cell costs a broadcast read of f1 per b-row and the columns
// share it. One FP32 cell takes four: they also share f1's conversion to FP64, and a tile is one
// round of the block. That pays where G comes from HBM (kFourColsStep, kFourColsOp: 30 steps of
// 2 x 328 and 2 x 352 states 1.48 and 1.73 against 1.52 and 1.83 ms, 8 of 2 x 1024 9.5 against 10.5;
// contractions of 268 to 540 MB 4 to 8 % faster), or on b-rows of 96 columns and more from a G of some size (30 steps of
// 128 + 384 states, 101 MB: 0.60 against 0.67 ms); not from a G that L2 serves (2 x 232 states,
// 100 MB: 0.79 against 0.68 ms; 32 + 480, 31 MB: 0.40 against 0.36), nor on rows of a few columns
// (2048 x 2048 x 16: 83 against 66 us). Rows of 513 to 768 columns take three: 5 % faster than four.
// With FP64 more columns cost more in idle threads than they save (40 steps of 2 x 128: 0.51
// against 0.45 ms).
GainPass gain_pass(int elem_size, int f_smem_len, int max_n2p, int n_cells, double g_bytes, double four_from) {
    GainPass p;
    const int nvr = max_n2p * elem_size / 16, n = 16 / elem_size;
    p.kv = nvr <= kGainConsumers ? 1 : (nvr <= 2 * kGainConsumers ? 2 : 4);
    if (elem_size == 8 && n_cells > 2) p.kv = std::max(p.kv, 2);
    if (elem_size == 4 && n_cells == 1) {
        if ((nvr >= 10 && g_bytes > four_from) || (nvr >= 96 && g_bytes > kFourColsWide)) p.kv = 4;
        if (nvr > 2 * kGainConsumers && nvr <= 3 * kGainConsumers) p.kv = 3;
    }
    int most = std::min(kGainMaxCells, 32 / (p.kv * n));
    if (elem_size == 8 && p.kv == 1) most = std::min(most, 2);
    if (p.kv == 4) most = elem_size == 4 ? 1 : (n_cells == 4 && nvr >= 864 ? 4 : 3);
    while (most > 1 && gain_stream_smem_bytes(elem_size, f_smem_len, most) > kGainSmemLimit) --most;
    const int passes = (n_cells + most - 1) / most;
    p.cells = passes > 0 ? (n_cells + passes - 1) / passes : 1;
    return p;
}

int gain_stream_blocks_per_sm(int elem_size, const GainPass& p, int f_smem_len) {
    return elem_size == 8 ? pass_blocks_per_sm<double>(p, f_smem_len) : pass_blocks_per_sm<float>(p, f_smem_len);
}

template <typename T>
cudaError_t launch_gain_stream(const GainPass& pass, const T* G, const GainUnit* units, int n_units, const T* f,
                               int n_mom, const int* sp_off_host, int n_species, int f_smem_len, double* partial,
                               int n_cells, int grid_x, int* err, cudaStream_t s, const int* cell_list, bool pdl) {
    // n_cells: cells to run (grid y: groups of pass.cells); cell_list maps them to cells, or null
    // for 0..n_cells-1. sp_off_host: [0..n_species] unpadded then [0..n_species] padded offsets
    SpOff so;
    so.n = n_species;
    for (int i = 0; i <= n_species; ++i) {
        so.off[i] = sp_off_host[i];
        so.offp[i] = sp_off_host[n_species + 1 + i];
    }
    // the instance's dynamic shared-memory limit was raised by gain_stream_blocks_per_sm
    const int smem = gain_stream_smem_bytes(sizeof(T), f_smem_len, pass.cells);
    const auto k = gain_kernel<T>(pass);
    dim3 grid(grid_x, (n_cells + pass.cells - 1) / pass.cells);
    // pdl: a step's own sequence (its G is static); a caller's G may be its predecessor's output,
    // which the producer (it starts before the dependency wait) must not read early
    if (pdl)
        return launch_pdl(k, grid, dim3(kGainThreads), (size_t)smem, s, G, units, n_units, f, n_mom, so, f_smem_len,
                          partial, err, cell_list, n_cells);
    k<<<grid, kGainThreads, smem, s>>>(G, units, n_units, f, n_mom, so, f_smem_len, partial, err, cell_list, n_cells);
    return cudaGetLastError();
}

template cudaError_t launch_gain_stream<double>(const GainPass&, const double*, const GainUnit*, int, const double*,
                                                int, const int*, int, int, double*, int, int, int*, cudaStream_t,
                                                const int*, bool);
template cudaError_t launch_gain_stream<float>(const GainPass&, const float*, const GainUnit*, int, const float*, int,
                                               const int*, int, int, double*, int, int, int*, cudaStream_t, const int*,
                                               bool);

// ------------------------------------------------------------------ euler_rows
template <typename T>
__global__ void __launch_bounds__(kRowsWarps * 32) euler_rows_kernel(RowOps<T> ops, const T* __restrict__ f_in,
                                                                     T* __restrict__ f_out, double dt_imm,
                                                                     const double* __restrict__ dt_arr,
                                                                     const unsigned long long* ctr, int kpos,
                                                                     int verbose, double* rec) {
    __shared__ double s_red[kRowsWarps][kStepRecFields];
    // The previous step's state and the step counter (which advances only between step
    // sequences) were final before this grid could launch: as a programmatic dependent it
    // follows this step's gain kernel, which lets it launch only after that kernel's own wait for
    // the kernels before it; without a gain kernel it launches in plain stream order. So the
    // flux, emission and loss products, which read only the state and static operands, run
    // before the wait for this step's gain partials (on SMs beside the gain kernel where it
    // leaves room); everything this grid writes is written after the wait.
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned long long step = *reinterpret_cast<const volatile unsigned long long*>(ctr) + (unsigned)kpos;
    const double dt_scale = dt_arr ? dt_arr[step] : dt_imm;
    const int i = blockIdx.x * kRowsWarps + warp;

    double m_cr = CUDART_INF, m_bin = CUDART_INF, m_emi = CUDART_INF, m_flux = CUDART_INF;
    double s_df = 0.0, s_f = 0.0;
    const int cell = i < ops.n_state ? i / ops.n_mom : 0;
    const int a = i - cell * ops.n_mom;
    int s = 0;
    double flux = 0.0, emi = 0.0, loss = 0.0;
    // binary term of this cell (SteppingMethods.jl:369): outside BinM.Domain it is zero
    const bool bin_here = i < ops.n_state && ops.has_bin && (ops.bin_on == nullptr || ops.bin_on[cell] != 0);
    // The row's unit range, old state and vectors are static or the previous step's: read them
    // before the wait too, so only the gain partials' round trip follows it.
    int u_lo = 0, u_hi = 0;
    int2 cut = make_int2(0, 0);
    T fa = T(0), iap = T(0), injv = T(0), volc = T(0);
    if (i < ops.n_state) {
        while (s + 1 < ops.n_species && a >= ops.sp_off[s + 1]) ++s;
        row_terms(ops, i, cell, a, s, bin_here, lane, [f_in](int k) { return (double)f_in[k]; }, flux, emi, loss);
        if (bin_here) {
            u_lo = ops.unit_ptr[a];
            u_hi = ops.unit_ptr[a + 1];
            cut = ops.cuts[a];
            volc = ops.vol[cell];
        }
        fa = f_in[i];
        iap = ops.invAp[i];
        if (ops.mode == 0) injv = ops.inj[i];
    }
    pdl_wait();  // this step's gain partials (and, in the space pass, the momentum pass) are complete
    if (threadIdx.x == 0) pdl_trigger();
    if (i < ops.n_state) {
        const double* pr = ops.partial + (size_t)cell * ops.n_units;
        const double gain = sum_partials(pr, u_lo, cut, u_hi);
        T dbin;
        const T df = row_df(ops, bin_here, fa, iap, volc, flux, emi, loss, gain, dt_scale, dbin);
        if (lane == 0 && ops.mode == 1) {
            // ForwardSymplecticEuler momentum pass (SteppingMethods.jl:140-160)
            const T fm = fa + df;
            f_out[i] = jl_mul_bool(fm, fm >= (T)ops.thr_mom);
            ops.dfm_out[i] = df;
        }
        if (lane == 0 && ops.mode == 0) {
            f_out[i] = row_update(ops, fa, df, injv, dt_scale);
            // :48-94 diagnostics on the old f
            const double fd = (double)fa;
            m_cr = nan_to_inf((double)df / fd);
            if (verbose == 3) {
                if (ops.has_bin) m_bin = nan_to_inf((double)dbin / fd);
                if (ops.has_emi) m_emi = nan_to_inf((double)(T)emi / fd);
                m_flux = nan_to_inf(-(double)(T)flux / fd);
            }
            s_df = (double)df;
            s_f = fd;
        }
    }
    if (ops.mode == 1) return;  // the space pass writes the step's records
    // this block's record; the step's records are reduced by step_diag_kernel, so no row
    // block waits for the others
    if (lane == 0) {
        s_red[warp][0] = m_cr;
        s_red[warp][1] = m_bin;
        s_red[warp][2] = m_emi;
        s_red[warp][3] = m_flux;
        s_red[warp][4] = s_df;
        s_red[warp][5] = s_f;
    }
    __syncthreads();
    if (threadIdx.x < kStepRecFields) {
        const int k = threadIdx.x;  // one thread per field, the warps in order
        double r = s_red[0][k];
        for (int w = 1; w < kRowsWarps; ++w) r = rec_join(k, r, s_red[w][k]);
        rec[(size_t)blockIdx.x * kStepRecFields + k] = r;
    }
}

int euler_rows_blocks(int n_state) { return (n_state + kRowsWarps - 1) / kRowsWarps; }

// Block k reduces the row-block records of step *ctr + k with a fixed assignment (record b to
// thread b mod 256, in order) and a fixed tree, so a step's record does not depend on block
// completion order or on how the steps were grouped into launches.
__global__ void __launch_bounds__(kRowsWarps * 32) step_diag_kernel(const double* __restrict__ blk_red,
                                                                    int n_blocks, int n_steps,
                                                                    unsigned long long* ctr, StepDiagDev* hist,
                                                                    long long hist_cap, int verbose,
                                                                    int has_bin, int has_emi, int sympl,
                                                                    unsigned* ticket, int n_state) {
    __shared__ double s_fin[kStepRecFields][kRowsWarps * 32];
    pdl_wait();  // the last step's row blocks have written their records
    // a gain kernel that follows may start streaming its (static) blocks; it reads the state and
    // the row kernel after it reads the counter only after this grid has finished
    if (threadIdx.x == 0) pdl_trigger();
    const unsigned long long step0 = *reinterpret_cast<volatile unsigned long long*>(ctr);
    const double* recs = blk_red + (size_t)blockIdx.x * (n_state > 0 ? n_state : n_blocks) * kStepRecFields;
    double r[kStepRecFields] = {CUDART_INF, CUDART_INF, CUDART_INF, CUDART_INF, 0.0, 0.0};
    for (int b = threadIdx.x; b < n_blocks; b += blockDim.x) {
        for (int k = 0; k < kStepRecFields; ++k) {
            double v;
            if (n_state > 0) {  // the record's rows in order, as euler_rows joins them
                const bool in = k == 0 || (k == 1 ? has_bin != 0 : k == 2 ? has_emi != 0 : true);
                if (k >= 1 && k <= 3 && (verbose != 3 || sympl)) continue;
                const auto field = [&](int i) {
                    const double fd = __ldcg(recs + 5 * (size_t)n_state + i);
                    if (k >= 4) return k == 5 ? fd : (sympl ? 0.0 : __ldcg(recs + i));
                    return in ? nan_to_inf(__ldcg(recs + (size_t)k * n_state + i) / fd) : CUDART_INF;
                };
                v = field(b * kRowsWarps);
                for (int i = b * kRowsWarps + 1; i < min(n_state, (b + 1) * kRowsWarps); ++i) v = rec_join(k, v, field(i));
            } else {
                v = __ldcg(recs + (size_t)b * kStepRecFields + k);
            }
            r[k] = rec_join(k, r[k], v);
        }
    }
    for (int k = 0; k < kStepRecFields; ++k) s_fin[k][threadIdx.x] = r[k];
    __syncthreads();
    for (int o = kRowsWarps * 16; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            for (int k = 0; k < 4; ++k) s_fin[k][threadIdx.x] = jl_min(s_fin[k][threadIdx.x], s_fin[k][threadIdx.x + o]);
            s_fin[4][threadIdx.x] += s_fin[4][threadIdx.x + o];
            s_fin[5][threadIdx.x] += s_fin[5][threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        for (int k = 0; k < kStepRecFields; ++k) r[k] = s_fin[k][0];
        StepDiagDev d;
        const bool on = (verbose == 1 || verbose == 2 || verbose == 3) && r[5] != 0.0;
        d.cr[0] = on ? -r[0] : 0.0;
        d.cr[1] = (on && verbose == 3 && has_bin && !sympl) ? -r[1] : 0.0;
        d.cr[2] = (on && verbose == 3 && has_emi && !sympl) ? -r[2] : 0.0;
        d.cr[3] = (on && verbose == 3 && !sympl) ? -r[3] : 0.0;
        d.sum_df = r[4];
        d.sum_f = r[5];
        // the symplectic method has no finite check (SteppingMethods.jl:120-243)
        d.finite = (sympl || isfinite(r[4])) ? 1 : 0;
        d.pad = 0;
        hist[(step0 + blockIdx.x) % (unsigned long long)hist_cap] = d;
        // every block has read the counter before it takes its ticket; the last one advances it
        __threadfence();
        const unsigned t = atomicAdd(ticket, 1u);
        if (t == gridDim.x - 1) {
            *ticket = 0u;
            *reinterpret_cast<volatile unsigned long long*>(ctr) = step0 + (unsigned long long)n_steps;
        }
    }
}

cudaError_t launch_step_diag(const double* blk_red, int n_blocks, int n_steps, unsigned long long* ctr,
                             StepDiagDev* hist, long long hist_cap, int verbose, int has_bin, int has_emi, int sympl,
                             unsigned* ticket, int n_state, cudaStream_t s) {
    return launch_pdl(step_diag_kernel, dim3(n_steps), dim3(kRowsWarps * 32), 0, s, blk_red, n_blocks, n_steps, ctr,
                      hist, hist_cap, verbose, has_bin, has_emi, sympl, ticket, n_state);
}

template <typename T>
cudaError_t launch_euler_rows(const RowOps<T>& ops, const T* f_in, T* f_out, double dt_imm, const double* dt_arr,
                              const unsigned long long* ctr, int kpos, int verbose, double* rec, bool pdl,
                              cudaStream_t s) {
    const int grid = euler_rows_blocks(ops.n_state);
    if (pdl)
        return launch_pdl(euler_rows_kernel<T>, grid, dim3(kRowsWarps * 32), 0, s, ops, f_in, f_out, dt_imm, dt_arr,
                          ctr, kpos, verbose, rec);
    euler_rows_kernel<T><<<grid, kRowsWarps * 32, 0, s>>>(ops, f_in, f_out, dt_imm, dt_arr, ctr, kpos, verbose, rec);
    return cudaGetLastError();
}

template cudaError_t launch_euler_rows<double>(const RowOps<double>&, const double*, double*, double, const double*,
                                               const unsigned long long*, int, int, double*, bool, cudaStream_t);
template cudaError_t launch_euler_rows<float>(const RowOps<float>&, const float*, float*, double, const double*,
                                              const unsigned long long*, int, int, double*, bool, cudaStream_t);

// ------------------------------------------------------------------ sympl_space
// ForwardSymplecticEuler space pass (SteppingMethods.jl:165-237): one warp per row,
// df_Space = -(X f_Momentum) invAp dt/dt0, f_Space = clamp(f_Momentum + df_Space, 1f-20), then
// f = f_Space + inj dt/dt0 clamped with the sign factor of :235 and the Inf fix of :237.
// Each block writes a record of its rows' (df_Space + df_Momentum) ./ f_old minimum and f_old
// sum in euler_rows' layout; step_diag reduces them to Cr = -min(...) (:217-218).
template <typename T>
__global__ void __launch_bounds__(kRowsWarps * 32) sympl_space_kernel(RowOps<T> ops, const T* __restrict__ f_old,
                                                                      const T* __restrict__ fm,
                                                                      const T* __restrict__ dfm, T* __restrict__ f_out,
                                                                      double dt_imm, const double* __restrict__ dt_arr,
                                                                      const unsigned long long* ctr, int kpos,
                                                                      double* rec) {
    __shared__ double s_red[kRowsWarps][2];
    pdl_wait();  // this step's inputs (gain partials, momentum pass)
    if (threadIdx.x == 0) pdl_trigger();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned long long step = *reinterpret_cast<const volatile unsigned long long*>(ctr) + (unsigned)kpos;
    const double dt_scale = dt_arr ? dt_arr[step] : dt_imm;
    const int i = blockIdx.x * kRowsWarps + warp;
    double m_cr = CUDART_INF, s_f = 0.0;
    if (i < ops.n_state) {
        double xf = 0.0;
        for (int k = lane; k < ops.x_ell_w; k += 32) {
            const int c = ops.x_ell_col[(size_t)i * ops.x_ell_w + k];
            if (c >= 0) xf = fma((double)ops.x_ell_val[(size_t)i * ops.x_ell_w + k], (double)fm[c], xf);
        }
        xf = warp_sum(xf);
        if (lane == 0) {
            T dsp;
            f_out[i] = row_space_update(ops, fm[i], xf, ops.invAp[i], ops.inj[i], dt_scale, dsp);
            const double fo = (double)f_old[i];
            m_cr = nan_to_inf((double)(dsp + dfm[i]) / fo);
            s_f = fo;
        }
    }
    if (lane == 0) {
        s_red[warp][0] = m_cr;
        s_red[warp][1] = s_f;
    }
    __syncthreads();
    if (threadIdx.x < kStepRecFields) {
        // fields 0 (minimum) and 5 (sum) over the warps in order; no per-term Crs, no df sum
        const int k = threadIdx.x;
        double r = k == 0 ? s_red[0][0] : (k == 5 ? s_red[0][1] : (k == 4 ? 0.0 : CUDART_INF));
        if (k == 0)
            for (int w = 1; w < kRowsWarps; ++w) r = jl_min(r, s_red[w][0]);
        if (k == 5)
            for (int w = 1; w < kRowsWarps; ++w) r += s_red[w][1];
        rec[(size_t)blockIdx.x * kStepRecFields + k] = r;
    }
}

template <typename T>
cudaError_t launch_sympl_space(const RowOps<T>& ops, const T* f_old, const T* fm, const T* dfm, T* f_out,
                               double dt_imm, const double* dt_arr, const unsigned long long* ctr, int kpos,
                               double* rec, cudaStream_t s) {
    const int grid = euler_rows_blocks(ops.n_state);
    return launch_pdl(sympl_space_kernel<T>, grid, dim3(kRowsWarps * 32), 0, s, ops, f_old, fm, dfm, f_out, dt_imm,
                      dt_arr, ctr, kpos, rec);
}
template cudaError_t launch_sympl_space<double>(const RowOps<double>&, const double*, const double*, const double*,
                                                double*, double, const double*, const unsigned long long*, int,
                                                double*, cudaStream_t);
template cudaError_t launch_sympl_space<float>(const RowOps<float>&, const float*, const float*, const float*, float*,
                                               double, const double*, const unsigned long long*, int, double*,
                                               cudaStream_t);

// ------------------------------------------------------------------ bounded-wait self-test
// One block waits on an mbarrier phase that nothing completes, with a limit of limit_ns, and
// reports the timeout through err: the same give-up path every pipeline wait in this library
// takes, exercised without a fault.
__global__ void bounded_wait_selftest_kernel(unsigned long long limit_ns, int* err) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&bar), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned long long t0 = globaltimer();
        bool done = false;
        while (!done) {
            done = mbar_try_wait(smem_u32(&bar), 0u);
            if (!done && globaltimer() - t0 > limit_ns) break;
        }
        if (!done) atomicOr(err, KERR_TIMEOUT_FULL);
        mbar_arrive(smem_u32(&bar));  // complete the phase so the barrier is left consistent
    }
}

cudaError_t launch_bounded_wait_selftest(unsigned long long limit_ns, int* err, cudaStream_t s) {
    bounded_wait_selftest_kernel<<<1, 32, 0, s>>>(limit_ns, err);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ helpers
template <typename Tin, typename Tout>
__global__ void pad_rows_kernel(const Tin* __restrict__ src, long long rows, int n, Tout* __restrict__ dst, int np) {
    const long long total = rows * (long long)np;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < total;
         k += (long long)gridDim.x * blockDim.x) {
        const long long r = k / np;
        const int c = (int)(k - r * np);
        dst[k] = c < n ? (Tout)src[r * n + c] : Tout(0);
    }
}

template <typename Tin, typename Tout>
cudaError_t launch_pad_rows(const Tin* src, long long rows, int n, Tout* dst, int np, cudaStream_t s) {
    pad_rows_kernel<Tin, Tout><<<148 * 8, 256, 0, s>>>(src, rows, n, dst, np);
    return cudaGetLastError();
}
template cudaError_t launch_pad_rows<double, double>(const double*, long long, int, double*, int, cudaStream_t);
template cudaError_t launch_pad_rows<float, float>(const float*, long long, int, float*, int, cudaStream_t);
template cudaError_t launch_pad_rows<double, float>(const double*, long long, int, float*, int, cudaStream_t);
template cudaError_t launch_pad_rows<float, double>(const float*, long long, int, double*, int, cudaStream_t);

// Per (cell, species) FP64 number and energy sums; out = [n_space][n_species][2].
template <typename T>
__global__ void moments_kernel(const T* __restrict__ f, int n_mom, const int* __restrict__ sp_off,
                               const double* __restrict__ w, double* __restrict__ out, int n_species) {
    __shared__ double s_n[256], s_e[256];
    const int s = blockIdx.x, cell = blockIdx.y;
    const int lo = sp_off[s], hi = sp_off[s + 1];
    double a = 0.0, e = 0.0;
    for (int k = lo + threadIdx.x; k < hi; k += blockDim.x) {
        const double v = (double)f[(size_t)cell * n_mom + k];
        a += v;
        e += v * w[k];
    }
    s_n[threadIdx.x] = a;
    s_e[threadIdx.x] = e;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            s_n[threadIdx.x] += s_n[threadIdx.x + o];
            s_e[threadIdx.x] += s_e[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        out[((size_t)cell * n_species + s) * 2 + 0] = s_n[0];
        out[((size_t)cell * n_species + s) * 2 + 1] = s_e[0];
    }
}

cudaError_t launch_moments_f64(const double* f, int n_mom, int n_space, const int* sp_off, int n_species,
                               const double* w, double* out, cudaStream_t s) {
    moments_kernel<double><<<dim3(n_species, n_space), 256, 0, s>>>(f, n_mom, sp_off, w, out, n_species);
    return cudaGetLastError();
}
cudaError_t launch_moments_f32(const float* f, int n_mom, int n_space, const int* sp_off, int n_species,
                               const double* w, double* out, cudaStream_t s) {
    moments_kernel<float><<<dim3(n_species, n_space), 256, 0, s>>>(f, n_mom, sp_off, w, out, n_species);
    return cudaGetLastError();
}

}  // namespace dtb
