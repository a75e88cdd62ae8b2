// Many plain Euler steps in one launch, with the gain blocks held in shared memory.
//
// A grid whose gain blocks fit the SMs' shared memory (about 33 MB: 2 x 128 states in FP64) is not
// bound by reading them but by what a step of two launches costs around that: G from L2 again, a
// round trip per tile of the streaming ring, two launch boundaries. Here one block per SM loads its
// work units once per launch and keeps them; the block that holds a row's first unit owns the row.
// A step is then
//   1. the units' contractions from shared memory, while a few warps form the owned rows' flux,
//      emission and loss,
//   2. the owned rows' update, with the sums of units in other blocks (a row spans at most three),
//      and
//   3. a gather of the whole new state by every block.
// What a block publishes (a segment of a row's units, a row's new value) is a 16-byte word of the
// value and the step's number, and is valid when it carries that number. So the exchange is its own
// synchronisation: no grid barrier (2,400 clocks on 148 blocks), and no acquire, which would drop
// the L1's copies of the static operands in every step. Publishing the new values, rather than all
// sums for every block to update every row, keeps the gather small: a few KB that 148 blocks read at
// once is what bounds it (about 40 sectors per clock from one hot region of L2).
// The words are double-buffered by step: a block publishes step k + 2 only after it has gathered
// every row of step k + 1, and whatever a row of step k + 1 needed was published after its block's
// own gather of step k.
// The work table, the sums' order and the rows' arithmetic are those of gain_stream, euler_rows and
// sympl_space, so states and step records agree bit for bit with steps run one by one.
//
// The launch is cooperative (the blocks wait on one another), every wait is bounded. Per step of long
// runs, against the two launches: 2 x 128 FP64 states 5.1 against 9.2 us; five FP32 cells of 140 + 126
// states, symplectic, 11.6 against 15.3; two cells of a sparse 2 x 84-state FP64 grid, 5.9 against 8.2.
// A step of the first takes about 9,900 clocks: 4,700 for the units (shared memory and a chain of
// latencies per unit, 16 warps), 2,500 for the sums and rows, the rest for words on their way. Three
// groups of unit warps at 72 registers (spills), rows handed out dynamically and one task per warp in
// the update were slower.
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include <algorithm>

#include "dtb_internal.h"
#include "plain_step.cuh"

namespace dtb {

namespace {

// kResGroups groups of kGainConsumers threads take one work unit at a time each
constexpr int kResUnitWarps = kResGroups * kGainConsumerWarps;
constexpr int kResRowWarps = 4;  // warps for the owned rows' flux, emission and loss
constexpr int kResWarps = kResUnitWarps + kResRowWarps;
constexpr int kResThreads = kResWarps * 32;  // 640: 96 registers
constexpr int kResStates = 3;  // states per thread in the update (or 1)

// One published sum: read and written as one 16-byte word, so value and step number belong together.
struct ResWord {
    double v;
    unsigned long long step;
};
__device__ __forceinline__ ResWord load_word(const ResWord* p) {
    unsigned long long lo, hi;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(lo), "=l"(hi)
                 : "l"(p)
                 : "memory");
    return {__longlong_as_double((long long)lo), hi};
}
__device__ __forceinline__ void store_word(ResWord* p, double v, unsigned long long step) {
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
                 "l"((unsigned long long)__double_as_longlong(v)), "l"(step)
                 : "memory");
}
// Waits until the word carries `step`; false when the wait gave up.
__device__ __forceinline__ bool wait_word(const ResWord* p, unsigned long long step, double& v) {
    ResWord w = load_word(p);
    if (w.step != step) {
        const unsigned long long t0 = globaltimer();
#pragma unroll 1
        for (int tries = 1; (w = load_word(p)).step != step; ++tries)  // the clock is slow to read
            if (tries % 64 == 0 && globaltimer() - t0 > kWaitLimitNs) return false;
    }
    v = w.v;
    return true;
}

// A block's copy of a work record: the unit's place in shared memory, its shape and its row, and
// the thread map of its b-rows (see UnitMap; r0 = tid / w as tid * inv >> 16, exact for 256 threads).
struct __align__(16) ResUnit {
    int soff, inv;
    unsigned short b_off, c_off, nb, nvr, w, dr, row, slot;
    int pad[2];
};
static_assert(sizeof(ResUnit) == 32, "ResUnit layout");

struct ResLayout {
    int f, fu, red, rest, unit, bar, bytes;  // byte offsets in shared memory; the units' data are at 0
};
// g: bytes of the units, cells: staged cells (whole passes), pad: species sizes are not all
// multiples of 8, so the rows' terms read an unpadded copy of the state.
__host__ __device__ inline ResLayout res_layout(int g, int esz_staged, int f_len, int cells, int n_space, int n_state,
                                                bool pad, int max_local, int max_own) {
    ResLayout L;
    L.f = round_up_int(g, 16);
    L.fu = L.f + round_up_int(f_len * cells * esz_staged, 16);
    L.red = L.fu + (pad ? round_up_int(n_state * esz_staged, 16) : 0);
    L.rest = L.red + max_local * kGainConsumerWarps * n_space * 8;
    L.unit = round_up_int(L.rest + max_own * n_space * 4 * 8, 16);
    L.bar = L.unit + max_local * (int)sizeof(ResUnit);
    L.bytes = L.bar + 16;
    return L;
}

template <typename T, int C, int KV, bool SY, int NS>
__global__ void __launch_bounds__(kResThreads, 1)
    resident_kernel(RowOps<T> ops, ResidentArgs r, SpOff so, const T* __restrict__ f_in, T* __restrict__ f_out,
                    const double* __restrict__ dt_arr, const unsigned long long* ctr, int n_steps, int verbose) {
    using S = typename StagedT<T, C>::type;
    extern __shared__ __align__(128) unsigned char smem[];
    const int n_space = ops.n_space, n_state = ops.n_state, n_mom = ops.n_mom;
    const int staged = (n_space + C - 1) / C * C;
    const ResLayout L = res_layout(r.g_bytes, sizeof(S), r.f_len, staged, n_space, n_state, r.pad != 0, r.max_local,
                                  r.max_own);
    S* f_s = reinterpret_cast<S*>(smem + L.f);
    S* fu = r.pad ? reinterpret_cast<S*>(smem + L.fu) : f_s;  // the state in its own order
    double* red = reinterpret_cast<double*>(smem + L.red);    // per unit, warp and cell
    double* rest = reinterpret_cast<double*>(smem + L.rest);  // per owned row and cell: flux, emission, loss, old f
    ResUnit* unit = reinterpret_cast<ResUnit*>(smem + L.unit);
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + L.bar);
    volatile int* ok = reinterpret_cast<volatile int*>(smem + L.bar + 8);  // 0: a wait gave up
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int grid = gridDim.x, blk = blockIdx.x;
    const int u0 = r.first[blk], n_local = r.first[blk + 1] - u0;
    const int own0 = r.own[blk], n_own = r.own[blk + 1] - own0;
    // thread of the rows' updates: the row warps first (they wait for the units), and neighbouring
    // rows in one warp, which then publishes them as one store
    const int first_task = tid >= kResUnitWarps * 32 ? tid - kResUnitWarps * 32 : tid + kResRowWarps * 32;

    // ---- the block's units, once: one barrier counts all their bytes
    if (tid == 0) {
        mbar_init(smem_u32(bar), 1);
        *ok = 1;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    if (tid == 0) {
        uint32_t total = 0;
#pragma unroll 1
        for (int l = 0; l < n_local; ++l) {
            const GainUnit U = r.units[u0 + l];
            const int nvr = U.n2p / Vec<T>::n, w = (nvr + KV - 1) / KV;
            ResUnit R{};
            R.soff = (int)total;
            R.inv = (65536 + w - 1) / w;
            R.b_off = (unsigned short)U.b_off;
            R.c_off = (unsigned short)U.c_off;
            R.nb = (unsigned short)U.nb;
            R.nvr = (unsigned short)nvr;
            R.w = (unsigned short)w;
            R.dr = (unsigned short)(kGainConsumers / w);
            R.row = (unsigned short)U.row;
            R.slot = (unsigned short)r.slot[u0 + l];
            unit[l] = R;
            total += (uint32_t)U.nb * U.n2p * sizeof(T);
        }
        mbar_arrive_expect_tx(smem_u32(bar), total);
#pragma unroll 1
        for (int l = 0; l < n_local; ++l) {
            const GainUnit U = r.units[u0 + l];
            bulk_g2s(smem_u32(smem + unit[l].soff), static_cast<const T*>(r.G) + U.g_off,
                     (uint32_t)U.nb * U.n2p * sizeof(T), smem_u32(bar));
        }
    }
    // ---- the state: padded per species and cell, and in its own order where the two differ
#pragma unroll 1
    for (int k = tid; k < r.f_len * staged; k += kResThreads) {
        const int cell = k / r.f_len, i = k - cell * r.f_len;
        int s = 0;
#pragma unroll 1
        while (s + 1 < so.n && i >= so.offp[s + 1]) ++s;
        const int j = i - so.offp[s];
        f_s[k] = cell < n_space && j < so.off[s + 1] - so.off[s] ? (S)f_in[(size_t)cell * n_mom + so.off[s] + j] : S(0);
    }
    if (r.pad)
#pragma unroll 1
        for (int k = tid; k < n_state; k += kResThreads) fu[k] = (S)f_in[k];
    // ---- this thread's states in the gather
    int pos_q[NS];  // place in f_s
#pragma unroll
    for (int q = 0; q < NS; ++q) {
        const int i = tid + q * kResThreads;
        pos_q[q] = 0;
        if (i < n_state) {
            const int cell = i / n_mom, a = i - cell * n_mom;
            int s = 0;
#pragma unroll 1
            while (s + 1 < so.n && a >= so.off[s + 1]) ++s;
            pos_q[q] = cell * r.f_len + so.offp[s] + a - so.off[s];
        }
    }
    volatile int never = 0;
    if (!mbar_wait_bounded(smem_u32(bar), 0u, &never)) {
        if (tid == 0) atomicOr(r.err, KERR_TIMEOUT_FULL);
        *ok = 0;
    }
    __syncthreads();
    const unsigned long long step0 = *reinterpret_cast<const volatile unsigned long long*>(ctr);
    const auto f_at = [fu](int k) { return (double)fu[k]; };

    for (int k = 0; k < n_steps && *ok; ++k) {
        const double dt_scale = dt_arr[step0 + (unsigned)k];
        const unsigned long long tag = r.base + (unsigned)k + 1;
        ResWord* partial = reinterpret_cast<ResWord*>(r.partial) + (size_t)(k & 1) * (kResSegs - 1) * n_state;
        ResWord* next = reinterpret_cast<ResWord*>(r.next) + (size_t)(k & 1) * n_state;
        double* diag = r.diag + (size_t)k * kStepRecFields * n_state;
        if (warp < kResUnitWarps) {
            // ---- 1. the block's units, a group of threads to each
            const int grp = tid / kGainConsumers, gt = tid - grp * kGainConsumers, gw = gt >> 5;
            constexpr int P = pow2_ceil(C), UB = P < 4 ? 4 / P : 1;  // units whose sums are reduced together
            for (int c0 = 0; c0 < n_space; c0 += C) {
                const S* fc = f_s + c0 * r.f_len;
                UnitSum<T, C, KV> sum;
                int c_off = -1, nvr = 0;  // the columns in sum's x
#pragma unroll 1
                for (int l0 = grp; l0 < n_local; l0 += kResGroups * UB) {
                    double part[UB * P] = {};
#pragma unroll
                    for (int ub = 0; ub < UB; ++ub) {
                        const int l = l0 + ub * kResGroups;
                        if (l >= n_local) continue;
                        const ResUnit U = unit[l];
                        UnitMap m;
                        m.nvr = U.nvr;
                        m.w = U.w;
                        m.dr = U.dr;
                        m.r0 = gt * U.inv >> 16;
                        m.cv = gt - m.r0 * m.w;
                        m.on = m.r0 < m.dr;
                        if (sum.kDotRows && (U.c_off != c_off || U.nvr != nvr)) {
                            c_off = U.c_off;
                            nvr = U.nvr;
                            sum.load_x(m, fc + c_off, r.f_len);
                        }
                        sum.begin();
                        int row = m.r0;
                        sum.tile(m, smem + U.soff, U.nb, row, fc + U.b_off, r.f_len);
                        sum.finish(m, fc + U.c_off, r.f_len);
#pragma unroll
                        for (int c = 0; c < C; ++c) part[ub * P + c] = sum.acc[c];
                    }
                    const double acc = warp_sum_n<UB * P>(part, lane);
                    constexpr int kLanes = 32 / (UB * P);
                    const int j = lane / kLanes, l = l0 + j / P * kResGroups, c = j % P;
                    if (lane % kLanes == 0 && l < n_local && c < C && c0 + c < n_space)
                        red[(l * kGainConsumerWarps + gw) * n_space + c0 + c] = acc;
                }
            }
        }
        // flux, emission and loss of the owned rows
        if (warp >= kResUnitWarps) {
#pragma unroll 1
            for (int t = warp - kResUnitWarps; t < n_own * n_space; t += kResRowWarps) {
                const int c = n_space == 1 ? 0 : t / n_own, a = own0 + t - c * n_own, i = c * n_mom + a;
                int s = 0;
#pragma unroll 1
                while (s + 1 < so.n && a >= so.off[s + 1]) ++s;
                double flux, emi, loss;
                row_terms(ops, i, c, a, s, ops.has_bin != 0, lane, f_at, flux, emi, loss);
                if (lane < 4) rest[t * 4 + lane] = lane == 0 ? flux : (lane == 1 ? emi : (lane == 2 ? loss : f_at(i)));
            }
        }
        __syncthreads();
        // ---- 2. a thread for every owned row and cell, and for what the block has of a row before
        bool there = true;
        const int n_far = unit[0].slot > 0 ? n_space : 0, n_task = n_own * n_space;
#pragma unroll 1
        for (int t = first_task; t < n_far + n_task; t += kResThreads) {
            const bool far = t >= n_task;
            const int tt = far ? t - n_task : t;
            const int c = n_space == 1 ? 0 : (far ? tt : tt / n_own), a = far ? unit[0].row : own0 + tt - c * n_own;
            const int i = c * n_mom + a;
            const int lo = max(__ldg(ops.unit_ptr + a) - u0, 0), hi = __ldg(ops.unit_ptr + a + 1) - u0;
            const int2 cut = __ldg(ops.cuts + a);
            // the row's units in this block: each over its warps in order, then the units in order
            double seg = 0.0;
            const int end = min(n_local, hi);
#pragma unroll 1
            for (int l = lo; l < end; l += 4) {  // four chains at a time
                double s[4] = {};
#pragma unroll
                for (int w = 0; w < kGainConsumerWarps; ++w)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (l + j < end) s[j] += red[((l + j) * kGainConsumerWarps + w) * n_space + c];
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (l + j < end) seg += s[j];
            }
            if (far) {
                store_word(partial + (size_t)(unit[0].slot - 1) * n_state + i, seg, tag);
                continue;
            }
            const T iap = __ldg(ops.invAp + i), injv = __ldg(ops.inj + i), volc = __ldg(ops.vol + c);
            const double flux = rest[t * 4], emi = rest[t * 4 + 1], loss = rest[t * 4 + 2];
            const T fa = (T)rest[t * 4 + 3];
            double g1 = 0.0, g2 = 0.0;
            if (cut.x - u0 < hi) there = wait_word(partial + i, tag, g1) && there;
            if (cut.y - u0 < hi) there = wait_word(partial + n_state + i, tag, g2) && there;
            T dbin;
            const T df = row_df(ops, ops.has_bin != 0, fa, iap, volc, flux, emi, loss, row_gain(seg, g1, g2), dt_scale, dbin);
            if (SY) {
                const T fm = fa + df;
                store_word(next + i, (double)jl_mul_bool(fm, fm >= (T)ops.thr_mom), tag);
                rest[t * 4] = (double)df;  // for the records below
            } else {
                store_word(next + i, (double)row_update(ops, fa, df, injv, dt_scale), tag);
                diag[i] = (double)df;
                diag[5 * n_state + i] = (double)fa;
                if (verbose == 3) {
                    diag[1 * n_state + i] = (double)dbin;
                    diag[2 * n_state + i] = (double)(T)emi;
                    diag[3 * n_state + i] = -(double)(T)flux;
                }
            }
        }
        // ---- 3. the whole new state (or f_Momentum); the old one is no longer read
#pragma unroll
        for (int q = 0; q < NS; ++q) {
            const int i = tid + q * kResThreads;
            double v = 0.0;
            // one lane waits first: a warp of polls would keep the slices of L2 busy that the words
            // still to come have to pass
            if (q == 0 && lane == 0 && i < n_state) there = wait_word(next + i, tag, v) && there;
            __syncwarp();
            if (i >= n_state) continue;
            there = wait_word(next + i, tag, v) && there;
            if (!SY) f_s[pos_q[q]] = (S)v;
            if (SY || r.pad) fu[i] = (S)v;  // without padding fu is f_s, in the same order
        }
        if (!there) {
            atomicOr(r.err, KERR_TIMEOUT_FULL);
            *ok = 0;
        }
        __syncthreads();
        if (SY) {
            // the space pass on the momentum pass's state, by every block for itself (the X flux's
            // slots summed as its warp does)
            const auto space = [&](int i, T& dsp) {
                double t[kResMaxX];
#pragma unroll
                for (int e = 0; e < kResMaxX; ++e) {
                    t[e] = 0.0;
                    if (e < ops.x_ell_w) {
                        const int c = __ldg(ops.x_ell_col + (size_t)i * ops.x_ell_w + e);
                        if (c >= 0) t[e] = fma((double)__ldg(ops.x_ell_val + (size_t)i * ops.x_ell_w + e), (double)fu[c], 0.0);
                    }
                }
                static_assert(kResMaxX == 8, "the warp's tree over eight slots");
                const double xf = ((t[0] + t[4]) + (t[2] + t[6])) + ((t[1] + t[5]) + (t[3] + t[7]));
                return row_space_update(ops, (T)fu[i], xf, __ldg(ops.invAp + i), __ldg(ops.inj + i), dt_scale, dsp);
            };
            S fn[NS];
            T dsp;
#pragma unroll
            for (int q = 0; q < NS; ++q) {
                const int i = tid + q * kResThreads;
                fn[q] = i < n_state ? (S)space(i, dsp) : S(0);
            }
#pragma unroll 1
            for (int t = first_task; t < n_task; t += kResThreads) {  // the threads that updated the rows
                const int c = n_space == 1 ? 0 : t / n_own, i = c * n_mom + own0 + t - c * n_own;
                space(i, dsp);
                diag[i] = (double)(T)(dsp + (T)rest[t * 4]);
                diag[5 * n_state + i] = rest[t * 4 + 3];
            }
            __syncthreads();
#pragma unroll
            for (int q = 0; q < NS; ++q) {
                const int i = tid + q * kResThreads;
                if (i >= n_state) continue;
                f_s[pos_q[q]] = fn[q];
                if (r.pad) fu[i] = fn[q];
            }
            __syncthreads();
        }
    }
    // every block holds the whole state: each writes its share
#pragma unroll 1
    for (int i = blk * kResThreads + tid; i < n_state; i += grid * kResThreads) f_out[i] = (T)fu[i];
}

template <typename T>
using ResKernel = void (*)(RowOps<T>, ResidentArgs, SpOff, const T*, T*, const double*, const unsigned long long*, int, int);

// At most kResAcc accumulators per thread (96 registers).
constexpr int kResAcc = 24;

// The instances that a state of at most resident_max_states() can ask for. Rows of more than 512
// FP64 or 1,024 FP32 states leave room for one cell (two with 513 to 960 FP64 states), and a state
// with them is longer than 640, except one cell's of 513 to 632 FP64 states.
template <typename T, int KV, int C>
ResKernel<T> res_kernel_upto(int cells, bool sy, bool one) {
    if constexpr (C > 1) {
        if (cells < C) return res_kernel_upto<T, KV, C - 1>(cells, sy, one);
    }
    if constexpr (KV == 1 || (KV == 2 && sizeof(T) == 8 && C != 2)) {
        if (one) return sy ? resident_kernel<T, C, KV, true, 1> : resident_kernel<T, C, KV, false, 1>;
    }
    return sy ? resident_kernel<T, C, KV, true, kResStates> : resident_kernel<T, C, KV, false, kResStates>;
}
template <typename T>
ResKernel<T> res_kernel(const GainPass& p, bool sy, int n_state) {
    constexpr int n = Vec<T>::n;
    const bool one = n_state <= kResThreads;
    if constexpr (sizeof(T) == 4) {
        return p.kv == 1 ? res_kernel_upto<T, 1, kResAcc / n>(p.cells, sy, one) : res_kernel_upto<T, 2, 1>(p.cells, sy, one);
    } else {
        if (p.kv == 1) return res_kernel_upto<T, 1, 2>(p.cells, sy, one);
        return p.kv == 2 ? res_kernel_upto<T, 2, kResAcc / (2 * n)>(p.cells, sy, one)
                         : res_kernel_upto<T, 4, 1>(p.cells, sy, one);
    }
}
// cells of a pass at most, by columns per thread: 0 where there is no instance
int res_cells(int elem_size, int kv) {
    if (elem_size == 4) return kv == 1 ? 6 : (kv == 2 ? 1 : 0);
    return kv == 1 ? 2 : (kv == 2 ? 6 : (kv == 4 ? 1 : 0));
}

}  // namespace

int resident_smem_bytes(const GainPass& p, int elem_size, int g_bytes, int f_len, int n_space, int n_state, bool pad,
                        int max_local, int max_own) {
    const int staged = (n_space + p.cells - 1) / p.cells * p.cells;
    return res_layout(g_bytes, p.cells == 1 ? elem_size : 8, f_len, staged, n_space, n_state, pad, max_local, max_own)
        .bytes;
}

// The pass over the resident units: gain_pass's columns per thread and the cells that the
// accumulators allow, split evenly (no cells: no such instance).
GainPass resident_pass(int elem_size, const GainPass& g, int n_space) {
    const int most = res_cells(elem_size, g.kv);
    const int passes = most > 0 ? (n_space + most - 1) / most : 0;
    GainPass p;
    p.kv = g.kv;
    p.cells = passes > 0 ? (n_space + passes - 1) / passes : 0;
    return p;
}

int resident_max_states() { return kResStates * kResThreads; }

template <typename T>
cudaError_t prepare_resident(const GainPass& p, bool sy, int n_state, int smem, int* blocks_per_sm) {
    const auto k = res_kernel<T>(p, sy, n_state);
    const cudaError_t e = allow_gain_smem(k);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k, kResThreads, smem);
}

template <typename T>
cudaError_t launch_resident(const GainPass& p, const RowOps<T>& ops, const ResidentArgs& r, const int* sp_off_host,
                            const T* f_in, T* f_out, const double* dt_arr, const unsigned long long* ctr, int n_steps,
                            int verbose, int grid, int smem, bool sy, cudaStream_t s) {
    SpOff so;
    so.n = ops.n_species;
    for (int i = 0; i <= so.n; ++i) {
        so.off[i] = sp_off_host[i];
        so.offp[i] = sp_off_host[so.n + 1 + i];
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kResThreads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, res_kernel<T>(p, sy, ops.n_state), ops, r, so, f_in, f_out, dt_arr, ctr, n_steps, verbose);
}

template cudaError_t prepare_resident<double>(const GainPass&, bool, int, int, int*);
template cudaError_t prepare_resident<float>(const GainPass&, bool, int, int, int*);
template cudaError_t launch_resident<double>(const GainPass&, const RowOps<double>&, const ResidentArgs&, const int*,
                                             const double*, double*, const double*, const unsigned long long*, int, int,
                                             int, int, bool, cudaStream_t);
template cudaError_t launch_resident<float>(const GainPass&, const RowOps<float>&, const ResidentArgs&, const int*,
                                            const float*, float*, const double*, const unsigned long long*, int, int,
                                            int, int, bool, cudaStream_t);

}  // namespace dtb
