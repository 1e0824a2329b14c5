// Forward kernels: spatial operator, CFL time step, fused SSPRK33 step, batched
// persistent stepping with per-instance dt, and the C ABI around them.
//
// Reference path replaced (alexfikl/pyshocks):
//   apply_operator      src/pyshocks/schemes.py:339-346
//   periodic ghost fill src/pyshocks/scalar.py:529-540
//   numerical fluxes    src/pyshocks/scalar.py:91-132,192-278,
//                       src/pyshocks/burgers/schemes.py:98-153,230-256
//   predict_timestep    src/pyshocks/burgers/schemes.py:42-49,121-127
//   step / SSPRK33      src/pyshocks/timestepping.py:89-152,312-320
//
// Periodic boundaries are applied by circular indexing of the n interior
// cells: with stencil reach 3 and 3 ghost cells the reference's interior
// outputs equal the circular ones (its zero padding reaches ghost outputs only).
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>
#include <vector>

#include "stencil.cuh"
#ifdef SHOCKS_BOUNDS_CHECK
#include "shocks_check.h"
#endif

namespace shk {

// ---------------------------------------------------------------------------
// batched persistent stepping kernel
// ---------------------------------------------------------------------------
// Persistent CTAs take (instance, tile) items; a window is loaded by bulk copies,
// three stages run in shared memory on shrinking ranges, one write of the state.
// HBM is idle (16 bytes a cell-step: 61 us of 1199 at 25.9 M cells). What bounds
// it: the integer-flux form, issue and the integer, FMA and FP64 pipes together
// (step_tile_fx); the other float64 forms, the FP64 pipe; float32, issue (241 us
// a step at that size); learned, the special-function pipe.
//
// One thread, when a tile of instance b is done in step k (s: the instance's
// step). The CTA that finishes the instance's last tile advances its time,
// records dt and clears the consumed maximum (every other tile has read both),
// so the steps of thousands of instances are not finalised by one CTA after all
// others are done (25.9 M cells in 4096 instances, us per step: float32 281 -> 241,
// float64 1139 -> 1121, learned 216 -> 213 at 2.8 M cells). True for that last tile.
__device__ __forceinline__ bool finish_tile(const PlanDev& P, int64_t k, int b, int tiles, const DtState& s) {
    __threadfence();
    if (atomicAdd(P.left + b, 1u) != static_cast<unsigned>(tiles) - 1u) return false;
    P.left[b] = 0u;
    double rec = 0.0;
    if (s.active) {
        if (s.finite) {
            P.t[b] = P.t[b] + s.dt;
            rec = s.dt;
        } else {
            atomicOr(P.status, ERR_NONFINITE);
        }
    }
    if (P.dt_hist && k < P.max_steps) P.dt_hist[size_t(k) * P.B + b] = rec;
    P.amax[size_t(k & 1) * P.B + b] = 0ull;
    return true;
}

// A tile whose maximum and completion are still to be reported. kDefer: the atomics
// (one returns a value, behind a fence) run while the next item's window is in flight
// instead of before its load. Measured, 4096 instances (25.9 M cells), ten float32
// steps: 2491 -> 2413 us; learned float64: 1051 -> 1039 us. The integer-flux kernel
// reports at once: eight CTAs on an SM hide each other's atomics already (4096
// instances, two steps: 2398 us, deferred 2413; 300 ragged instances, ten steps:
// 693 us, deferred 731). wmax: the warps' maxima of |f'|, as double bits.
template <int FLUX>
inline constexpr bool kDefer = FLUX != kFluxRusanovFx;
struct PendingTile {
    unsigned long long wmax[32];
    DtState dt;
    int b, tiles;  // b < 0: none
};
__device__ __forceinline__ void pending_fill(PendingTile& pt, unsigned long long mx, int b, int tiles,
                                             const DtState& dt) {
    mx = warp_max(mx);
    if ((threadIdx.x & 31) == 0) pt.wmax[threadIdx.x >> 5] = mx;
    if (threadIdx.x == 0) {
        pt.dt = dt;
        pt.b = b;
        pt.tiles = tiles;
    }
}
// thread 0, after a barrier
__device__ __forceinline__ void pending_flush(PendingTile& pt, const PlanDev& P, int64_t k, unsigned long long* amax) {
    if (pt.b < 0) return;
    unsigned long long m = pt.wmax[0];
    for (int w = 1; w < static_cast<int>(blockDim.x >> 5); ++w) m = pt.wmax[w] > m ? pt.wmax[w] : m;
    atomicMax(amax + pt.b, m);
    finish_tile(P, k, pt.b, pt.tiles, pt.dt);
}

template <class T, int EQ, int REC, int FLUX>
__global__ void __launch_bounds__(flux_threads<FLUX>(), FLUX == kFluxRusanovFx ? 8 : (REC == SHK_REC_LEARNED ? 3 : (REC == SHK_REC_WENOJS53 ? (sizeof(T) == 8 ? 3 : 4) : 1))) batched_step_kernel(PlanDev P, const T* __restrict__ uin,
                                                                T* __restrict__ uout, OpParams<T> p) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ PendingTile pending;         // kDefer
    __shared__ unsigned long long red[32];  // else
    __shared__ DtState item_dt;  // the item's step, computed once per CTA
    __shared__ T item_dtdx, item_dx;
    constexpr int HL = step_halo<T>();
    using B = typename Bits<T>::type;

    Smem<T> sm;
    carve_step<T, REC, FLUX>(sm, smem_raw, P.tile + 2 * HL);
    if (threadIdx.x == 0) {
        if constexpr (kDefer<FLUX>) pending.b = -1;
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    learned_stage<REC>(p.lp);
    uint32_t phase = 0;
    const int64_t k = *reinterpret_cast<volatile int64_t*>(P.step);
    const int cur = static_cast<int>(k & 1), nxt = cur ^ 1;
    bool ok = true;
    const int64_t total = P.offsets[P.B];
    const Win<const T> guin = make_win(uin, total);
    const Win<T> guout = make_win(uout, total);

    __shared__ int s_item[2];
    for (ItemQueue<REC != SHK_REC_LEARNED> items(P, 0, s_item); items.more(); items.end()) {
        const PlanItem it = items.begin();
        const int b = it.b, te = it.te;
        const int64_t off = it.off, n = it.n, s0 = int64_t(it.tile) * P.tile;
        // one thread evaluates the step (double divisions: a 1/64-rate pipe on
        // this GPU) while the window is in flight, and shares it; the previous
        // item's readers are past the barrier that ended that item
        ok = load_window<T>(sm.U, uin + off, n, s0 - HL, te + 2 * HL, &bar, phase, [&] {
            if constexpr (kDefer<FLUX>) {
                if (threadIdx.x == 0) pending_flush(pending, P, k, P.amax + size_t(nxt) * P.B);
            }
            if (threadIdx.x == 32) {
                const DtState d = plan_dt(P, k, b, from_bits(P.amax[size_t(cur) * P.B + b]));
                item_dt = d;
                item_dtdx = static_cast<T>(d.dt * P.inv_dx[b]);
                item_dx = static_cast<T>(1.0 / P.inv_dx[b]);
            }
        });
        if (!ok) {
            if (threadIdx.x == 0) {
                atomicOr(P.status, ERR_TIMEOUT);
                if constexpr (kDefer<FLUX>) pending.b = -1;
            }
            break;
        }
        const DtState ds = item_dt;
        B mx = 0;
        if (!(ds.active && ds.finite)) {
            // instance finished or frozen: copy the tile through
            for (int i = threadIdx.x; i < te; i += blockDim.x) {
                const T v = guin[off + s0 + i];
                guout[off + s0 + i] = v;
                const B bb = abs_bits(wave_speed<EQ>(v, p.c));
                mx = bb > mx ? bb : mx;
            }
        } else {
            const T dtdx = item_dtdx;
            OpParams<T> pb = p;
            pb.dx = item_dx;
            mx = step_tile<T, EQ, REC, FLUX>(sm, guout + (off + s0), te, dtdx, pb, plan_bc(P, b, k),
                                             s0 - HL, n);
        }
        if constexpr (kDefer<FLUX>) {
            pending_fill(pending, to_double_bits<T>(mx), b, it.tiles, ds);
        } else {
            const B bm = block_max<B>(mx, reinterpret_cast<B*>(red));
            if (threadIdx.x == 0) {
                atomicMax(P.amax + size_t(nxt) * P.B + b, to_double_bits<T>(bm));
                finish_tile(P, k, b, it.tiles, ds);
            }
        }
    }

    // the last CTA of the step increments the step counter (no host round trip)
    if (threadIdx.x == 0) {
        if constexpr (kDefer<FLUX>) pending_flush(pending, P, k, P.amax + size_t(nxt) * P.B);
        __threadfence();
        if (atomicAdd(P.done, 1u) == gridDim.x - 1) {
            __threadfence();
            *reinterpret_cast<volatile unsigned*>(P.done) = 0u;
            atomicExch(P.sched, 0u);  // every CTA has taken its last item
            *reinterpret_cast<volatile int64_t*>(P.step) = k + 1;
            __threadfence();
        }
    }
}

// ---------------------------------------------------------------------------
// several steps of short instances in one launch
// ---------------------------------------------------------------------------
// A step of a batch that does not fill the GPU costs its latency: a launch, the
// item's and the instance's data, the window, three stages, the completion
// atomics. Instances do not couple, so where every instance has a CTA of its own
// (Plan::resident), one launch takes all steps with the state in shared memory:
// each step's result is written over its window, the halo is refilled from the
// interior, and the maximum the next CFL step needs stays in a register. Same
// tile code and so the same values as the step-by-step launches.
// u_cur / u_prev: the buffers of the state after the last and the last but one
// step (u_prev is written when nsteps > 1). Measured (us per step, smooth states,
// 24 instances; launched one by one -> resident): 240 cells 14.4 -> 7.1, 1000
// cells 24.6 -> 13.8; 100 to 1000 cells with fronts 33 -> 19.
constexpr int kResidentThreads = 1024;
template <class T, int EQ, int REC, int FLUX>
__global__ void __launch_bounds__(kResidentThreads, 1) resident_steps_kernel(
    PlanDev P, const T* uin, T* u_cur, T* u_prev, OpParams<T> p, int W, int nsteps) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ unsigned long long red[32];
    __shared__ DtState step_dt;
    constexpr int HL = step_halo<T>();
    using B = typename Bits<T>::type;
    Smem<T> sm;
    carve_step<T, REC, FLUX>(sm, smem_raw, W);
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    uint32_t phase = 0;
    const int64_t k0 = *reinterpret_cast<volatile int64_t*>(P.step);
    const int b = blockIdx.x;
    const int64_t off = P.offsets[b];
    const int n = static_cast<int>(P.offsets[b + 1] - off);
    const double inv_dx = P.inv_dx[b];
    unsigned long long amax = P.amax[size_t(k0 & 1) * P.B + b];  // thread 0 keeps it up to date
    bool ok = load_window<T>(sm.U, uin + off, n, -HL, n + 2 * HL, &bar, phase);
    if (!ok && threadIdx.x == 0) atomicOr(P.status, ERR_TIMEOUT);  // (and no state is written)
    const Win<T> ug = make_win(u_cur, P.offsets[P.B]) + off;
    const Win<T> pg = make_win(u_prev, P.offsets[P.B]) + off;
    OpParams<T> pb = p;
    pb.dx = static_cast<T>(1.0 / inv_dx);
    for (int s = 0; s < nsteps && ok; ++s) {
        const int64_t k = k0 + s;
        if (threadIdx.x == 0) {
            const DtState d = plan_dt(P, k, b, from_bits(amax));
            double rec = 0.0;
            if (d.active) {
                if (d.finite) {
                    P.t[b] = P.t[b] + d.dt;
                    rec = d.dt;
                } else {
                    atomicOr(P.status, ERR_NONFINITE);
                }
            }
            if (P.dt_hist && k < P.max_steps) P.dt_hist[size_t(k) * P.B + b] = rec;
            step_dt = d;
        }
        if (s > 0 && s == nsteps - 1)
            for (int i = threadIdx.x; i < n; i += blockDim.x) pg[i] = sm.U[HL + i];
        __syncthreads();
        const DtState ds = step_dt;
        if (ds.active && ds.finite) {
            const T dtdx = static_cast<T>(ds.dt * inv_dx);
            const B mx = step_tile<T, EQ, REC, FLUX>(sm, sm.U + HL, n, dtdx, pb, plan_bc(P, b, k), -HL, n);
            const B bm = block_max<B>(mx, reinterpret_cast<B*>(red));  // (its barriers end the tile's writes)
            if (threadIdx.x == 0) amax = to_double_bits<T>(bm);
            for (int i = threadIdx.x; i < 2 * HL; i += blockDim.x) {
                const int w = i < HL ? i : n + i;
                const int c = (w - HL) % n;
                sm.U[w] = sm.U[HL + (c < 0 ? c + n : c)];
            }
        }
        __syncthreads();
    }
    if (ok)
        for (int i = threadIdx.x; i < n; i += blockDim.x) ug[i] = sm.U[HL + i];
    if (threadIdx.x == 0) {
        P.amax[size_t((k0 + nsteps) & 1) * P.B + b] = amax;
        P.amax[size_t((k0 + nsteps + 1) & 1) * P.B + b] = 0ull;
        __threadfence();
        if (atomicAdd(P.done, 1u) == gridDim.x - 1) {
            *reinterpret_cast<volatile unsigned*>(P.done) = 0u;
            *reinterpret_cast<volatile int64_t*>(P.step) = k0 + nsteps;
            __threadfence();
        }
    }
}

// ---------------------------------------------------------------------------
// batched global Lax-Friedrichs: one launch per SSPRK33 stage
// ---------------------------------------------------------------------------
// The wave speed of the global Lax-Friedrichs flux is the maximum of |f'| over
// the whole instance, for each stage state (scalar.py:258-278 under
// timestepping.py:312-320), so the stages cannot be fused with halo
// recompute. Stage S reads a window of its input k (u, k1 or k2) and u, writes
// its output (k1, k2 or u+) and accumulates the instance maximum of |f'| of the
// output for the next stage (amax_out). Stage 1 uses the step's own maximum
// (amax[cur], which is also the CFL maximum), and every stage evaluates the
// instance's dt the same way; the last CTA of stage 3 finalises the step as
// batched_step_kernel does and clears the stage maxima. float64 states,
// periodic instances, the reference's stage formulas:
//   k1 = u + dt L(u),  k2 = 3/4 u + 1/4 (k1 + dt L(k1)),  u+ = 1/3 u + 2/3 (k2 + dt L(k2)).
// FX: the fluxes of fixed_flux.cuh, in 128-thread CTAs (512 instances, 1.2 M cells:
// 425 -> 117 us per step of three launches). Bound by issue as the fused step, and
// by the tail of each launch: 2600 tiles on 1216 CTA slots.
template <int EQ, int STAGE, bool FX>
__global__ void __launch_bounds__(FX ? kFxThreads : kThreads, FX ? 8 : 1) batched_lf_stage_kernel(
    PlanDev P, const double* __restrict__ u, const double* __restrict__ kin, double* __restrict__ kout,
    const unsigned long long* __restrict__ amax_in, unsigned long long* amax_out,
    unsigned long long* amax_clear, OpParams<double> p) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ unsigned long long red[32];
    __shared__ DtState item_dt;
    __shared__ double item_dtdx, item_amax;
    constexpr int HL = op_halo<double>();
    Smem<double> sm;
    if constexpr (FX) sm.carve_lf_stage(smem_raw, P.tile + 2 * HL);
    else sm.carve(smem_raw, P.tile + 2 * HL);
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    uint32_t phase = 0;
    const int64_t k = *reinterpret_cast<volatile int64_t*>(P.step);
    const int cur = static_cast<int>(k & 1);
    const int64_t total = P.offsets[P.B];
    const Win<const double> gu = make_win(u, total);
    const Win<double> gout = make_win(kout, total);
    // stage 1 reads the step's own maximum, stage 3 writes the next step's
    // (the parity of the device step counter picks the slot)
    const unsigned long long* ain = STAGE == 1 ? P.amax + size_t(cur) * P.B : amax_in;
    unsigned long long* aout = STAGE == 3 ? P.amax + size_t(cur ^ 1) * P.B : amax_out;
    bool ok = true;
    [[maybe_unused]] int slot = 0;
    __shared__ int s_item[2];
    for (ItemQueue<> items(P, 6, s_item); items.more(); items.end()) {
        const PlanItem it = items.begin();
        const int b = it.b, te = it.te;
        const int64_t off = it.off, n = it.n, s0 = int64_t(it.tile) * P.tile;
        ok = load_window<double>(sm.U, kin + off, n, s0 - HL, te + 2 * HL, &bar, phase, [&] {
            if (threadIdx.x == 32) {
                const DtState d = plan_dt(P, k, b, from_bits(P.amax[size_t(cur) * P.B + b]));
                item_dt = d;
                item_dtdx = d.dt * P.inv_dx[b];
                item_amax = from_bits(ain[b]);
            }
        });
        if (!ok) {
            if (threadIdx.x == 0) atomicOr(P.status, ERR_TIMEOUT);
            break;
        }
        const DtState ds = item_dt;
        unsigned long long mx = 0;
        if (!(ds.active && ds.finite)) {
            // instance finished or frozen: every stage state is u
            for (int i = threadIdx.x; i < te; i += blockDim.x) {
                const double v = gu[off + s0 + i];
                gout[off + s0 + i] = v;
                const unsigned long long bb = abs_bits(wave_speed<EQ>(v, p.c));
                mx = bb > mx ? bb : mx;
            }
        } else {
            double dtdx = item_dtdx;
            if constexpr (FX) {
                // (the list's counters 0 and 1 alternate)
                fx_fluxes<true>(sm.U, HL - 1, HL + te, sm, p, slot,
                                StoreFaces<Win<double>>{Win<double>(), Win<double>(), 0, 0, 0}, item_amax);
                slot ^= 1;
                dtdx *= 1.0 / 288.0;
            } else {
                OpParams<double> pb = p;
                pb.hnu_amax = p.hnu * item_amax;
                face_fluxes<double, EQ, SHK_REC_WENOJS53, SHK_FLUX_LF>(sm.U, HL, HL + te, sm, pb);
            }
            for (int i = threadIdx.x; i < te; i += blockDim.x) {
                const int w = HL + i;
                const double kk = fma(dtdx, sm.D[w - 1] - sm.D[w], sm.U[w]);  // k + dt L(k)
                double v;
                if constexpr (STAGE == 1) v = kk;
                else if constexpr (STAGE == 2) v = fma(1.0 / 4.0, kk, (3.0 / 4.0) * gu[off + s0 + i]);
                else v = fma(2.0 / 3.0, kk, (1.0 / 3.0) * gu[off + s0 + i]);
                gout[off + s0 + i] = v;
                const unsigned long long bb = abs_bits(wave_speed<EQ>(v, p.c));
                mx = bb > mx ? bb : mx;
            }
        }
        const unsigned long long bm = block_max<unsigned long long>(mx, red);
        if (threadIdx.x == 0) {
            atomicMax(aout + b, bm);
            if constexpr (STAGE == 3) {
                // the instance's stage maxima are consumed too
                if (finish_tile(P, k, b, it.tiles, ds)) amax_clear[b] = amax_clear[P.B + b] = 0ull;
            }
        }
    }
    if constexpr (STAGE < 3) {
        finish_items(P, 6);
    } else if (threadIdx.x == 0) {
        // the last CTA of the step increments the step counter
        __threadfence();
        if (atomicAdd(P.done, 1u) == gridDim.x - 1) {
            __threadfence();
            *reinterpret_cast<volatile unsigned*>(P.done) = 0u;
            atomicExch(P.sched + 6, 0u);
            atomicExch(P.sched + 7, 0u);
            *reinterpret_cast<volatile int64_t*>(P.step) = k + 1;
            __threadfence();
        }
    }
}

// plan reset in one launch (a memset per array cost the host stepper's chunks more
// than their steps: a host batch of 1024 instances, one step, 527 us -> 374 with this
// and the maximum below): counters, maxima and per-instance times; t0 / tfinal null: 0 /
// no final time
__global__ void reset_kernel(PlanDev P, unsigned long long* amax_lf, double* tfinal_dev, const double* t0,
                             const double* tfinal) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 2 * P.B) {
        P.amax[i] = 0ull;
        if (amax_lf) amax_lf[i] = 0ull;
    }
    if (i < P.B) {
        P.left[i] = 0u;
        P.t[i] = t0 ? t0[i] : 0.0;
        tfinal_dev[i] = tfinal ? tfinal[i] : DBL_MAX;
    }
    if (i < 8) P.sched[i] = 0u;
    if (i == 0) {
        *P.step = 0;
        *P.done = 0u;
        *P.status = 0;
    }
}

// max |f'(u)| per instance into amax[cur] (plan reset / priming): one read of the
// state, eight loads in flight per thread (22 MB: 21 us with one at a time, 9 now)
template <class T, int EQ>
__global__ void __launch_bounds__(kThreads) batched_max_kernel(PlanDev P, const T* __restrict__ u, T c,
                                                               int slot) {
    __shared__ unsigned long long red[32];
    using B = typename Bits<T>::type;
    for (int q = blockIdx.x; q < P.nitems; q += gridDim.x) {
        const PlanItem it = P.items[q];
        const T* v = u + it.off + int64_t(it.tile) * P.tile;
        B mx = 0;
        for (int i0 = threadIdx.x; i0 < it.te; i0 += 8 * kThreads) {
            T x[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int i = i0 + k * kThreads;
                x[k] = v[i < it.te ? i : i0];
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const B bb = abs_bits(wave_speed<EQ>(x[k], c));
                mx = bb > mx ? bb : mx;
            }
        }
        const B bm = block_max<B>(mx, reinterpret_cast<B*>(red));
        if (threadIdx.x == 0) atomicMax(P.amax + size_t(slot) * P.B + it.b, to_double_bits<T>(bm));
    }
}

// deterministic FP64 reductions: per-item partials, then per-instance ordered sums
template <class T>
__global__ void __launch_bounds__(kThreads) batched_partial_kernel(PlanDev P, const T* __restrict__ u,
                                                                   int mode) {
    __shared__ double red[32];
    for (int item = blockIdx.x; item < P.nitems; item += gridDim.x) {
        const int b = P.item_inst[item];
        const int64_t off = P.offsets[b];
        const int64_t n = P.offsets[b + 1] - off;
        const int64_t s0 = int64_t(P.item_tile[item]) * P.tile;
        const int te = static_cast<int>(imin64(P.tile, n - s0));
        double acc = 0.0;
        for (int i = threadIdx.x; i < te; i += blockDim.x) {
            const double v = static_cast<double>(u[off + s0 + i]);
            if (mode == 0) acc += v;
            else if (mode == 1) acc += fabs(v);
            else if (mode == 2) acc = fma(v, v, acc);
            else acc = fmax(acc, fabs(v));
        }
        // fixed-shape tree: deterministic for a given launch shape
        if (mode == -1) {
            for (int o = 16; o > 0; o >>= 1) acc = fmax(acc, __shfl_xor_sync(0xffffffffu, acc, o));
        } else {
            acc = warp_sum(acc);
        }
        __syncthreads();
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
        __syncthreads();
        if (threadIdx.x == 0) {
            double r = red[0];
            for (int w = 1; w < (blockDim.x >> 5); ++w) r = mode == -1 ? fmax(r, red[w]) : r + red[w];
            P.partial[item] = r;
        }
        __syncthreads();
    }
}
__global__ void instance_sum_kernel(PlanDev P, const int32_t* item_first, int mode, double* out) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= P.B) return;
    double r = 0.0;
    for (int i = item_first[b]; i < item_first[b + 1]; ++i)
        r = mode == -1 ? fmax(r, P.partial[i]) : r + P.partial[i];
    out[b] = r;
}

// ---------------------------------------------------------------------------
// single-instance kernels on the reference's ghosted layout (n + 2g cells)
// ---------------------------------------------------------------------------
// the boundary of a single-instance call (kernel parameter copy)
__device__ __forceinline__ BcView call_bc(const shk_boundary& b, double dx) {
    BcView v;
    v.left = b.left;
    v.right = b.right;
    v.dir = &b.dirichlet[0][0][0];
    v.dir_ss = 6;
    v.neu = &b.neumann[0][0];
    v.neu_ss = 2;
    v.dx = dx;
    return v;
}

// ghost cells of a single-instance output after a non-periodic call: the
// boundary at `stage` applied to the new interior (Neumann mirrors it), or 0
// (zero_ghosts: the operator output, whose ghost values are unspecified)
template <class T>
__global__ void bc_ghost_kernel(T* __restrict__ out, int64_t n, int g, shk_boundary b, double dx,
                                int stage, int zero_ghosts) {
    const int t = threadIdx.x;
    if (t >= 2 * g) return;
    const int side = t / g, k = t - g * side;
    const int kind = side ? b.right : b.left;
    const int64_t gidx = side ? g + n + k : g - 1 - k;  // ghosted index of ghost k
    if (kind == SHK_BC_PERIODIC) return;
    if (zero_ghosts || k >= 3) {
        out[gidx] = T(0);
    } else if (kind == SHK_BC_DIRICHLET) {
        out[gidx] = static_cast<T>(b.dirichlet[stage][side][k]);
    } else {
        const int64_t mirror = side ? g + n - 1 - k : g + k;
        out[gidx] = out[mirror] - static_cast<T>((2 * k + 1) * dx * b.neumann[stage][side]);
    }
}

template <class T, int EQ, int REC, int FLUX>
__global__ void __launch_bounds__(kThreads) apply_operator_kernel(const T* __restrict__ u, T* __restrict__ out,
                                                                  int64_t n, int g, int tile, T dx,
                                                                  const double* amax, OpParams<T> p,
                                                                  int32_t* err, shk_boundary bcp) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar;
    constexpr int HL = op_halo<T>();
    Smem<T> sm;
    sm.carve(smem_raw, tile + 2 * HL);
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    learned_stage<REC>(p.lp);
    uint32_t phase = 0;
    if constexpr (FLUX == SHK_FLUX_LF) p.hnu_amax = p.hnu * static_cast<T>(*amax);
    const int64_t s0 = int64_t(blockIdx.x) * tile;
    const int te = static_cast<int>(imin64(tile, n - s0));
    if (!load_window<T>(sm.U, u + g, n, s0 - HL, te + 2 * HL, &bar, phase)) {
        if (threadIdx.x == 0 && err) atomicOr(err, ERR_TIMEOUT);
        return;
    }
    const BcView bc = call_bc(bcp, static_cast<double>(dx));
    const bool periodic = bc.periodic();
    if (!periodic) apply_bc(sm.U, s0 - HL, n, 0, te + 2 * HL, bc, 0);
    face_fluxes<T, EQ, REC, FLUX>(sm.U, HL, HL + te, sm, p);
    const Win<T> gout = make_win(out, n + 2 * g);
    for (int i = threadIdx.x; i < te; i += blockDim.x) {
        const int w = HL + i;
        // -(f[1:] - f[:-1]) / dx  (schemes.py:346)
        const T r = -((sm.D[w] - sm.D[w - 1]) * p.fscale) / dx;
        const int64_t gi = s0 + i;
        gout[g + gi] = r;
        // ghost cells of the output: periodic image of the interior output
        if (periodic) {
            if (gi < g) gout[g + n + gi] = r;
            if (gi >= n - g) gout[gi - (n - g)] = r;
        }
    }
}

template <class T, int EQ>
__global__ void max_wavespeed_kernel(const T* __restrict__ u, int64_t n, T c, unsigned long long* out) {
    __shared__ unsigned long long red[32];
    using B = typename Bits<T>::type;
    B mx = 0;
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
         i += int64_t(gridDim.x) * blockDim.x) {
        const B bb = abs_bits(wave_speed<EQ>(u[i], c));
        mx = bb > mx ? bb : mx;
    }
    const B bm = block_max<B>(mx, reinterpret_cast<B*>(red));
    if (threadIdx.x == 0) atomicMax(out, to_double_bits<T>(bm));
}

__global__ void finalize_dt_kernel(double* dt, double cfl, double theta) {
    const double smax = from_bits(*reinterpret_cast<unsigned long long*>(dt));
    // theta * (0.5 dx^(2-alpha) / smax)   (burgers/schemes.py:127, examples/burgers.py:162)
    *dt = theta * (cfl / smax);
}

// both in one CTA: a short state's CFL step in one launch instead of three (us, three
// launches / one: 256 cells 7.2 / 3.2, 8192 7.3 / 4.9, 12000 7.3 / 6.2, 24000 7.3 / 8.3, 32768
// 7.3 / 8.5; with the read of dt by the host 8192 21.8 / 19.5, 12000 21.8 / 23.1)
constexpr int64_t kBlockDtCells = 8192;
template <int EQ>
__global__ void __launch_bounds__(1024) block_dt_kernel(const double* __restrict__ u, int n, double c, double cfl,
                                                        double theta, double* dt) {
    __shared__ unsigned long long red[32];
    unsigned long long mx = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const unsigned long long bb = abs_bits(wave_speed<EQ>(u[i], c));
        mx = bb > mx ? bb : mx;
    }
    const unsigned long long bm = block_max<unsigned long long>(mx, red);
    if (threadIdx.x == 0) *dt = theta * (cfl / from_bits(bm));
}

template <class T, int EQ, int REC, int FLUX>
__global__ void __launch_bounds__(kThreads) single_step_kernel(const T* __restrict__ u, T* __restrict__ uout,
                                                               int64_t n, int g, int tile, T dtdx,
                                                               OpParams<T> p, int32_t* err,
                                                               shk_boundary bcp, double dx) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar;
    constexpr int HL = step_halo<T>();
    Smem<T> sm;
    carve_step<T, REC, FLUX>(sm, smem_raw, tile + 2 * HL);
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    learned_stage<REC>(p.lp);
    uint32_t phase = 0;
    const int64_t s0 = int64_t(blockIdx.x) * tile;
    const int te = static_cast<int>(imin64(tile, n - s0));
    if (!load_window<T>(sm.U, u + g, n, s0 - HL, te + 2 * HL, &bar, phase)) {
        if (threadIdx.x == 0 && err) atomicOr(err, ERR_TIMEOUT);
        return;
    }
    const BcView bc = call_bc(bcp, dx);
    const Win<T> gout = make_win(uout, n + 2 * g);
    step_tile<T, EQ, REC, FLUX>(sm, gout + (g + s0), te, dtdx, p, bc, s0 - HL, n);
    __syncthreads();
    if (!bc.periodic()) return;  // ghosts: bc_ghost_kernel after the step
    // periodic ghost image of the new state
    for (int i = threadIdx.x; i < te; i += blockDim.x) {
        const int64_t gi = s0 + i;
        const T v = gout[g + gi];
        if (gi < g) gout[g + n + gi] = v;
        if (gi >= n - g) gout[gi - (n - g)] = v;
    }
}

}  // namespace shk

// ===========================================================================
// host side
// ===========================================================================
using namespace shk;

namespace {

cudaStream_t as_stream(void* s) { return static_cast<cudaStream_t>(s); }

int cuda_check(cudaError_t e) {
    if (e != cudaSuccess) {
        std::fprintf(stderr, "libshocks: CUDA error %s\n", cudaGetErrorString(e));
        return SHK_ECUDA;
    }
    return SHK_OK;
}
#define SHK_CUDA(call)                                  \
    do {                                                \
        int _st = cuda_check(call);                     \
        if (_st != SHK_OK) return _st;                  \
    } while (0)

// The library's tile when the caller gives none, by the plan's cells: long tiles
// waste the least on halos, short ones give a small batch more CTAs and a shorter
// step. Where the lines lie (us per step, or per forward + reverse step of plans
// that keep a dt history; 152 SMs):
//   integer fluxes, forward: 65 k cells 20.7 (tile 226) / 22.8 (466) / 28.9 (946);
//     442 k 50 / 39.8 / 43.2; 819 k 69 / 68 / 57 (706: 55.5); 4.1 M 253 / 221 / 213
//   Lax-Friedrichs stages: 131 k 39.6 / 41.6 / 48.2; 1.2 M 134 / 111 / 119
//   float32, forward: 65 k 10.7 (484) / 12.6 (2048); 819 k 22.8 / 16.7
//   learned, forward: 65 k 20.6 (512) / 26.9 (1024) / 41.0 (2048); 262 k 48 / 36.5 /
//     41; 3.3 M 279 / 255 / 240
//   with history: integer fluxes 65 k 92 (216) / 104 (448), 262 k 187 / 206, 819 k
//     429 / 403; float32 65 k 37.0 (512) / 42.3 (1024), 262 k 56 / 50; learned 65 k
//     74 (512) / 98 (1024), 262 k 161 / 130
// The integer-flux tiles are 60 faces (reverse: 58 cells) a warp in full rounds.
int default_tile(const shk_scheme* s, int dtype, int max_steps, int64_t cells) {
    const bool history = max_steps > 0;
    if (s->rec == SHK_REC_LEARNED) {
        if (cells <= 100000) return 512;
        return history || cells <= 500000 ? 1024 : 2048;
    }
    if (dtype == SHK_F64 && fixed_flux_scheme(s)) {
        if (history) return cells <= 400000 ? 216 : 448;
        return cells <= 140000 ? 226 : (cells <= 600000 ? 466 : (cells <= 3000000 ? 706 : 946));
    }
    if (dtype == SHK_F64 && fixed_flux_scheme(s, SHK_FLUX_LF))
        return cells <= 140000 ? 226 : (cells <= 2000000 ? 466 : 946);
    if (s->rec == SHK_REC_WENOJS53 && s->flux == SHK_FLUX_RUSANOV) {
        if (dtype == SHK_F32) return cells <= 120000 ? (history ? 512 : 484) : (history ? 1024 : 2048);
        return history ? 512 : kDefaultTile;
    }
    return kDefaultTile;
}

bool valid_scheme(const shk_scheme* s) {
    if (!s) return false;
    if (s->flux < 0 || s->flux > SHK_FLUX_EO) return false;
    if (s->rec < 0 || s->rec > SHK_REC_MUSCLS) return false;
    if (s->rec == SHK_REC_MUSCL || s->rec == SHK_REC_MUSCLS) {
        if (s->limiter < SHK_LIM_NONE || s->limiter > SHK_LIM_KOREN) return false;
        if (s->rec == SHK_REC_MUSCLS && s->limiter == SHK_LIM_KOREN) return false;  // no slope form
        if (s->limiter == SHK_LIM_MINMOD && !(s->delta >= 1.0 && s->delta <= 2.0)) return false;
        if (s->limiter == SHK_LIM_VANALBADA && s->delta != 1.0 && s->delta != 2.0) return false;
    }
    if (s->equation < 0 || s->equation > SHK_EQ_LWR) return false;
    if ((s->flux == SHK_FLUX_ESWENO) != (s->rec == SHK_REC_ESWENO32)) return false;
    if (s->rec == SHK_REC_LEARNED && (s->flux != SHK_FLUX_RUSANOV || !s->mlp)) return false;
    // the upwind and Engquist-Osher fluxes are the reference's Burgers schemes;
    // the constant and WENO-JS3 reconstructions run with Rusanov, Godunov or EO
    if ((s->flux == SHK_FLUX_GODUNOV || s->flux == SHK_FLUX_EO) &&
        (s->equation != SHK_EQ_BURGERS || s->rec == SHK_REC_LEARNED))
        return false;
    if ((s->rec == SHK_REC_CONSTANT || s->rec == SHK_REC_WENOJS32 || s->rec == SHK_REC_MUSCL ||
         s->rec == SHK_REC_MUSCLS) && s->flux == SHK_FLUX_LF)
        return false;
    return true;
}

shk_boundary periodic_boundary() {
    shk_boundary b;
    std::memset(&b, 0, sizeof(b));
    b.left = b.right = SHK_BC_PERIODIC;
    return b;
}

// both sides periodic, or each Dirichlet / Neumann
// cells a reconstruction reads on each side of a cell (the reference's
// stencil_width): the single-instance entry points need that many ghosts
int rec_reach(int rec) {
    switch (rec) {
        case SHK_REC_CONSTANT: return 1;
        case SHK_REC_WENOJS32:
        case SHK_REC_ESWENO32:
        case SHK_REC_MUSCL:
        case SHK_REC_MUSCLS: return 2;
        default: return 3;
    }
}

bool valid_boundary(const shk_boundary& b) {
    auto ok = [](int k) { return k >= SHK_BC_PERIODIC && k <= SHK_BC_NEUMANN; };
    if (!ok(b.left) || !ok(b.right)) return false;
    return (b.left == SHK_BC_PERIODIC) == (b.right == SHK_BC_PERIODIC);
}

template <class T>
OpParams<T> make_params(const shk_scheme* s) {
    OpParams<T> p;
    p.eps = static_cast<T>(s->eps);
    p.delta = static_cast<T>(s->delta);
    p.hnu = static_cast<T>(0.5 * s->nu);
    p.c = static_cast<T>(s->speed);
    p.hnu_amax = T(0);
    p.lim = s->limiter;
    p.lim_param = static_cast<T>(s->delta);
    p.atol = static_cast<T>(s->eps);
    p.dx = T(1);  // set per call / per instance
    p.lp = LearnedParams{s->mlp, static_cast<float>(s->eps), s->tau, s->band, s->dev,
                         norm_floor(s->norm_eps)};
    // FP64 Burgers-Rusanov with nu = 1 stores 4 F (see face_fluxes)
    p.fscale = (sizeof(T) == 8 && s->flux == SHK_FLUX_RUSANOV && s->rec == SHK_REC_WENOJS53 &&
                s->equation == SHK_EQ_BURGERS && s->nu == 1.0) ? T(0.25) : T(1);
    p.e4h = static_cast<float>(4.0 * s->eps);
    p.e4l = static_cast<float>(4.0 * s->eps - static_cast<double>(p.e4h));
    return p;
}

int sm_count() {
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 1;
    }
    return n;
}

// dispatch helpers: call F.template operator()<T, EQ, REC, FLUX>()
// Burgers with the Godunov / Engquist-Osher flux and a WENO-JS5, WENO-JS3 or
// constant reconstruction
template <class T, class F>
int dispatch_upwind(const shk_scheme* s, F&& f) {
    constexpr int EQ = SHK_EQ_BURGERS;
    if (s->flux == SHK_FLUX_GODUNOV) {
        if (s->rec == SHK_REC_MUSCL) return f.template operator()<T, EQ, SHK_REC_MUSCL, SHK_FLUX_GODUNOV>();
        if (s->rec == SHK_REC_MUSCLS) return f.template operator()<T, EQ, SHK_REC_MUSCLS, SHK_FLUX_GODUNOV>();
        if (s->rec == SHK_REC_CONSTANT) return f.template operator()<T, EQ, SHK_REC_CONSTANT, SHK_FLUX_GODUNOV>();
        if (s->rec == SHK_REC_WENOJS32) return f.template operator()<T, EQ, SHK_REC_WENOJS32, SHK_FLUX_GODUNOV>();
        return f.template operator()<T, EQ, SHK_REC_WENOJS53, SHK_FLUX_GODUNOV>();
    }
    if (s->rec == SHK_REC_MUSCL) return f.template operator()<T, EQ, SHK_REC_MUSCL, SHK_FLUX_EO>();
    if (s->rec == SHK_REC_MUSCLS) return f.template operator()<T, EQ, SHK_REC_MUSCLS, SHK_FLUX_EO>();
    if (s->rec == SHK_REC_CONSTANT) return f.template operator()<T, EQ, SHK_REC_CONSTANT, SHK_FLUX_EO>();
    if (s->rec == SHK_REC_WENOJS32) return f.template operator()<T, EQ, SHK_REC_WENOJS32, SHK_FLUX_EO>();
    return f.template operator()<T, EQ, SHK_REC_WENOJS53, SHK_FLUX_EO>();
}

template <class T, class F>
int dispatch_scheme(const shk_scheme* s, F&& f) {
    switch (s->equation) {
#define SHK_EQ_CASE(EQ)                                                                 \
    case EQ:                                                                            \
        if constexpr (EQ == SHK_EQ_BURGERS) {                                           \
            if (s->flux == SHK_FLUX_GODUNOV || s->flux == SHK_FLUX_EO)                  \
                return dispatch_upwind<T>(s, f);                                        \
        }                                                                               \
        if constexpr (EQ == SHK_EQ_BURGERS && sizeof(T) == 8) {                         \
            if (fixed_flux_scheme(s))                                                   \
                return f.template operator()<T, EQ, SHK_REC_WENOJS53, kFluxRusanovFx>(); \
        }                                                                               \
        if (s->rec == SHK_REC_CONSTANT)                                                 \
            return f.template operator()<T, EQ, SHK_REC_CONSTANT, SHK_FLUX_RUSANOV>();  \
        if (s->rec == SHK_REC_WENOJS32)                                                 \
            return f.template operator()<T, EQ, SHK_REC_WENOJS32, SHK_FLUX_RUSANOV>();  \
        if (s->rec == SHK_REC_MUSCL)                                                    \
            return f.template operator()<T, EQ, SHK_REC_MUSCL, SHK_FLUX_RUSANOV>();     \
        if (s->rec == SHK_REC_MUSCLS)                                                   \
            return f.template operator()<T, EQ, SHK_REC_MUSCLS, SHK_FLUX_RUSANOV>();    \
        if (s->rec == SHK_REC_LEARNED)                                                  \
            return f.template operator()<T, EQ, SHK_REC_LEARNED, SHK_FLUX_RUSANOV>();   \
        if (s->rec == SHK_REC_ESWENO32) return f.template operator()<T, EQ, SHK_REC_ESWENO32, SHK_FLUX_ESWENO>(); \
        if (s->flux == SHK_FLUX_LF) return f.template operator()<T, EQ, SHK_REC_WENOJS53, SHK_FLUX_LF>(); \
        return f.template operator()<T, EQ, SHK_REC_WENOJS53, SHK_FLUX_RUSANOV>();
        SHK_EQ_CASE(SHK_EQ_BURGERS)
        SHK_EQ_CASE(SHK_EQ_ADVECTION)
        SHK_EQ_CASE(SHK_EQ_LWR)
#undef SHK_EQ_CASE
    }
    return SHK_EINVAL;
}


// launch functors (namespace scope: member templates are not allowed in local classes)
struct ApplyOpLaunch {
    const double* u; double* out; int64_t n; int g; int tile; double dx; const double* amax;
    OpParams<double> p; size_t smem; int blocks; cudaStream_t st; shk_boundary bc;
    template <class T, int EQ, int REC, int FLUX> int operator()() {
        auto k = apply_operator_kernel<T, EQ, REC, FLUX == kFluxRusanovFx ? SHK_FLUX_RUSANOV : FLUX>;
        SHK_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k<<<blocks, kThreads, smem, st>>>(u, out, n, g, tile, dx, amax, p, nullptr, bc);
        return cuda_check(cudaGetLastError());
    }
};

struct SingleStepLaunch {
    const double* u; double* uo; int64_t n; int g; int tile; double dtdx;
    OpParams<double> p; size_t smem; int blocks; cudaStream_t st; shk_boundary bc; double dx;
    bool fixed;  // (of a scheme with a kFluxRusanovFx form)
    template <class T, int EQ, int REC, int FLUX> int operator()() {
        if constexpr (FLUX == SHK_FLUX_LF) {
            return SHK_EUNSUPPORTED;
        } else {
            auto k = single_step_kernel<T, EQ, REC, FLUX>;
            if constexpr (FLUX == kFluxRusanovFx)
                if (!fixed) k = single_step_kernel<T, EQ, REC, SHK_FLUX_RUSANOV>;
            SHK_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            k<<<blocks, kThreads, smem, st>>>(u, uo, n, g, tile, dtdx, p, nullptr, bc, dx);
            return cuda_check(cudaGetLastError());
        }
    }
};

template <class TS>
struct BatchedStepLaunch {
    PlanDev D; const TS* uin; TS* uout; OpParams<TS> p; size_t smem; int grid; cudaStream_t st;
    template <class T, int EQ, int REC, int FLUX> int operator()() {
        if constexpr (FLUX == SHK_FLUX_LF) {
            return SHK_EUNSUPPORTED;
        } else {
            auto k = batched_step_kernel<T, EQ, REC, FLUX>;
            SHK_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            k<<<grid, flux_threads<FLUX>(), smem, st>>>(D, uin, uout, p);
            return cuda_check(cudaGetLastError());
        }
    }
};

// the schemes with a resident form
template <class T, int EQ, int REC, int FLUX>
constexpr bool kHasResident = FLUX == kFluxRusanovFx ||
                              (sizeof(T) == 4 && REC == SHK_REC_WENOJS53 && FLUX == SHK_FLUX_RUSANOV);
inline bool resident_scheme(const shk_scheme* s, int dtype) {
    return dtype == SHK_F64 ? fixed_flux_scheme(s)
                            : s->rec == SHK_REC_WENOJS53 && s->flux == SHK_FLUX_RUSANOV;
}
template <class TS>
struct ResidentLaunch {
    PlanDev D; const TS* uin; TS* ucur; TS* uprev; OpParams<TS> p; size_t smem; int threads; int W;
    int nsteps; cudaStream_t st;
    template <class T, int EQ, int REC, int FLUX> int operator()() {
        if constexpr (!kHasResident<T, EQ, REC, FLUX>) {
            return SHK_EUNSUPPORTED;
        } else {
            auto k = resident_steps_kernel<T, EQ, REC, FLUX>;
            SHK_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            k<<<D.B, threads, smem, st>>>(D, uin, ucur, uprev, p, W, nsteps);
            return cuda_check(cudaGetLastError());
        }
    }
};

// one global Lax-Friedrichs step of a plan: the three stage launches
struct BatchedLfLaunch {
    PlanDev D; const double* uin; double* uout; double* k1; double* k2; unsigned long long* amax_lf;
    OpParams<double> p; size_t smem; int grid; cudaStream_t st;
    template <int EQ, bool FX = false> int run() {
        constexpr int kThr = FX ? kFxThreads : kThreads;
        auto s1 = batched_lf_stage_kernel<EQ, 1, FX>;
        auto s2 = batched_lf_stage_kernel<EQ, 2, FX>;
        auto s3 = batched_lf_stage_kernel<EQ, 3, FX>;
        for (auto k : {s1, s2, s3})
            SHK_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        const int B = D.B;
        s1<<<grid, kThr, smem, st>>>(D, uin, uin, k1, nullptr, amax_lf, amax_lf, p);
        SHK_CUDA(cudaGetLastError());
        s2<<<grid, kThr, smem, st>>>(D, uin, k1, k2, amax_lf, amax_lf + B, amax_lf, p);
        SHK_CUDA(cudaGetLastError());
        s3<<<grid, kThr, smem, st>>>(D, uin, k2, uout, amax_lf + B, nullptr, amax_lf, p);
        return cuda_check(cudaGetLastError());
    }
};

// resident CTAs per SM of the step kernel a scheme dispatches to, at the
// given dynamic shared memory (registers and shared memory both counted)
struct StepOccupancy {
    size_t smem; int* out; bool fixed;  // fixed: a Lax-Friedrichs plan on fixed_flux.cuh
    template <class T, int EQ, int REC, int FLUX> int operator()() {
        if constexpr (FLUX == SHK_FLUX_LF) {
            if constexpr (sizeof(T) != 8) {
                return SHK_EUNSUPPORTED;
            } else {
                auto k = batched_lf_stage_kernel<EQ, 2, false>;
                if constexpr (EQ == SHK_EQ_BURGERS)
                    if (fixed) k = batched_lf_stage_kernel<EQ, 2, true>;
                SHK_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
                SHK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(out, k, fixed ? kFxThreads : kThreads, smem));
                return SHK_OK;
            }
        } else {
            auto k = batched_step_kernel<T, EQ, REC, FLUX>;
            SHK_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            SHK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(out, k, flux_threads<FLUX>(), smem));
            return SHK_OK;
        }
    }
};

}  // namespace

struct shk_plan {
    shk_scheme scheme;
    int dtype = SHK_F64;
    int B = 0, tile = 0, nitems = 0, max_steps = 0, grid = 0;
    int64_t total_cells = 0;
    double theta = 1.0;
    // device buffers
    int32_t* item_inst = nullptr;
    int32_t* item_tile = nullptr;
    int32_t* item_first = nullptr;
    int64_t* offsets = nullptr;
    double* cfl = nullptr;
    double* inv_dx = nullptr;
    double* tfinal = nullptr;
    unsigned long long* amax = nullptr;
    double* t = nullptr;
    double* dt_hist = nullptr;
    int64_t* step = nullptr;
    unsigned int* done = nullptr;
    int32_t* status = nullptr;
    double* partial = nullptr;
    double* dt_fixed = nullptr;  // prescribed steps [fixed_cap][B], active when fixed_steps > 0
    int64_t fixed_cap = 0, fixed_steps = 0;
    int bc_left = SHK_BC_PERIODIC, bc_right = SHK_BC_PERIODIC;
    double* bc_dir = nullptr;  // [B][2][3]
    double* bc_neu = nullptr;  // [B][2], or per-step [bc_steps][3][B][2]
    int64_t bc_steps = 0;      // 0: time-independent boundary data
    size_t bc_dir_cap = 0, bc_neu_cap = 0;  // doubles allocated
    PlanItem* items = nullptr;  // [nitems] longest first
    unsigned int* left = nullptr;  // [B] finished tiles of the running step
    unsigned int* sched = nullptr;  // [8] scheduling counters
    // host mirror of the number of steps launched since reset
    int64_t host_steps = 0;
    // global Lax-Friedrichs plans: stage states k1, k2 and their maxima [2][B]
    double* lf_k1 = nullptr;
    double* lf_k2 = nullptr;
    unsigned long long* amax_lf = nullptr;
    // all steps of a call in one launch, one CTA per instance: its threads (0: no)
    // and window length
    int resident = 0, resident_W = 0;
    bool too_long = false;  // tile beyond the FP64 formula's layout (see shk_plan_create)
    // captured two-step graph
    cudaGraphExec_t graph = nullptr;
    void* graph_a = nullptr;
    void* graph_b = nullptr;

    PlanDev dev() const {
        PlanDev P;
        P.item_inst = item_inst; P.item_tile = item_tile; P.offsets = offsets; P.cfl = cfl;
        P.inv_dx = inv_dx; P.tfinal = tfinal; P.theta = theta; P.amax = amax; P.t = t;
        P.dt_hist = dt_hist; P.step = step; P.done = done; P.status = status;
        P.partial = partial; P.B = B;
        P.dt_fixed = fixed_steps > 0 ? dt_fixed : nullptr; P.fixed_steps = fixed_steps;
        P.bc_left = bc_left; P.bc_right = bc_right; P.bc_dir = bc_dir; P.bc_neu = bc_neu; P.nitems = nitems; P.tile = tile; P.max_steps = max_steps;
        P.items = items; P.left = left; P.sched = sched; P.bc_steps = bc_steps;
        return P;
    }
};

namespace {
template <class T>
int launch_max(shk_plan* P, const void* u, int slot, cudaStream_t st) {
    const PlanDev D = P->dev();
    const T c = static_cast<T>(P->scheme.speed);
    const T* uu = static_cast<const T*>(u);
    const int grid = std::min(P->nitems, 8 * sm_count());
    switch (P->scheme.equation) {
        case SHK_EQ_BURGERS: batched_max_kernel<T, SHK_EQ_BURGERS><<<grid, kThreads, 0, st>>>(D, uu, c, slot); break;
        case SHK_EQ_ADVECTION: batched_max_kernel<T, SHK_EQ_ADVECTION><<<grid, kThreads, 0, st>>>(D, uu, c, slot); break;
        default: batched_max_kernel<T, SHK_EQ_LWR><<<grid, kThreads, 0, st>>>(D, uu, c, slot); break;
    }
    return cuda_check(cudaGetLastError());
}

constexpr size_t kStepStatic = 312;  // static shared memory of the FP64 formula's step

template <class T>
int launch_step(shk_plan* P, const void* uin, void* uout, cudaStream_t st) {
    if (P->too_long) return SHK_ECUDA;
    const PlanDev D = P->dev();
    if (P->scheme.flux == SHK_FLUX_LF) {
        if constexpr (sizeof(T) != 8) {
            return SHK_EUNSUPPORTED;
        } else {
            const bool fixed = fixed_flux_scheme(&P->scheme, SHK_FLUX_LF);
            const size_t smem = Smem<double>::lf_stage_bytes(P->tile + 2 * op_halo<double>(), fixed);
            BatchedLfLaunch f{D, static_cast<const double*>(uin), static_cast<double*>(uout), P->lf_k1,
                              P->lf_k2, P->amax_lf, make_params<double>(&P->scheme), smem, P->grid, st};
            switch (P->scheme.equation) {
                case SHK_EQ_BURGERS: return fixed ? f.run<SHK_EQ_BURGERS, true>() : f.run<SHK_EQ_BURGERS>();
                case SHK_EQ_ADVECTION: return f.run<SHK_EQ_ADVECTION>();
                default: return f.run<SHK_EQ_LWR>();
            }
        }
    }
    const size_t smem = Smem<T>::step_bytes(P->tile + 2 * step_halo<T>(), P->scheme.rec, fixed_flux_scheme(&P->scheme));
    OpParams<T> p = make_params<T>(&P->scheme);
    BatchedStepLaunch<T> f{D, static_cast<const T*>(uin), static_cast<T*>(uout), p, smem, P->grid, st};
    return dispatch_scheme<T>(&P->scheme, f);
}
}  // namespace

namespace {
// most steps of one resident launch (some 10 ms): nothing can stop a kernel
constexpr int kResidentSteps = 512;
// steps of a resident plan (see shk_plan_create)
template <class T>
int launch_resident(shk_plan* P, void* u_a, void* u_b, int nsteps, cudaStream_t st) {
    const bool even = P->host_steps % 2 == 0, even_end = (P->host_steps + nsteps) % 2 == 0;
    T* cur = static_cast<T*>(even_end ? u_a : u_b);
    T* prev = static_cast<T*>(even_end ? u_b : u_a);
    const size_t smem = Smem<T>::step_bytes(P->resident_W, P->scheme.rec, fixed_flux_scheme(&P->scheme));
    ResidentLaunch<T> f{P->dev(), static_cast<const T*>(even ? u_a : u_b), cur, prev,
                        make_params<T>(&P->scheme), smem, P->resident, P->resident_W, nsteps, st};
    return dispatch_scheme<T>(&P->scheme, f);
}
}  // namespace

namespace shk {
int plan_view(shk_plan* plan, PlanDev* dev, int* dtype, int* grid, shk_scheme* scheme,
              int64_t* total_cells, int64_t* host_steps) {
    if (!plan) return SHK_EINVAL;
    if (host_steps) *host_steps = plan->host_steps;
    *dev = plan->dev();
    *dtype = plan->dtype;
    *grid = plan->grid;
    *scheme = plan->scheme;
    *total_cells = plan->total_cells;
    return SHK_OK;
}
}  // namespace shk

extern "C" {

const char* shk_strerror(int status) {
    switch (status) {
        case SHK_OK: return "ok";
        case SHK_EINVAL: return "invalid argument";
        case SHK_ENONFINITE: return "Time step is not finite";
        case SHK_ETIMEOUT: return "bounded device wait expired";
        case SHK_ECUDA: return "CUDA runtime error";
        case SHK_ENOMEM: return "out of device memory";
        case SHK_EUNSUPPORTED: return "unsupported scheme combination";
        case SHK_ETOOLARGE: return "size exceeds the static scratch of the no-allocation entry point";
        default: return "unknown status";
    }
}

int shk_version(void) { return 1; }

int shk_max_wavespeed_f64(const shk_scheme* scheme, const double* u, int64_t n, int32_t nghosts,
                          double* amax, void* stream) {
    // only the wave speed of the equation matters here (any flux and
    // reconstruction, e.g. Lax-Friedrichs with the constant reconstruction)
    if (!scheme || scheme->equation < SHK_EQ_BURGERS || scheme->equation > SHK_EQ_LWR || !u || !amax ||
        n <= 0 || nghosts < 0)
        return SHK_EINVAL;
    cudaStream_t st = as_stream(stream);
    SHK_CUDA(cudaMemsetAsync(amax, 0, sizeof(double), st));
    const int blocks = static_cast<int>(imin64((n + kThreads - 1) / kThreads, 4 * sm_count()));
    const double c = scheme->speed;
    auto* out = reinterpret_cast<unsigned long long*>(amax);
    switch (scheme->equation) {
        case SHK_EQ_BURGERS: max_wavespeed_kernel<double, SHK_EQ_BURGERS><<<blocks, kThreads, 0, st>>>(u + nghosts, n, c, out); break;
        case SHK_EQ_ADVECTION: max_wavespeed_kernel<double, SHK_EQ_ADVECTION><<<blocks, kThreads, 0, st>>>(u + nghosts, n, c, out); break;
        default: max_wavespeed_kernel<double, SHK_EQ_LWR><<<blocks, kThreads, 0, st>>>(u + nghosts, n, c, out); break;
    }
    return cuda_check(cudaGetLastError());
}

int shk_apply_operator_bc_f64(const shk_scheme* scheme, const shk_boundary* bc, const double* u,
                              double* out, int64_t n, int32_t nghosts, double dx,
                              const double* amax, void* stream) {
    if (!valid_scheme(scheme) || !u || !out || n < 3 || nghosts < rec_reach(scheme->rec) || !(dx > 0))
        return SHK_EINVAL;
    if (scheme->flux == SHK_FLUX_LF && !amax) return SHK_EINVAL;
    const shk_boundary b = bc ? *bc : periodic_boundary();
    if (!valid_boundary(b)) return SHK_EINVAL;
    cudaStream_t st = as_stream(stream);
    const int tile = 512;
    const int W = tile + 2 * op_halo<double>();
    const size_t smem = Smem<double>::host_bytes(W);
    const int blocks = static_cast<int>((n + tile - 1) / tile);
    OpParams<double> p = make_params<double>(scheme);
    p.dx = dx;
    ApplyOpLaunch f{u, out, n, nghosts, tile, dx, amax, p, smem, blocks, st, b};
    const int r = dispatch_scheme<double>(scheme, f);
    if (r != SHK_OK || (b.left == SHK_BC_PERIODIC && b.right == SHK_BC_PERIODIC)) return r;
    bc_ghost_kernel<double><<<1, 64, 0, st>>>(out, n, nghosts, b, dx, 0, 1);
    return cuda_check(cudaGetLastError());
}

int shk_apply_operator_f64(const shk_scheme* scheme, const double* u, double* out, int64_t n,
                           int32_t nghosts, double dx, const double* amax, void* stream) {
    return shk_apply_operator_bc_f64(scheme, nullptr, u, out, n, nghosts, dx, amax, stream);
}

int shk_predict_timestep_f64(const shk_scheme* scheme, const double* u, int64_t n, int32_t nghosts,
                             double cfl, double theta, double* dt, void* stream) {
    if (scheme && u && dt && n > 0 && n <= kBlockDtCells && nghosts >= 0 && scheme->equation >= SHK_EQ_BURGERS &&
        scheme->equation <= SHK_EQ_LWR) {
        const int m = static_cast<int>(n), threads = static_cast<int>(std::min<int64_t>(1024, (n + 31) / 32 * 32));
        const double* v = u + nghosts;
        const double c = scheme->speed;
        cudaStream_t s = as_stream(stream);
        switch (scheme->equation) {
            case SHK_EQ_BURGERS: block_dt_kernel<SHK_EQ_BURGERS><<<1, threads, 0, s>>>(v, m, c, cfl, theta, dt); break;
            case SHK_EQ_ADVECTION: block_dt_kernel<SHK_EQ_ADVECTION><<<1, threads, 0, s>>>(v, m, c, cfl, theta, dt); break;
            default: block_dt_kernel<SHK_EQ_LWR><<<1, threads, 0, s>>>(v, m, c, cfl, theta, dt); break;
        }
        return cuda_check(cudaGetLastError());
    }
    int st = shk_max_wavespeed_f64(scheme, u, n, nghosts, dt, stream);
    if (st != SHK_OK) return st;
    finalize_dt_kernel<<<1, 1, 0, as_stream(stream)>>>(dt, cfl, theta);
    return cuda_check(cudaGetLastError());
}

// longest array that the single step leaves to the FP64 formula: on the coarsest grids
// most faces are left to FP64 anyhow (us, FP64 formula / fixed fluxes, smooth and random
// states: 64 cells 12.4 / 14.3, 20.8; 96 12.6 / 14.5, 20.8; 128 14.6 / 13.5, 20.8; 192
// 16.6 / 8.4, 20.8; 256 26.9 / 8.5, 22.7)
static constexpr int64_t kFxStepCells = 96;

int shk_ssprk33_step_bc_f64(const shk_scheme* scheme, const shk_boundary* bc, const double* u,
                            double* u_out, int64_t n, int32_t nghosts, double dx, double dt,
                            void* stream) {
    if (!valid_scheme(scheme) || !u || !u_out || n < 3 || nghosts < rec_reach(scheme->rec) || !(dx > 0))
        return SHK_EINVAL;
    if (!std::isfinite(dt)) return SHK_ENONFINITE;
    if (scheme->flux == SHK_FLUX_LF) return SHK_EUNSUPPORTED;  // global max per stage
    const shk_boundary b = bc ? *bc : periodic_boundary();
    if (!valid_boundary(b)) return SHK_EINVAL;
    cudaStream_t st = as_stream(stream);
    // fixed fluxes: 8 warps x 60 faces cover a tile and its first stage's halo
    const bool fixed = fixed_flux_scheme(scheme) && n > kFxStepCells;
    const int tile = fixed ? 466 : 512;
    const int W = tile + 2 * step_halo<double>();
    const size_t smem = Smem<double>::step_bytes(W, scheme->rec, fixed);
    const int blocks = static_cast<int>((n + tile - 1) / tile);
    OpParams<double> p = make_params<double>(scheme);
    p.dx = dx;
    SingleStepLaunch f{u, u_out, n, nghosts, tile, dt / dx, p, smem, blocks, st, b, dx, fixed};
    const int r = dispatch_scheme<double>(scheme, f);
    if (r != SHK_OK || (b.left == SHK_BC_PERIODIC && b.right == SHK_BC_PERIODIC)) return r;
    bc_ghost_kernel<double><<<1, 64, 0, st>>>(u_out, n, nghosts, b, dx, 1, 0);
    return cuda_check(cudaGetLastError());
}

int shk_ssprk33_step_f64(const shk_scheme* scheme, const double* u, double* u_out, int64_t n,
                         int32_t nghosts, double dx, double dt, void* stream) {
    return shk_ssprk33_step_bc_f64(scheme, nullptr, u, u_out, n, nghosts, dx, dt, stream);
}

// ---------------------------------------------------------------------------
// plans
// ---------------------------------------------------------------------------
int shk_plan_destroy(shk_plan* plan) {
    if (!plan) return SHK_OK;
    if (plan->graph) cudaGraphExecDestroy(plan->graph);
    void* ptrs[] = {plan->item_inst, plan->item_tile, plan->item_first, plan->offsets, plan->cfl,
                    plan->inv_dx, plan->tfinal, plan->amax, plan->t, plan->dt_hist, plan->step,
                    plan->done, plan->status, plan->partial, plan->dt_fixed, plan->bc_dir,
                    plan->bc_neu, plan->items, plan->left, plan->sched, plan->lf_k1, plan->lf_k2,
                    plan->amax_lf};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    delete plan;
    return SHK_OK;
}

int shk_plan_create(const shk_scheme* scheme, int32_t batch, const int64_t* h_offsets,
                    const double* h_dx, const double* h_cfl, double theta,
                    const shk_plan_opts* opts, shk_plan** out) {
    if (!out) return SHK_EINVAL;
    *out = nullptr;
    if (!valid_scheme(scheme) || batch <= 0 || !h_offsets || !h_dx || !h_cfl) return SHK_EINVAL;
    const int dtype = opts ? opts->dtype : SHK_F64;
    if (dtype != SHK_F64 && dtype != SHK_F32) return SHK_EINVAL;
    // global Lax-Friedrichs: float64 stage states kept between the stage launches
    const bool lf = scheme->flux == SHK_FLUX_LF;
    if (lf && dtype != SHK_F64) return SHK_EUNSUPPORTED;
    int tile = (opts && opts->tile > 0) ? opts->tile : default_tile(scheme, dtype, opts ? opts->max_steps : 0,
                                                                  h_offsets[batch] - h_offsets[0]);
    const int align = dtype == SHK_F64 ? 2 : 4;
    if (tile % align || tile < 16 || tile > 8192) return SHK_EINVAL;
    // the learned phase's warp scratch lives in the window's free arrays
    if (scheme->rec == SHK_REC_LEARNED && tile < kLearnedMinTile) return SHK_EINVAL;
    std::vector<int32_t> inst, tl, first(batch + 1, 0);
    for (int b = 0; b < batch; ++b) {
        const int64_t n = h_offsets[b + 1] - h_offsets[b];
        if (n < 3 || !(h_dx[b] > 0)) return SHK_EINVAL;
        const int64_t ntiles = (n + tile - 1) / tile;
        first[b] = static_cast<int32_t>(inst.size());
        for (int64_t j = 0; j < ntiles; ++j) {
            inst.push_back(b);
            tl.push_back(static_cast<int32_t>(j));
        }
    }
    first[batch] = static_cast<int32_t>(inst.size());
    // scheduling order: longest items first (full tiles, then partial tiles
    // by decreasing length), ties in packing order
    std::vector<int32_t> order(inst.size());
    std::vector<int64_t> len(inst.size());
    for (size_t i = 0; i < inst.size(); ++i) {
        order[i] = static_cast<int32_t>(i);
        const int64_t n = h_offsets[inst[i] + 1] - h_offsets[inst[i]];
        len[i] = std::min<int64_t>(tile, n - int64_t(tl[i]) * tile);
    }
    std::stable_sort(order.begin(), order.end(), [&](int32_t x, int32_t y) { return len[x] > len[y]; });
    std::vector<PlanItem> items(inst.size());
    for (size_t q = 0; q < order.size(); ++q) {
        const int32_t i = order[q], b = inst[i];
        items[q] = PlanItem{h_offsets[b], h_offsets[b + 1] - h_offsets[b], b, static_cast<int32_t>(len[i]),
                            tl[i], first[b + 1] - first[b]};
    }
    auto* P = new (std::nothrow) shk_plan();
    if (!P) return SHK_ENOMEM;
    P->scheme = *scheme;
    P->dtype = dtype;
    P->B = batch;
    P->tile = tile;
    P->nitems = static_cast<int>(inst.size());
    P->max_steps = opts ? std::max(0, opts->max_steps) : 0;
    P->theta = theta;
    P->total_cells = h_offsets[batch] - h_offsets[0];
    std::vector<double> inv(batch), inf(batch, DBL_MAX);
    for (int b = 0; b < batch; ++b) inv[b] = 1.0 / h_dx[b];
    auto alloc = [&](void** p, size_t bytes) { return cudaMalloc(p, bytes) == cudaSuccess; };
    bool ok = alloc((void**)&P->item_inst, sizeof(int32_t) * P->nitems) &&
              alloc((void**)&P->item_tile, sizeof(int32_t) * P->nitems) &&
              alloc((void**)&P->item_first, sizeof(int32_t) * (batch + 1)) &&
              alloc((void**)&P->offsets, sizeof(int64_t) * (batch + 1)) &&
              alloc((void**)&P->cfl, sizeof(double) * batch) &&
              alloc((void**)&P->inv_dx, sizeof(double) * batch) &&
              alloc((void**)&P->tfinal, sizeof(double) * batch) &&
              alloc((void**)&P->amax, sizeof(unsigned long long) * 2 * batch) &&
              alloc((void**)&P->t, sizeof(double) * batch) &&
              alloc((void**)&P->step, sizeof(int64_t)) && alloc((void**)&P->done, sizeof(unsigned)) &&
              alloc((void**)&P->status, sizeof(int32_t)) &&
              alloc((void**)&P->partial, sizeof(double) * P->nitems) &&
              alloc((void**)&P->items, sizeof(PlanItem) * P->nitems) &&
              alloc((void**)&P->left, sizeof(unsigned) * batch) &&
              alloc((void**)&P->sched, sizeof(unsigned) * 8);
    if (ok && P->max_steps > 0)
        ok = alloc((void**)&P->dt_hist, sizeof(double) * size_t(P->max_steps) * batch);
    if (ok && lf)
        ok = alloc((void**)&P->lf_k1, sizeof(double) * size_t(P->total_cells)) &&
             alloc((void**)&P->lf_k2, sizeof(double) * size_t(P->total_cells)) &&
             alloc((void**)&P->amax_lf, sizeof(unsigned long long) * 2 * batch) &&
             cudaMemset(P->amax_lf, 0, sizeof(unsigned long long) * 2 * batch) == cudaSuccess;
    if (!ok) {
        shk_plan_destroy(P);
        return SHK_ENOMEM;
    }
    ok = cudaMemcpy(P->item_inst, inst.data(), sizeof(int32_t) * P->nitems, cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemcpy(P->item_tile, tl.data(), sizeof(int32_t) * P->nitems, cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemcpy(P->items, items.data(), sizeof(PlanItem) * P->nitems, cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemset(P->left, 0, sizeof(unsigned) * batch) == cudaSuccess &&
         cudaMemset(P->sched, 0, sizeof(unsigned) * 8) == cudaSuccess &&
         cudaMemcpy(P->item_first, first.data(), sizeof(int32_t) * (batch + 1), cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemcpy(P->offsets, h_offsets, sizeof(int64_t) * (batch + 1), cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemcpy(P->cfl, h_cfl, sizeof(double) * batch, cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemcpy(P->inv_dx, inv.data(), sizeof(double) * batch, cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemcpy(P->tfinal, inf.data(), sizeof(double) * batch, cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemset(P->amax, 0, sizeof(unsigned long long) * 2 * batch) == cudaSuccess &&
         cudaMemset(P->t, 0, sizeof(double) * batch) == cudaSuccess &&
         cudaMemset(P->step, 0, sizeof(int64_t)) == cudaSuccess &&
         cudaMemset(P->done, 0, sizeof(unsigned)) == cudaSuccess &&
         cudaMemset(P->status, 0, sizeof(int32_t)) == cudaSuccess;
    if (!ok) {
        shk_plan_destroy(P);
        return SHK_ECUDA;
    }
    // The integer-flux layouts are shorter than the FP64 formula's, but which tiles a
    // plan takes does not depend on eps or nu: a tile beyond that formula's layout is
    // refused (here, or by the step where the caller names the CTAs)
    const bool fixed_lf = fixed_flux_scheme(scheme, SHK_FLUX_LF);
    int per_sm = opts && opts->ctas_per_sm > 0 ? opts->ctas_per_sm : 0;
    if (dtype == SHK_F64 && (fixed_lf || fixed_flux_scheme(scheme))) {
        const size_t bytes = lf ? Smem<double>::lf_stage_bytes(tile + 2 * op_halo<double>(), false)
                                : Smem<double>::step_bytes(tile + 2 * step_halo<double>(), scheme->rec);
        int dev = 0, optin = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        P->too_long = bytes + kStepStatic > static_cast<size_t>(optin);
        if (P->too_long && per_sm == 0) {
            shk_plan_destroy(P);
            return SHK_EINVAL;
        }
    }
    // persistent grid: resident CTAs per SM x SMs
    if (per_sm == 0) {
        const size_t smem = lf ? Smem<double>::lf_stage_bytes(tile + 2 * op_halo<double>(), fixed_lf)
                               : (dtype == SHK_F64 ? Smem<double>::step_bytes(tile + 2 * step_halo<double>(), scheme->rec, fixed_flux_scheme(scheme))
                                                   : Smem<float>::step_bytes(tile + 2 * step_halo<float>(), scheme->rec));
        int resident = 0;
        const int r = dtype == SHK_F64 ? dispatch_scheme<double>(scheme, StepOccupancy{smem, &resident, fixed_lf})
                                       : dispatch_scheme<float>(scheme, StepOccupancy{smem, &resident, fixed_lf});
        if (r != SHK_OK || resident < 1) {
            shk_plan_destroy(P);
            return r != SHK_OK ? r : SHK_EINVAL;  // the window does not fit one SM
        }
        per_sm = std::min(resident, 8);
    }
    P->grid = std::max(1, std::min(P->nitems, per_sm * sm_count()));
    // Resident steps where every instance can have a CTA at once (so no instance
    // waits for another's steps) and is short enough for one: up to 1536 cells a
    // CTA of its share of an SM's 32 warps needs at most two rounds of 60 faces a
    // warp where an SM has one or two; longer instances are faster spread over several
    // SMs. A caller that names a launch shape gets that shape. Four warps at least: each
    // quarter of an SM has its own FP64 pipe (24 instances of 32 cells, where nearly all
    // faces are left to FP64: 20.0 us a step with one warp, 12.0 with four; FP64 formula,
    // launched: 16.6). Double states, whose steps are long, stay launched where most of
    // the cells (`bulk`, the mean length of a cell's instance) lie in instances that take
    // several rounds while the others' CTAs idle. Us per step of a call of ten, resident /
    // launched, by instances per SM:
    //   all 1000 cells (bulk / mean length 1.0): 1 15 / 21, 2 23 / 29, 3 29 / 40, 5 43 / 59
    //   uniform 100 to 1536 (1.25): 2 29 / 32, 3 37 / 36, 4 42 / 44, 5 50 / 54
    //   logarithmic 300 to 1536 (1.21): 2 29 / 29, 3 39 / 35, 4 43 / 40, 5 54 / 49
    //   logarithmic 100 to 600 (1.26): 1 15 / 25, 3 20 / 30, 5 27 / 34, 8 35 / 49
    //   logarithmic 100 to 1536 (1.57): 1 20 / 27, 2 28 / 29, 3 38 / 33, 4 40 / 36, 5 48 / 42
    //   half 200, half 1500 (1.58): 1 20 / 23, 2 31 / 28, 3 42 / 36, 5 61 / 52
    //   a tenth 1500, the others 200 (2.4): 1 20 / 21, 2 22 / 23, 3 36 / 25, 5 43 / 31
    //   one 1536, the others 100 (1.3 to 2.1): 1 22 / 28, 3 27 / 31, 5 33 / 41
    if (!(opts && (opts->tile > 0 || opts->ctas_per_sm > 0)) && resident_scheme(scheme, dtype)) {
        int64_t nmax = 0;
        double cells = 0.0, squares = 0.0;
        for (int b = 0; b < batch; ++b) {
            const int64_t n = h_offsets[b + 1] - h_offsets[b];
            nmax = std::max(nmax, n);
            cells += double(n);
            squares += double(n) * double(n);
        }
        const int share = (batch + sm_count() - 1) / sm_count();
        if (nmax <= 1536 && share <= 8) {
            const int W = static_cast<int>((nmax + 3) / 4 * 4) +
                          2 * (dtype == SHK_F64 ? step_halo<double>() : step_halo<float>());
            const size_t smem = dtype == SHK_F64 ? Smem<double>::step_bytes(W, scheme->rec, true)
                                                 : Smem<float>::step_bytes(W, scheme->rec);
            const int warps = std::min<int>(std::max<int>(4, static_cast<int>((nmax + 14 + 59) / 60)), 32 / share);
            const double bulk = squares / cells, mean = cells / batch;
            const bool idle = dtype == SHK_F64 && bulk + 14 > 60 * warps && bulk > 1.3 * mean;
            if (share * (smem + 2048) <= size_t(227) * 1024 && !idle) {
                P->resident = 32 * std::max(1, warps);
                P->resident_W = W;
            }
        }
    }
    *out = P;
    return SHK_OK;
}

int shk_plan_state(shk_plan* plan, double** t, double** dt_hist, int64_t** step_counter) {
    if (!plan) return SHK_EINVAL;
    if (t) *t = plan->t;
    if (dt_hist) *dt_hist = plan->dt_hist;
    if (step_counter) *step_counter = plan->step;
    return SHK_OK;
}

int shk_plan_copy_time(shk_plan* plan, double* t_out, void* stream) {
    if (!plan || !t_out) return SHK_EINVAL;
    return cuda_check(cudaMemcpyAsync(t_out, plan->t, sizeof(double) * plan->B,
                                      cudaMemcpyDeviceToDevice, as_stream(stream)));
}

int shk_plan_copy_dt_history(shk_plan* plan, double* out, void* stream) {
    if (!plan || !out || !plan->dt_hist) return SHK_EINVAL;
    return cuda_check(cudaMemcpyAsync(out, plan->dt_hist,
                                      sizeof(double) * size_t(plan->max_steps) * plan->B,
                                      cudaMemcpyDeviceToDevice, as_stream(stream)));
}

int shk_plan_status(shk_plan* plan, int32_t* h_status, void* stream) {
    if (!plan || !h_status) return SHK_EINVAL;
    SHK_CUDA(cudaMemcpyAsync(h_status, plan->status, sizeof(int32_t), cudaMemcpyDeviceToHost,
                             as_stream(stream)));
    SHK_CUDA(cudaStreamSynchronize(as_stream(stream)));
#ifdef SHOCKS_BOUNDS_CHECK
    // the bounds-check build also reports a recorded out-of-bounds index
    int32_t flag = 0;
    const int r = shk_check_bounds(0, &flag, nullptr, nullptr, nullptr, nullptr);
    if (r != SHK_OK) return r;
    if (flag) *h_status |= ERR_BOUNDS;
#endif
    return SHK_OK;
}


int shk_plan_reset(shk_plan* plan, const void* u, const double* t0, const double* tfinal,
                   void* stream) {
    if (!plan || !u) return SHK_EINVAL;
    cudaStream_t st = as_stream(stream);
    const int B = plan->B;
    const int threads = std::max(8, 2 * B);
    reset_kernel<<<(threads + kThreads - 1) / kThreads, kThreads, 0, st>>>(plan->dev(), plan->amax_lf, plan->tfinal,
                                                                         t0, tfinal);
    SHK_CUDA(cudaGetLastError());
    if (plan->dt_hist)
        SHK_CUDA(cudaMemsetAsync(plan->dt_hist, 0, sizeof(double) * size_t(plan->max_steps) * B, st));
    plan->host_steps = 0;
    return plan->dtype == SHK_F64 ? launch_max<double>(plan, u, 0, st) : launch_max<float>(plan, u, 0, st);
}

int shk_plan_step(shk_plan* plan, void* u_a, void* u_b, int32_t nsteps, void* stream) {
    if (!plan || !u_a || !u_b || u_a == u_b || nsteps < 0) return SHK_EINVAL;
    cudaStream_t st = as_stream(stream);
    if (plan->resident) {
        while (nsteps > 0) {
            const int k = std::min(nsteps, kResidentSteps);
            const int r = plan->dtype == SHK_F64 ? launch_resident<double>(plan, u_a, u_b, k, st)
                                                 : launch_resident<float>(plan, u_a, u_b, k, st);
            if (r != SHK_OK) return r;
            plan->host_steps += k;
            nsteps -= k;
        }
        return SHK_OK;
    }
    for (int i = 0; i < nsteps; ++i) {
        const bool even = (plan->host_steps % 2) == 0;
        void* in = even ? u_a : u_b;
        void* out = even ? u_b : u_a;
        const int r = plan->dtype == SHK_F64 ? launch_step<double>(plan, in, out, st)
                                             : launch_step<float>(plan, in, out, st);
        if (r != SHK_OK) return r;
        plan->host_steps++;
    }
    return SHK_OK;
}

int shk_plan_set_fixed_dt(shk_plan* plan, const double* dt, int32_t nsteps, void* stream) {
    if (!plan || nsteps < 0 || (nsteps > 0 && !dt)) return SHK_EINVAL;
    cudaStream_t st = as_stream(stream);
    if (nsteps > plan->fixed_cap) {
        SHK_CUDA(cudaStreamSynchronize(st));
        if (plan->dt_fixed) cudaFree(plan->dt_fixed);
        plan->dt_fixed = nullptr;
        plan->fixed_cap = plan->fixed_steps = 0;
        if (cudaMalloc(&plan->dt_fixed, sizeof(double) * size_t(nsteps) * plan->B) != cudaSuccess)
            return SHK_ENOMEM;
        plan->fixed_cap = nsteps;
    }
    if (nsteps > 0)
        SHK_CUDA(cudaMemcpyAsync(plan->dt_fixed, dt, sizeof(double) * size_t(nsteps) * plan->B,
                                 cudaMemcpyDefault, st));
    plan->fixed_steps = nsteps;
    // the kernels take the plan's device view by value: a captured graph is stale now
    if (plan->graph) {
        cudaGraphExecDestroy(plan->graph);
        plan->graph = nullptr;
    }
    return SHK_OK;
}

}  // extern "C"

namespace {
// boundary kinds and data for every instance: `rows` sets of [B][2][3]
// Dirichlet values / [B][2] Neumann gradients (1: time-independent; else
// steps x 3 stages)
int set_plan_boundary(shk_plan* plan, int32_t left, int32_t right, const double* dirichlet,
                      const double* neumann, int64_t rows, int64_t steps, void* stream) {
    if (!plan || rows < 1) return SHK_EINVAL;
    shk_boundary b = periodic_boundary();
    b.left = left;
    b.right = right;
    if (!valid_boundary(b)) return SHK_EINVAL;
    // the global Lax-Friedrichs speed would also span the ghost values
    if (plan->scheme.flux == SHK_FLUX_LF && left != SHK_BC_PERIODIC) return SHK_EUNSUPPORTED;
    const bool need_dir = left == SHK_BC_DIRICHLET || right == SHK_BC_DIRICHLET;
    const bool need_neu = left == SHK_BC_NEUMANN || right == SHK_BC_NEUMANN;
    if ((need_dir && !dirichlet) || (need_neu && !neumann)) return SHK_EINVAL;
    cudaStream_t st = as_stream(stream);
    const size_t B = static_cast<size_t>(plan->B);
    auto ensure = [&](double** buf, size_t* cap, size_t n) {
        if (*cap >= n) return true;
        if (*buf) {
            if (cudaStreamSynchronize(st) != cudaSuccess) return false;  // a step may still read it
            cudaFree(*buf);
        }
        *buf = nullptr;
        *cap = 0;
        if (cudaMalloc(reinterpret_cast<void**>(buf), sizeof(double) * n) != cudaSuccess) return false;
        *cap = n;
        return true;
    };
    const size_t ndir = 6 * B * size_t(rows), nneu = 2 * B * size_t(rows);
    if (need_dir && !ensure(&plan->bc_dir, &plan->bc_dir_cap, ndir)) return SHK_ENOMEM;
    if (need_neu && !ensure(&plan->bc_neu, &plan->bc_neu_cap, nneu)) return SHK_ENOMEM;
    if (need_dir)
        SHK_CUDA(cudaMemcpyAsync(plan->bc_dir, dirichlet, sizeof(double) * ndir, cudaMemcpyDefault, st));
    if (need_neu)
        SHK_CUDA(cudaMemcpyAsync(plan->bc_neu, neumann, sizeof(double) * nneu, cudaMemcpyDefault, st));
    plan->bc_left = left;
    plan->bc_right = right;
    plan->bc_steps = steps;
    if (plan->graph) {  // kernels take the plan's device view by value
        cudaGraphExecDestroy(plan->graph);
        plan->graph = nullptr;
    }
    return SHK_OK;
}
}  // namespace

extern "C" {

int shk_plan_set_boundary(shk_plan* plan, int32_t left, int32_t right, const double* dirichlet,
                          const double* neumann, void* stream) {
    return set_plan_boundary(plan, left, right, dirichlet, neumann, 1, 0, stream);
}

int shk_plan_set_boundary_steps(shk_plan* plan, int32_t left, int32_t right,
                                const double* dirichlet, const double* neumann, int32_t nsteps,
                                void* stream) {
    if (nsteps < 1) return SHK_EINVAL;
    return set_plan_boundary(plan, left, right, dirichlet, neumann, 3 * int64_t(nsteps), nsteps,
                             stream);
}

int shk_plan_step_graph(shk_plan* plan, void* u_a, void* u_b, int32_t nsteps, void* stream) {
    if (!plan || !u_a || !u_b || u_a == u_b || nsteps < 0 || nsteps % 2) return SHK_EINVAL;
    if (plan->host_steps % 2) return SHK_EINVAL;
    cudaStream_t st = as_stream(stream);
    if (st == nullptr) return SHK_EINVAL;  // capture needs a non-default stream
    if (plan->resident) return shk_plan_step(plan, u_a, u_b, nsteps, stream);  // one launch already
    if (!plan->graph || plan->graph_a != u_a || plan->graph_b != u_b) {
        if (plan->graph) {
            cudaGraphExecDestroy(plan->graph);
            plan->graph = nullptr;
        }
        cudaGraph_t g;
        SHK_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        const int64_t saved = plan->host_steps;
        int r = shk_plan_step(plan, u_a, u_b, 2, stream);
        plan->host_steps = saved;
        cudaError_t e = cudaStreamEndCapture(st, &g);
        if (r != SHK_OK) return r;
        SHK_CUDA(e);
        e = cudaGraphInstantiate(&plan->graph, g, 0);
        cudaGraphDestroy(g);
        SHK_CUDA(e);
        plan->graph_a = u_a;
        plan->graph_b = u_b;
    }
    for (int i = 0; i < nsteps / 2; ++i) SHK_CUDA(cudaGraphLaunch(plan->graph, st));
    plan->host_steps += nsteps;
    return SHK_OK;
}

int shk_plan_reduce(shk_plan* plan, const void* u, int32_t p, double* out, void* stream) {
    if (!plan || !u || !out || (p != 0 && p != 1 && p != 2 && p != -1)) return SHK_EINVAL;
    cudaStream_t st = as_stream(stream);
    const PlanDev D = plan->dev();
    if (plan->dtype == SHK_F64)
        batched_partial_kernel<double><<<plan->grid, kThreads, 0, st>>>(D, static_cast<const double*>(u), p);
    else
        batched_partial_kernel<float><<<plan->grid, kThreads, 0, st>>>(D, static_cast<const float*>(u), p);
    SHK_CUDA(cudaGetLastError());
    instance_sum_kernel<<<(plan->B + 127) / 128, 128, 0, st>>>(D, plan->item_first, p, out);
    return cuda_check(cudaGetLastError());
}

}  // extern "C"

// ===========================================================================
// Lax-Friedrichs operator without any device allocation
// ===========================================================================
// Some callers cannot allocate device memory of their own. The main case for
// this library is an integration as a JAX custom call: JAX reserves most of the
// GPU for its own pool up front and hands a handler only its input and output
// buffers, so a cudaMalloc in the handler competes with (or fails against)
// that pool. The regular Lax-Friedrichs path needs one scratch value (the
// instance-wide max |f'(u)|) that the caller allocates; this variant keeps its
// scratch -- one partial maximum per 512-cell tile plus the final maximum -- in
// a fixed array compiled into the library instead.
//
// The array lives in every GPU's memory from the moment the library is loaded
// on that GPU until the process exits (kNoAllocMaxTiles + 1 doubles, 32 KiB).
// All calls share it: a call overwrites every slot it reads, so nothing has to
// start at zero, but two calls that overlap on the GPU (different streams, or
// different host threads) race on it and must be serialised by the caller.
namespace {

constexpr int kNoAllocTile = 512;          // cells per tile, as shk_apply_operator_f64
constexpr int kNoAllocMaxTiles = 4096;     // => at most 2,097,152 interior cells per call

static __device__ __align__(256) double g_noalloc_scratch[kNoAllocMaxTiles + 1];

constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mutex;
struct NoAllocAddr {
    unsigned long long ctx_id = 0;  // cuCtxGetId of the context the address belongs to
    double* addr = nullptr;
};
NoAllocAddr g_noalloc_addr[kMaxDevices];

using CtxGetCurrentFn = CUresult (*)(CUcontext*);
using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long*);

// Unique ID of the calling thread's current CUDA context (0 if none). The
// driver functions come through the runtime's entry-point query, so the
// library does not link libcuda itself.
unsigned long long current_context_id() {
    static CtxGetCurrentFn get_current = nullptr;
    static CtxGetIdFn get_id = nullptr;
    if (!get_current || !get_id) {
        void* f1 = nullptr;
        void* f2 = nullptr;
        cudaDriverEntryPointQueryResult q1, q2;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f1, 12000, cudaEnableDefault, &q1) !=
                cudaSuccess ||
            cudaGetDriverEntryPointByVersion("cuCtxGetId", &f2, 12000, cudaEnableDefault, &q2) !=
                cudaSuccess ||
            q1 != cudaDriverEntryPointSuccess || q2 != cudaDriverEntryPointSuccess)
            return 0;
        get_current = reinterpret_cast<CtxGetCurrentFn>(f1);
        get_id = reinterpret_cast<CtxGetIdFn>(f2);
    }
    CUcontext ctx = nullptr;
    unsigned long long id = 0;
    if (get_current(&ctx) != CUDA_SUCCESS || !ctx || get_id(ctx, &id) != CUDA_SUCCESS) return 0;
    return id;
}

// Device address of g_noalloc_scratch in the current device's context. In host
// code the symbol itself is only a host-side stand-in, so the address must come
// from cudaGetSymbolAddress with that device current. It is looked up once per
// context: a context created after cudaDeviceReset loads the module again, so
// the address of an earlier context is not reused.
int noalloc_scratch(double** out) {
    int dev = 0;
    SHK_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return SHK_EUNSUPPORTED;
    const unsigned long long id = current_context_id();  // 0 before the runtime made one current
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    NoAllocAddr& slot = g_noalloc_addr[dev];
    if (!slot.addr || id == 0 || slot.ctx_id != id) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            std::fprintf(stderr, "libshocks: cudaGetSymbolAddress failed: %s\n", cudaGetErrorString(e));
            return SHK_ECUDA;
        }
        slot.addr = static_cast<double*>(p);
        slot.ctx_id = current_context_id();  // the context the lookup ran in
    }
    *out = slot.addr;
    return SHK_OK;
}

// per-tile max |f'(u)| into partial[tile]
template <int EQ>
__global__ void __launch_bounds__(kThreads) noalloc_tile_max_kernel(const double* __restrict__ u, int64_t n,
                                                                    double c, double* partial) {
    __shared__ unsigned long long red[32];
    const int64_t s0 = int64_t(blockIdx.x) * kNoAllocTile;
    const int te = static_cast<int>(imin64(kNoAllocTile, n - s0));
    unsigned long long mx = 0;
    for (int i = threadIdx.x; i < te; i += blockDim.x) {
        const unsigned long long b = abs_bits(wave_speed<EQ>(u[s0 + i], c));
        mx = b > mx ? b : mx;
    }
    const unsigned long long bm = block_max<unsigned long long>(mx, red);
    if (threadIdx.x == 0) partial[blockIdx.x] = from_bits(bm);
}

// max of the ntiles partials into partial[kNoAllocMaxTiles]
__global__ void __launch_bounds__(kThreads) noalloc_reduce_kernel(double* partial, int ntiles) {
    __shared__ unsigned long long red[32];
    unsigned long long mx = 0;
    for (int i = threadIdx.x; i < ntiles; i += blockDim.x) {
        const unsigned long long b = abs_bits(partial[i]);
        mx = b > mx ? b : mx;
    }
    const unsigned long long bm = block_max<unsigned long long>(mx, red);
    if (threadIdx.x == 0) partial[kNoAllocMaxTiles] = from_bits(bm);
}

}  // namespace

extern "C" int shk_apply_operator_lf_noalloc_f64(const shk_scheme* scheme, const double* u,
                                                 double* out, int64_t n, int32_t nghosts,
                                                 double dx, void* stream) {
    if (!valid_scheme(scheme) || scheme->flux != SHK_FLUX_LF || !u || !out || n < 3 ||
        nghosts < 3 || !(dx > 0))
        return SHK_EINVAL;
    const int64_t ntiles = (n + kNoAllocTile - 1) / kNoAllocTile;
    if (ntiles > kNoAllocMaxTiles) {
        std::fprintf(stderr,
                     "libshocks: shk_apply_operator_lf_noalloc_f64: n = %lld exceeds the static "
                     "scratch limit of %lld cells\n",
                     static_cast<long long>(n),
                     static_cast<long long>(kNoAllocMaxTiles) * kNoAllocTile);
        return SHK_ETOOLARGE;
    }
    double* scratch = nullptr;
    const int st0 = noalloc_scratch(&scratch);
    if (st0 != SHK_OK) return st0;
    cudaStream_t st = as_stream(stream);
    const double c = scheme->speed;
    const int nt = static_cast<int>(ntiles);
    switch (scheme->equation) {
        case SHK_EQ_BURGERS: noalloc_tile_max_kernel<SHK_EQ_BURGERS><<<nt, kThreads, 0, st>>>(u + nghosts, n, c, scratch); break;
        case SHK_EQ_ADVECTION: noalloc_tile_max_kernel<SHK_EQ_ADVECTION><<<nt, kThreads, 0, st>>>(u + nghosts, n, c, scratch); break;
        default: noalloc_tile_max_kernel<SHK_EQ_LWR><<<nt, kThreads, 0, st>>>(u + nghosts, n, c, scratch); break;
    }
    SHK_CUDA(cudaGetLastError());
    noalloc_reduce_kernel<<<1, kThreads, 0, st>>>(scratch, nt);
    SHK_CUDA(cudaGetLastError());
    // the operator itself is the regular one, reading the max from the scratch
    const int W = kNoAllocTile + 2 * op_halo<double>();
    const size_t smem = Smem<double>::host_bytes(W);
    OpParams<double> p = make_params<double>(scheme);
    p.dx = dx;
    ApplyOpLaunch f{u, out, n, nghosts, kNoAllocTile, dx, scratch + kNoAllocMaxTiles, p, smem, nt, st,
                    periodic_boundary()};
    return dispatch_scheme<double>(scheme, f);
}

extern "C" int64_t shk_apply_operator_lf_noalloc_max_cells(void) {
    return static_cast<int64_t>(kNoAllocMaxTiles) * kNoAllocTile;
}

// ===========================================================================
// bounds-check build (libshocks_check.so): logs and test hooks
// ===========================================================================
#ifdef SHOCKS_BOUNDS_CHECK
extern "C" int shk_check_tu_adjoint(shk::BoundsLog* out, int32_t reset);
extern "C" int shk_check_tu_ghosted(shk::BoundsLog* out, int32_t reset);

extern "C" int shk_check_bounds(int32_t reset, int32_t* flag, int32_t* block, int32_t* thread,
                                int64_t* offset, int64_t* extent) {
    SHK_CUDA(cudaDeviceSynchronize());
    shk::BoundsLog logs[3] = {};
    SHK_CUDA(shk::bounds_log_read(&logs[0], reset != 0));
    int r = shk_check_tu_adjoint(&logs[1], reset);
    if (r == SHK_OK) r = shk_check_tu_ghosted(&logs[2], reset);
    if (r != SHK_OK) return r;
    const shk::BoundsLog* hit = nullptr;
    for (const shk::BoundsLog& l : logs)
        if (!hit && l.flag) hit = &l;
    if (flag) *flag = hit ? 1 : 0;
    if (block) *block = hit ? hit->block : -1;
    if (thread) *thread = hit ? hit->thread : -1;
    if (offset) *offset = hit ? hit->offset : 0;
    if (extent) *extent = hit ? hit->extent : 0;
    return SHK_OK;
}

extern "C" int shk_check_force_timeout(uint32_t extra_bytes, int64_t wait_limit) {
    const long long lim = static_cast<long long>(wait_limit);
    SHK_CUDA(cudaMemcpyToSymbol(shk::g_test_extra_tx, &extra_bytes, sizeof(extra_bytes)));
    SHK_CUDA(cudaMemcpyToSymbol(shk::g_test_wait_limit, &lim, sizeof(lim)));
    return SHK_OK;
}
#endif
