// Many independent circuits in one persistent launch, each with its own
// gate list and Pauli-string Hamiltonian: the <H> of every circuit.
//
// The reference answers each request of BatchExecution::exp_value with a
// fresh simulator that replays the gates and sums the strings
// (kbw src/quantum_execution.rs:392-405, 109-158).  Here the host plans
// every circuit with the sweep planner (planner.cpp) into the gate programs
// the tile kernels run, and cuts the work into items that persistent CTAs take
// from one queue:
//   * n <= K: one item, the whole circuit on a K-qubit tile that never leaves
//     the SM (qubits n..K-1 stay |0>), its sweeps applied to the tile in
//     registers and shared memory;
//   * n > K: the state has its place in a global buffer, and an item is a few
//     tiles of one planned sweep (TMA bulk loads one tile ahead, bounded waits,
//     coalesced stores, as k_sweep walks a handle's state) or of one <H> pass.
//     An item waits until its circuit's earlier sweeps are done (a counter per
//     circuit).  The queue is ordered by sweep, so every item that another one
//     waits for was taken before it: the first unfinished item never waits,
//     whatever the number of resident CTAs.
// One CTA per circuit would leave the largest circuits to single SMs: 1024
// circuits of 8..20 qubits took 55 ms, the time of one 20-qubit circuit's CTA.
// <H> = sum_k c_k <P_k> with P = i^{ny} X^x Z^z: the strings are grouped by
// flip mask x, and for each group one loop over the amplitudes forms
// conj(a_s) a_{s^x} once and adds every string's signed share, accumulated
// FP64-grade.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <exception>
#include <functional>
#include <memory>
#include <mutex>
#include <thread>
#include <unordered_map>
#include <vector>

#include "../../include/kbwg.h"
#include "retry.h"
#include "kernels.h"
#include "sim.h"
#include "sweep_dev.cuh"

namespace kbwg {

struct BatchSweep {
    uint32_t l, m, nstages, gate_count;
    uint32_t gate_off, data_count;
    uint8_t hq[16];
    uint8_t stage_layout[kMaxStages];
    uint16_t stage_end[kMaxStages];
};

struct BatchJob {
    uint32_t n, nsweeps, sweep_off, nterms;
    uint32_t term_off, id, pad;
    uint32_t pass_off, npasses;  // tiled <H> passes (registers larger than a tile)
    uint32_t items, part_off, nparts;  // items of the circuit; its partial sums of <H>
    uint64_t state_off;                // first amplitude of its state (n > K)
};

// What an item of the queue does: part `part` of task `task`.
enum { BT_WHOLE = 0, BT_SWEEP = 1, BT_PASS = 2, BT_WIDE = 3 };
struct BatchTask {
    uint32_t job, kind;
    uint32_t index;  // sweep or pass of the circuit
    uint32_t need;   // items of the circuit that must be done first
    uint32_t per;    // tiles per part (BT_WIDE: log2 of the amplitudes per part)
    uint32_t slot;   // partial sum of part 0 (BT_PASS, BT_WIDE), within the circuit's
};
struct BatchItem {
    uint32_t task, part;
};

struct BatchTerm {
    uint64_t x, z;
    double cr, ci;  // c_k * i^{ny}: the string's share of conj(a_s) a_{s^x} is sign * (cr p.re - ci p.im)
};

// One tiled <H> pass of a register larger than a tile: tiles of 2^K
// amplitudes (2^l contiguous ones per chunk, the chunks picked by the m
// qubits hq) hold both a_s and a_{s^x} for every string of the pass.
struct BatchPass {
    uint32_t l, m, term_off, nterms;
    uint8_t hq[16];
};
// A string of a pass: flip and phase masks on the tile's local bits, phase
// mask on the qubits outside it; `last` closes a run of strings with the
// same flip mask and coefficient (their signs are counted, the coefficient
// applied once).
struct BatchTileTerm {
    uint32_t xl, zl;
    uint64_t zo;
    double cr, ci;
    uint32_t last, pad;
};

struct BatchArgs {
    const BatchJob *jobs;
    const BatchTask *tasks;
    const BatchItem *items;
    uint32_t nitems;
    unsigned *next;
    unsigned *done;      // finished items per job
    double *partials;
    const BatchSweep *sweeps;
    const TileGate *prog;
    const BatchTerm *terms;
    const BatchPass *passes;
    const BatchTileTerm *tterms;
    double *energies;
    void *states;
    int *err;
};

template <class P, int K, int R>
struct BatchKernel {
    using Mem = typename P::Mem;
    static constexpr int kThreads = 32 << (K - kLaneBits - R);
    static constexpr size_t kTileBytes = sizeof(Mem) << K;
    // complex64: three CTAs with one tile buffer each rather than two with two
    // (24 warps hide the dispatch's latency better than the load ahead does:
    // 1024 circuits 26.5 -> 23.3 ms; four CTAs spill, 28.2 ms).
    static constexpr int kBuffers = sizeof(Mem) == 8 ? 1 : 2;
    static constexpr int kCtas = sizeof(Mem) == 8 ? 3 : 2;
    static constexpr size_t kSmem = kBuffers * kTileBytes + 256 * sizeof(uint64_t) + kMaxSweepGates * sizeof(TileGate) + 64 +
                                    32 * 8 + 64;
};

// Wait until `need` items of a circuit are done (polled by one thread, at
// most ~10 s); false, with the error flag set, if they never are.  Then orders
// the circuit's amplitudes, written by other CTAs through the generic proxy,
// before this CTA's TMA loads.
__device__ __forceinline__ bool batch_wait(const unsigned *done, uint32_t need, int *err) {
    bool ok = true;
    if (threadIdx.x == 0) {
        ok = false;
        for (uint32_t spin = 0; spin < (1u << 25); spin++) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(done) : "memory");
            if (v >= need) {
                ok = true;
                break;
            }
            if ((spin & 1023u) == 1023u && *(volatile int *)err) break;  // another wait ran out
            __nanosleep(200);
        }
        if (!ok) atomicExch(err, 1);
    }
    if (__syncthreads_or(!ok)) return false;
    __threadfence();
    asm volatile("fence.proxy.async;" ::: "memory");
    return true;
}

// Sum of v over the CTA (every thread must call it); valid in thread 0.
__device__ __forceinline__ double batch_block_sum(double v, double *red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
    __syncthreads();
    return t;
}

// FP64-grade sum of float shares (short float runs, then widened) or of
// double shares
template <class T> struct BatchAcc {
    double v = 0.0;
    T part = (T)0;
    int cnt = 0;
    __device__ __forceinline__ void add(T x) {
        part += x;
        if (++cnt == 16) {
            v += (double)part;
            part = (T)0;
            cnt = 0;
        }
    }
    __device__ __forceinline__ double value() { return v + (double)part; }
};

template <class Mem>
__device__ __forceinline__ Mem batch_basis(bool one) {
    Mem m;
    m.re = one ? 1 : 0;
    m.im = 0;
    return m;
}

// Part of one tiled <H> pass of a register larger than a tile: tiles [t0, t1),
// each staged once (TMA, one tile ahead), every string of the pass summed from
// shared memory.  (Its own function: the sweep loop keeps its register
// allocation.)
template <class P, int K, int R>
__device__ __noinline__ bool batch_energy_pass(const BatchArgs &a, const BatchPass &bp, uint32_t n,
                                               typename P::Mem *state, uint64_t t0, uint64_t t1,
                                               typename P::Mem *tiles_mem, uint64_t *chunk_off, uint64_t *bar,
                                               uint32_t *phase, double &sum) {
    using Mem = typename P::Mem;
    using T = decltype(Mem{}.re);
    BatchAcc<T> acc;  // (local: the caller's accumulator would live in memory across the call)
    using BK = BatchKernel<P, K, R>;
    constexpr int NR = 1 << R;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t l = bp.l, m = bp.m;
    const uint32_t chunk = 1u << l, nchunks = 1u << m;
    for (uint32_t c = threadIdx.x; c < nchunks; c += blockDim.x) {
        uint64_t off = 0;
        for (uint32_t j = 0; j < m; j++) off |= (uint64_t)((c >> j) & 1u) << bp.hq[j];
        chunk_off[c] = off;
    }
    __syncthreads();
    auto tile_base = [&](uint64_t t) {
        uint64_t b = t << l;
        for (uint32_t j = 0; j < m; j++) b = insert_zero_at(b, bp.hq[j]);
        return b;
    };
    auto issue_load = [&](uint64_t t, uint32_t buf) {
        if (warp == 0) {
            const uint64_t b = tile_base(t);
            if (lane == 0) mbar_expect_tx(bar + buf, (uint32_t)BK::kTileBytes);
            __syncwarp();
            for (uint32_t c = lane; c < nchunks; c += 32)
                tma_load(tiles_mem + ((size_t)buf << K) + (size_t)c * chunk, state + b + chunk_off[c],
                         chunk * (uint32_t)sizeof(Mem), bar + buf);
        }
    };
    const BatchTileTerm *tt = a.tterms + bp.term_off;
    issue_load(t0, 0);
    if (BK::kBuffers > 1 && t0 + 1 < t1) issue_load(t0 + 1, 1);
    for (uint64_t tau = t0; tau < t1; tau++) {
        const uint32_t buf = (uint32_t)(tau - t0) % (uint32_t)BK::kBuffers;
        const Mem *tile_mem = tiles_mem + ((size_t)buf << K);
        const uint64_t base = tile_base(tau);
        if (!tile_wait(bar + buf, phase[buf] & 1u, a.err)) return false;
        phase[buf]++;
        // each thread's NR amplitudes u = tid + i * threads in registers;
        // strings outer (their fields read once per tile), signs counted
        // per amplitude, the product formed once per run
        T ar[NR], ai[NR];
        int cnt[NR];
#pragma unroll
        for (int i = 0; i < NR; i++) {
            const Mem m2 = tile_mem[threadIdx.x + (uint32_t)i * BK::kThreads];
            ar[i] = m2.re;
            ai[i] = m2.im;
            cnt[i] = 0;
        }
        for (uint32_t k = 0; k < bp.nterms; k++) {
            const BatchTileTerm t = tt[k];
            const uint32_t op = (uint32_t)__popcll(base & t.zo) & 1u;
#pragma unroll
            for (int i = 0; i < NR; i++) {
                const uint32_t u = threadIdx.x + (uint32_t)i * BK::kThreads;
                cnt[i] += (((uint32_t)__popc((u ^ t.xl) & t.zl) + op) & 1u) ? -1 : 1;
            }
            if (t.last) {  // (uniform)
#pragma unroll
                for (int i = 0; i < NR; i++) {
                    const uint32_t u = threadIdx.x + (uint32_t)i * BK::kThreads;
                    T pr, pim;  // conj(a_u) a_{u^x}
                    if (t.xl == 0u) {
                        pr = ar[i] * ar[i] + ai[i] * ai[i];
                        pim = (T)0;
                    } else {
                        const Mem ax = tile_mem[u ^ t.xl];
                        pr = ar[i] * ax.re + ai[i] * ax.im;
                        pim = ar[i] * ax.im - ai[i] * ax.re;
                    }
                    acc.add((T)cnt[i] * ((T)t.cr * pr - (T)t.ci * pim));
                    cnt[i] = 0;
                }
            }
        }
        __syncthreads();  // the tile is read no more: a load may land in its buffer
        if (tau + BK::kBuffers < t1) issue_load(tau + BK::kBuffers, buf);
    }
    sum = acc.value();
    return true;
}

template <class P, int K, int R>
__global__ void __launch_bounds__(BatchKernel<P, K, R>::kThreads, BatchKernel<P, K, R>::kCtas) k_batch_circuits(const __grid_constant__ BatchArgs a) {
    using Amp = typename P::Amp;
    using Mem = typename P::Mem;
    using T = decltype(Mem{}.re);
    using BK = BatchKernel<P, K, R>;
    static_assert(sizeof(Amp) == sizeof(Mem), "register and memory amplitudes share the tile buffers");
    constexpr int NR = 1 << R;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    Amp *tile = reinterpret_cast<Amp *>(smem_raw);  // kBuffers tiles
    Mem *tile_mem = reinterpret_cast<Mem *>(smem_raw);
    unsigned char *q = smem_raw + BK::kBuffers * BK::kTileBytes;
    uint64_t *chunk_off = reinterpret_cast<uint64_t *>(q);
    q += 256 * sizeof(uint64_t);
    TileGate *sg = reinterpret_cast<TileGate *>(q);
    q += kMaxSweepGates * sizeof(TileGate);
    uint32_t *meta = reinterpret_cast<uint32_t *>(q);
    q += 64;
    double *red = reinterpret_cast<double *>(q);
    q += 32 * 8;
    uint64_t *bar = reinterpret_cast<uint64_t *>(q);  // one per tile buffer

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t FA = (uint32_t)lane | ((uint32_t)warp << (kLaneBits + R));
    const uint32_t FB = (uint32_t)lane | ((uint32_t)warp << kLaneBits);
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        mbar_init(bar + 1, 1);
        fence_mbar_init();
    }
    uint32_t phase[2] = {0, 0};
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) meta[0] = atomicAdd(a.next, 1u);
        __syncthreads();
        const uint32_t ix = meta[0];
        if (ix >= a.nitems) break;
        const BatchItem item = a.items[ix];
        const BatchTask task = a.tasks[item.task];
        const BatchJob &job = a.jobs[task.job];
        const uint32_t n = job.n;
        Mem *state = reinterpret_cast<Mem *>(a.states) + job.state_off;
        if (task.need && !batch_wait(a.done + task.job, task.need, a.err)) return;
        double energy = 0.0;  // this thread's share of <H>
        if (task.kind == BT_WHOLE || task.kind == BT_SWEEP) {
            const bool whole = task.kind == BT_WHOLE;
            const uint32_t s0 = whole ? 0u : task.index, s1 = whole ? job.nsweeps : task.index + 1;
            const uint64_t ntiles = whole ? 1ull : (1ull << (n - K));
            const uint64_t t0 = whole ? 0 : (uint64_t)item.part * task.per;
            const uint64_t t1 = whole ? 1 : min(ntiles, t0 + task.per);
            if (whole)  // |0...0>
                for (uint32_t u = threadIdx.x; u < (1u << K); u += blockDim.x) tile[u] = P::from_mem(batch_basis<Mem>(u == 0));
            for (uint32_t sw = s0; sw < s1; sw++) {
                const BatchSweep &bs = a.sweeps[job.sweep_off + sw];
                const uint32_t l = bs.l, m = bs.m, nst = bs.nstages;
                for (uint32_t i = threadIdx.x; i < bs.gate_count + bs.data_count; i += blockDim.x)
                    sg[i] = a.prog[bs.gate_off + i];
                for (uint32_t c = threadIdx.x; c < (1u << m); c += blockDim.x) {
                    uint64_t off = 0;
                    for (uint32_t j = 0; j < m; j++) off |= (uint64_t)((c >> j) & 1u) << bs.hq[j];
                    chunk_off[c] = off;
                }
                __syncthreads();
                const uint32_t chunk = 1u << l, nchunks = 1u << m;
                const uint64_t lowmask = chunk - 1;
                auto tile_base = [&](uint64_t t) {
                    uint64_t b = t << l;
                    for (uint32_t j = 0; j < m; j++) b = insert_zero_at(b, bs.hq[j]);
                    return b;
                };
                auto issue_load = [&](uint64_t t, uint32_t buf) {
                    if (warp == 0) {
                        const uint64_t b = tile_base(t);
                        if (lane == 0) mbar_expect_tx(bar + buf, (uint32_t)BK::kTileBytes);
                        __syncwarp();
                        for (uint32_t c = lane; c < nchunks; c += 32)
                            tma_load(tile_mem + ((size_t)buf << K) + (size_t)c * chunk, state + b + chunk_off[c],
                                     chunk * (uint32_t)sizeof(Mem), bar + buf);
                    }
                };
                // the first sweep starts from |0...0>: nothing is read
                const bool load = !whole && sw > 0;
                if (load) {
                    issue_load(t0, 0);
                    if (BK::kBuffers > 1 && t0 + 1 < t1) issue_load(t0 + 1, 1);
                }
                for (uint64_t tau = t0; tau < t1; tau++) {
                    const uint32_t buf = whole ? 0u : (uint32_t)(tau - t0) % (uint32_t)BK::kBuffers;
                    Amp *tb = tile + ((size_t)buf << K);
                    const uint64_t base = tile_base(tau);
                    int layout = bs.stage_layout[0];
                    int R0 = (layout == LAYOUT_A) ? kLaneBits : (K - R);
                    uint32_t F = (layout == LAYOUT_A) ? FA : FB;
                    Amp v[NR];
                    if (whole) {
#pragma unroll
                        for (int j = 0; j < NR; j++) v[j] = tb[F | ((uint32_t)j << R0)];
                    } else if (load) {
                        if (!tile_wait(bar + buf, phase[buf] & 1u, a.err)) return;
                        phase[buf]++;
                        const Mem *tm = tile_mem + ((size_t)buf << K);
#pragma unroll
                        for (int j = 0; j < NR; j++) v[j] = P::from_mem(tm[F | ((uint32_t)j << R0)]);
                    } else {
#pragma unroll
                        for (int j = 0; j < NR; j++) v[j] = P::from_mem(batch_basis<Mem>(base == 0 && F == 0 && j == 0));
                    }
                    uint32_t g0 = 0;
                    for (uint32_t s = 0; s < nst; s++) {
                        const int nl = bs.stage_layout[s];
                        if (nl != layout) {
#pragma unroll
                            for (int j = 0; j < NR; j++) tb[F | ((uint32_t)j << R0)] = v[j];
                            __syncthreads();
                            layout = nl;
                            R0 = (layout == LAYOUT_A) ? kLaneBits : (K - R);
                            F = (layout == LAYOUT_A) ? FA : FB;
#pragma unroll
                            for (int j = 0; j < NR; j++) v[j] = tb[F | ((uint32_t)j << R0)];
                        }
                        const uint32_t g1 = bs.stage_end[s];
                        for (uint32_t gi = g0; gi < g1; gi++) tile_gate<P, K, R, uint64_t>(sg[gi], v, R0, F, base);
                        g0 = g1;
                    }
                    if (whole) {
                        // every thread rewrites the positions it read in this layout
#pragma unroll
                        for (int j = 0; j < NR; j++) tb[F | ((uint32_t)j << R0)] = v[j];
                    } else {
                        // the tile buffer is read no more (the load after next) once all threads pass here
                        fence_proxy_async();
                        __syncthreads();
                        if (load && tau + BK::kBuffers < t1) issue_load(tau + BK::kBuffers, buf);
#pragma unroll
                        for (int j = 0; j < NR; j++) {
                            const uint32_t u = F | ((uint32_t)j << R0);
                            state[base + chunk_off[u >> l] + (u & lowmask)] = P::to_mem(v[j]);
                        }
                    }
                }
                __syncthreads();
            }
        } else if (task.kind == BT_PASS) {
            const uint64_t t0 = (uint64_t)item.part * task.per, t1 = min(1ull << (n - K), (unsigned long long)(t0 + task.per));
            if (!batch_energy_pass<P, K, R>(a, a.passes[job.pass_off + task.index], n, state, t0, t1, tile_mem, chunk_off,
                                            bar, phase, energy))
                return;
        }
        if (task.kind == BT_WHOLE || task.kind == BT_WIDE) {
            // <H> string by string: a register held on the tile, or flip masks too wide for any tile
            const bool whole = task.kind == BT_WHOLE;
            const uint64_t a0 = whole ? 0 : (uint64_t)item.part << task.per;
            const uint64_t a1 = whole ? (1ull << n) : min(1ull << n, (unsigned long long)(a0 + (1ull << task.per)));
            BatchAcc<T> acc;
            for (uint32_t t0 = 0; t0 < job.nterms;) {
                const uint64_t x = a.terms[job.term_off + t0].x;
                uint32_t t1 = t0 + 1;
                while (t1 < job.nterms && a.terms[job.term_off + t1].x == x) t1++;
                for (uint64_t s = a0 + threadIdx.x; s < a1; s += blockDim.x) {
                    Mem as, ax;
                    if (whole) {
                        as = P::to_mem(tile[s]);
                        ax = P::to_mem(tile[s ^ x]);
                    } else {
                        as = state[s];
                        ax = state[s ^ x];
                    }
                    // conj(a_s) a_{s^x}
                    const T pr = as.re * ax.re + as.im * ax.im, pi = as.re * ax.im - as.im * ax.re;
                    T share = (T)0;
                    for (uint32_t k = t0; k < t1; k++) {
                        const BatchTerm &tk = a.terms[job.term_off + k];
                        const T w = (T)tk.cr * pr - (T)tk.ci * pi;
                        share += (__popcll((s ^ x) & tk.z) & 1) ? -w : w;
                    }
                    acc.add(share);
                }
                t0 = t1;
            }
            energy = acc.value();
        }
        if (task.kind != BT_SWEEP) {
            const double e = batch_block_sum(energy, red);
            if (threadIdx.x == 0) {
                if (task.kind == BT_WHOLE) a.energies[job.id] = e;
                else a.partials[job.part_off + task.slot + item.part] = e;
            }
        }
        if (task.kind == BT_WHOLE) continue;
        // the item is done: its stores before the counter, for the generic
        // reads and the TMA loads of the items that wait for it; the circuit's
        // last item adds up its partial sums, in their order
        __threadfence();
        asm volatile("fence.proxy.async;" ::: "memory");
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned old;
            asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(a.done + task.job) : "memory");
            if (old + 1 == job.items) {
                double t = 0.0;
                for (uint32_t k = 0; k < job.nparts; k++) t += __ldcg(a.partials + job.part_off + k);
                a.energies[job.id] = t;
            }
        }
    }
}

// ---- host side -----------------------------------------------------------------------
// Room for the states of circuits larger than a tile in one launch (more
// circuits run in further launches on the same buffer).
constexpr uint64_t kBatchStateBytes = 16ull << 30;

struct BatchCircuitIn {
    uint32_t n;
    std::vector<GateDesc> gates;
    std::vector<BatchTerm> terms;  // sorted by flip mask
    // the circuit's plan (batch_run)
    std::vector<BatchSweep> sweeps;
    std::vector<TileGate> prog;
    std::vector<BatchPass> passes;       // tiled <H> passes (n > K); then `terms`
    std::vector<BatchTileTerm> tterms;   // holds only the strings too wide for a tile
    bool placed = true;
    // validation result
    int32_t status = KBWG_OK;
    const char *error = nullptr;
};

// Host threads of one call: its steps run fn(i) for i in [0, n), items taken
// one at a time, on the calling thread and the workers.  Started once per call
// and only for enough gates (starting one takes ~60 us here, planning 4,000
// gates about as long; a set of 16 for every step cost 1 ms each time).  An
// exception in any item (an allocation failing) stops the step's remaining
// items and is rethrown by run(), on the calling thread, when no worker is in
// it any more.
class BatchWorkers {
public:
    explicit BatchWorkers(size_t gates) {
        const size_t hw = std::max(1u, std::thread::hardware_concurrency());
        const size_t nt = std::min(hw, 1 + gates / 4000);
        try {
            for (size_t t = 1; t < nt; t++) threads_.emplace_back([this] { loop(); });
        } catch (...) {  // fewer threads than asked: the ones started and the caller share the items
        }
    }
    ~BatchWorkers() {
        {
            std::lock_guard<std::mutex> lk(mu_);
            stop_ = true;
        }
        start_.notify_all();
        for (std::thread &t : threads_) t.join();
    }
    void run(size_t n, const std::function<void(size_t)> &fn) {
        if (threads_.empty() || n < 2) {
            for (size_t i = 0; i < n; i++) fn(i);
            return;
        }
        {
            std::lock_guard<std::mutex> lk(mu_);
            fn_ = &fn;
            n_ = n;
            next_.store(0);
            busy_ = threads_.size();
            step_++;
        }
        start_.notify_all();
        items();
        std::unique_lock<std::mutex> lk(mu_);
        done_.wait(lk, [&] { return busy_ == 0; });
        fn_ = nullptr;
        if (first_) {
            const std::exception_ptr e = first_;
            first_ = nullptr;
            std::rethrow_exception(e);
        }
    }

private:
    void items() {
        try {
            for (size_t i; (i = next_.fetch_add(1, std::memory_order_relaxed)) < n_;) (*fn_)(i);
        } catch (...) {
            std::lock_guard<std::mutex> lk(mu_);
            if (!first_) first_ = std::current_exception();
            next_.store(n_);
        }
    }
    void loop() {
        uint64_t seen = 0;
        for (;;) {
            {
                std::unique_lock<std::mutex> lk(mu_);
                start_.wait(lk, [&] { return stop_ || step_ != seen; });
                if (stop_) return;
                seen = step_;
            }
            items();
            std::lock_guard<std::mutex> lk(mu_);
            if (--busy_ == 0) done_.notify_one();
        }
    }
    std::vector<std::thread> threads_;
    std::mutex mu_;
    std::condition_variable start_, done_;
    const std::function<void(size_t)> *fn_ = nullptr;
    size_t n_ = 0, busy_ = 0;
    std::atomic<size_t> next_{0};
    uint64_t step_ = 0;
    std::exception_ptr first_;
    bool stop_ = false;
};

// Device buffer of a call, kept for the next one (the largest up to
// kBatchKeepBytes, one per process): allocating and freeing a gigabyte costs
// milliseconds of a call.  Calls that overlap take their own; a call's work
// is finished when it gives its buffer back.  kbwg_batch_release frees it.
constexpr size_t kBatchKeepBytes = 4ull << 30;
static std::mutex g_batch_mu;
static int g_batch_dev = -1;
static void *g_batch_buf = nullptr;
static size_t g_batch_cap = 0;

static cudaError_t batch_take(int dev, size_t bytes, char **buf, size_t *cap) {
    {
        std::lock_guard<std::mutex> lk(g_batch_mu);
        if (g_batch_buf && g_batch_dev == dev && g_batch_cap >= bytes) {
            *buf = (char *)g_batch_buf;
            *cap = g_batch_cap;
            g_batch_buf = nullptr;
            return cudaSuccess;
        }
    }
    *cap = bytes;
    return device_malloc((void **)buf, bytes);  // (a kept buffer that is too small may be what is missing)
}

static void batch_give(int dev, char *buf, size_t cap) {
    void *drop = buf;  // (the one kept before is on this device too)
    if (cap <= kBatchKeepBytes) {
        std::lock_guard<std::mutex> lk(g_batch_mu);
        if (!g_batch_buf || (g_batch_dev == dev && g_batch_cap < cap)) {
            drop = g_batch_buf;
            g_batch_buf = buf;
            g_batch_cap = cap;
            g_batch_dev = dev;
        }
    }
    if (drop) cudaFree(drop);
}

size_t batch_kept_bytes() {
    std::lock_guard<std::mutex> lk(g_batch_mu);
    return g_batch_buf ? g_batch_cap : 0;
}

cudaError_t device_malloc(void **p, size_t bytes) {
    return alloc_or_release(
        cudaErrorMemoryAllocation,
        [&] {
            const cudaError_t e = cudaMalloc(p, bytes);
            if (e != cudaSuccess) cudaGetLastError();
            return e;
        },
        batch_release_workspace);
}

bool batch_release_workspace() {
    void *buf = nullptr;
    int dev = -1, cur = -1;
    {
        std::lock_guard<std::mutex> lk(g_batch_mu);
        buf = g_batch_buf;
        dev = g_batch_dev;
        g_batch_buf = nullptr;
        g_batch_cap = 0;
    }
    if (!buf) return false;
    cudaGetDevice(&cur);
    if (cur != dev) cudaSetDevice(dev);
    cudaFree(buf);
    if (cur != dev && cur >= 0) cudaSetDevice(cur);
    return true;
}

template <class P, int K, int R>
static int32_t batch_run(int arith, BatchWorkers &workers, std::vector<BatchCircuitIn> &circs, double *energies) {
    using BK = BatchKernel<P, K, R>;
    using Mem = typename P::Mem;
    auto fail = [](cudaError_t e, const char *what) {
        cudaGetLastError();
        set_error(e == cudaErrorMemoryAllocation ? KBWG_ENOMEM : KBWG_ECUDA,
                  std::string("batch circuits: ") + what + ": " + cudaGetErrorString(e));
        return e == cudaErrorMemoryAllocation ? (int32_t)KBWG_ENOMEM : (int32_t)KBWG_ECUDA;
    };
    // plan every circuit (in parallel: the circuits are independent), those of
    // one structure (register size, kinds, targets, controls) once
    std::vector<std::vector<uint64_t>> sigs(circs.size());
    workers.run(circs.size(), [&](size_t c) {
        BatchCircuitIn &ci = circs[c];
        ci.gates = defer_factors(arith, ci.gates.data(), ci.gates.size());
        std::vector<uint64_t> &sig = sigs[c];
        sig.reserve(2 * ci.gates.size() + 1);
        sig.push_back(ci.n);
        for (const GateDesc &g : ci.gates) {
            sig.push_back((uint64_t)g.kind | ((uint64_t)g.target << 8));
            sig.push_back(g.ctrl);
        }
    });
    struct SigHash {
        size_t operator()(const std::vector<uint64_t> *v) const {
            uint64_t h = 1469598103934665603ull;  // FNV-1a over the words
            for (uint64_t w : *v) {
                h ^= w;
                h *= 1099511628211ull;
            }
            return (size_t)h;
        }
    };
    struct SigEqual {
        bool operator()(const std::vector<uint64_t> *a, const std::vector<uint64_t> *b) const { return *a == *b; }
    };
    std::unordered_map<const std::vector<uint64_t> *, size_t, SigHash, SigEqual> known;
    std::vector<size_t> plan_of(circs.size()), first;
    for (size_t c = 0; c < circs.size(); c++) {
        const auto ins = known.emplace(&sigs[c], first.size());
        if (ins.second) first.push_back(c);
        plan_of[c] = ins.first->second;
    }
    std::vector<std::vector<PlannedSweep>> plans(first.size());
    std::vector<char> plan_ok(first.size());
    workers.run(first.size(), [&](size_t k) {
        const BatchCircuitIn &ci = circs[first[k]];
        const uint32_t nplan = std::max<uint32_t>(ci.n, (uint32_t)K);  // small registers padded with |0> qubits
        plans[k] = plan_sweeps(nplan, K, R, ci.gates.data(), ci.gates.size(), false, kMaxSweepGates);
        size_t placed = 0;
        for (PlannedSweep &sw : plans[k]) {
            placed += sw.gates.size();
            merge_signs(sw, K, R);
        }
        plan_ok[k] = placed == ci.gates.size() ? 1 : 0;
    });
    workers.run(circs.size(), [&](size_t c) {
        BatchCircuitIn &ci = circs[c];
        const std::vector<PlannedSweep> &plan = plans[plan_of[c]];
        for (const PlannedSweep &sw : plan) {
            BatchSweep b;
            memset(&b, 0, sizeof b);
            b.l = sw.l;
            b.m = sw.m;
            memcpy(b.hq, sw.hq, sizeof b.hq);
            b.nstages = (uint32_t)sw.stage_layout.size();
            b.gate_count = (uint32_t)sw.gates.size();
            b.data_count = (uint32_t)sw.data.size();
            b.gate_off = (uint32_t)ci.prog.size();  // within the circuit; rebased below
            for (uint32_t i = 0; i < b.nstages; i++) {
                b.stage_layout[i] = sw.stage_layout[i];
                b.stage_end[i] = sw.stage_end[i];
            }
            for (size_t i = 0; i < sw.gates.size(); i++) {
                TileGate t = sw.gates[i];
                if (sw.src[i] != kNoSource) {
                    memcpy(t.c, ci.gates[sw.src[i]].c, sizeof t.c);
                    P::pack_host(t);
                }
                ci.prog.push_back(t);
            }
            ci.prog.insert(ci.prog.end(), sw.data.begin(), sw.data.end());
            ci.sweeps.push_back(b);
        }
        ci.placed = plan_ok[plan_of[c]] != 0;
        if (ci.sweeps.empty() && ci.n > (uint32_t)K) {  // no gates: a sweep that writes |0...0>
            BatchSweep b;
            memset(&b, 0, sizeof b);
            b.l = (uint32_t)K;
            b.nstages = 1;
            b.stage_layout[0] = LAYOUT_A;
            ci.sweeps.push_back(b);
        }
        if (ci.n > (uint32_t)K && !ci.terms.empty()) {
            std::vector<uint64_t> xm;
            for (const BatchTerm &t : ci.terms) xm.push_back(t.x);
            std::vector<size_t> wide;
            const std::vector<PauliPass> pp = plan_pauli_passes(ci.n, K, xm, (size_t)-1, wide);
            for (const PauliPass &ps : pp) {
                BatchPass b;
                memset(&b, 0, sizeof b);
                b.l = ps.l;
                b.m = ps.m;
                memcpy(b.hq, ps.hq, sizeof b.hq);
                b.term_off = (uint32_t)ci.tterms.size();  // within the circuit; rebased below
                std::vector<BatchTileTerm> ts;
                for (size_t k : ps.members) {
                    const BatchTerm &t = ci.terms[k];
                    BatchTileTerm q;
                    memset(&q, 0, sizeof q);
                    q.xl = ps.local(t.x);
                    q.zl = ps.local(t.z & ps.tile_mask);
                    q.zo = t.z & ~ps.tile_mask;
                    q.cr = t.cr;
                    q.ci = t.ci;
                    ts.push_back(q);
                }
                std::stable_sort(ts.begin(), ts.end(), [](const BatchTileTerm &x, const BatchTileTerm &y) {
                    if (x.xl != y.xl) return x.xl < y.xl;
                    if (x.cr != y.cr) return x.cr < y.cr;
                    return x.ci < y.ci;
                });
                for (size_t j = 0; j < ts.size(); j++) {
                    const bool end = j + 1 == ts.size() || ts[j + 1].xl != ts[j].xl || ts[j + 1].cr != ts[j].cr ||
                                     ts[j + 1].ci != ts[j].ci;
                    ts[j].last = end ? 1u : 0u;
                }
                b.nterms = (uint32_t)ts.size();
                ci.tterms.insert(ci.tterms.end(), ts.begin(), ts.end());
                ci.passes.push_back(b);
            }
            std::vector<BatchTerm> rest;  // (wide keeps the flip-mask order)
            for (size_t k : wide) rest.push_back(ci.terms[k]);
            ci.terms.swap(rest);
        }
    });
    // lay the programs out one after another: offsets first, then the copies
    // (in parallel again) into arrays sized once
    std::vector<BatchJob> jobs(circs.size());
    size_t nsweeps = 0, nprog = 0, nterms = 0, npass = 0, ntt = 0;
    std::vector<uint32_t> tt_off(circs.size());
    uint32_t nmax = 0;
    for (size_t c = 0; c < circs.size(); c++) {
        const BatchCircuitIn &ci = circs[c];
        if (!ci.placed) {
            set_error(KBWG_EINVAL, "batch circuits: the planner could not place a circuit's gates");
            return KBWG_EINVAL;
        }
        BatchJob &j = jobs[c];
        memset(&j, 0, sizeof j);
        j.n = ci.n;
        j.id = (uint32_t)c;
        j.sweep_off = (uint32_t)nsweeps;
        j.nsweeps = (uint32_t)ci.sweeps.size();
        j.term_off = (uint32_t)nterms;
        j.nterms = (uint32_t)ci.terms.size();
        j.pad = (uint32_t)nprog;  // the circuit's first gate, for the copies below
        j.pass_off = (uint32_t)npass;
        j.npasses = (uint32_t)ci.passes.size();
        tt_off[c] = (uint32_t)ntt;
        nsweeps += ci.sweeps.size();
        nprog += ci.prog.size();
        nterms += ci.terms.size();
        npass += ci.passes.size();
        ntt += ci.tterms.size();
        nmax = std::max(nmax, ci.n);
    }
    if (nprog > UINT32_MAX || nsweeps > UINT32_MAX || nterms > UINT32_MAX || ntt > UINT32_MAX) {
        set_error(KBWG_EINVAL, "batch circuits: more than 2^32 planned gates, sweeps or strings");
        return KBWG_EINVAL;
    }
    std::unique_ptr<BatchSweep[]> sweeps(new BatchSweep[std::max<size_t>(nsweeps, 1)]);
    std::unique_ptr<TileGate[]> prog(new TileGate[std::max<size_t>(nprog, 1)]);
    std::unique_ptr<BatchTerm[]> terms(new BatchTerm[std::max<size_t>(nterms, 1)]);
    std::unique_ptr<BatchPass[]> passes(new BatchPass[std::max<size_t>(npass, 1)]);
    std::unique_ptr<BatchTileTerm[]> tterms(new BatchTileTerm[std::max<size_t>(ntt, 1)]);
    workers.run(circs.size(), [&](size_t c) {
        BatchCircuitIn &ci = circs[c];
        BatchJob &j = jobs[c];
        const uint32_t base = j.pad;
        j.pad = 0;
        for (size_t i = 0; i < ci.sweeps.size(); i++) {
            BatchSweep b = ci.sweeps[i];
            b.gate_off += base;
            sweeps[j.sweep_off + i] = b;
        }
        if (!ci.prog.empty()) memcpy(&prog[base], ci.prog.data(), ci.prog.size() * sizeof(TileGate));
        if (!ci.terms.empty()) memcpy(&terms[j.term_off], ci.terms.data(), ci.terms.size() * sizeof(BatchTerm));
        for (size_t i = 0; i < ci.passes.size(); i++) {
            BatchPass b = ci.passes[i];
            b.term_off += tt_off[c];
            passes[j.pass_off + i] = b;
        }
        if (!ci.tterms.empty())
            memcpy(&tterms[tt_off[c]], ci.tterms.data(), ci.tterms.size() * sizeof(BatchTileTerm));
    });
    // largest first (the queue's order within a sweep)
    std::vector<uint32_t> order(jobs.size());
    for (size_t k = 0; k < order.size(); k++) order[k] = (uint32_t)k;
    std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) {
        const BatchJob &jx = jobs[x], &jy = jobs[y];
        const double cx = (double)(1ull << jx.n) * (1.0 + jx.nsweeps + 0.25 * jx.nterms);
        const double cy = (double)(1ull << jy.n) * (1.0 + jy.nsweeps + 0.25 * jy.nterms);
        return cx > cy;
    });
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = ensure_smem_limit((const void *)k_batch_circuits<P, K, R>, BK::kSmem);
    if (e != cudaSuccess) return fail(e, "setup");
    int occ = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_batch_circuits<P, K, R>, BK::kThreads, BK::kSmem);
    if (e != cudaSuccess) return fail(e, "occupancy");
    const size_t max_grid = (size_t)sms * std::max(occ, 1);
    // Rounds: the circuits whose states are in memory together.  A round
    // takes circuits until their states reach the room (at least one).
    const uint64_t slot = nmax > (uint32_t)K ? (1ull << nmax) : 0;
    size_t free_b = 0, total_b = 0;
    e = cudaMemGetInfo(&free_b, &total_b);
    if (e != cudaSuccess) return fail(e, "memory query");
    const uint64_t room =
        std::max<uint64_t>(slot, std::min<uint64_t>(kBatchStateBytes, free_b / 10 * 8) / sizeof(Mem));
    std::vector<size_t> round_end;
    uint64_t state_elems = 0;
    {
        uint64_t used = 0;
        for (size_t k = 0; k < order.size(); k++) {
            BatchJob &j = jobs[order[k]];
            if (j.n <= (uint32_t)K) continue;
            if (used + (1ull << j.n) > room) {
                round_end.push_back(k);
                used = 0;
            }
            j.state_off = used;
            used += 1ull << j.n;
            state_elems = std::max(state_elems, used);
        }
        round_end.push_back(order.size());
    }
    // the queue: per round, sweep by sweep over its large circuits, then their
    // <H> parts, then the circuits that stay on one SM
    std::vector<BatchTask> tasks;
    std::vector<BatchItem> items;
    std::vector<size_t> round_items;
    uint64_t nparts = 0;
    {
        size_t k0 = 0;
        for (size_t ke : round_end) {
            std::vector<uint32_t> large, small;
            for (size_t k = k0; k < ke; k++) (jobs[order[k]].n > (uint32_t)K ? large : small).push_back(order[k]);
            k0 = ke;
            auto add = [&](uint32_t jx, uint32_t kind, uint32_t index, uint32_t per, uint32_t parts, uint32_t sl) {
                BatchJob &j = jobs[jx];
                tasks.push_back(BatchTask{jx, kind, index, 0, per, sl});
                for (uint32_t p = 0; p < parts; p++) items.push_back(BatchItem{(uint32_t)tasks.size() - 1, p});
                j.items += parts;
            };
            uint32_t deepest = 0;
            for (uint32_t jx : large) deepest = std::max(deepest, jobs[jx].nsweeps);
            for (uint32_t sw = 0; sw < deepest; sw++)
                for (uint32_t jx : large) {
                    BatchJob &j = jobs[jx];
                    if (sw >= j.nsweeps) continue;
                    const uint32_t tiles = 1u << (j.n - K), per = std::min(8u, std::max(1u, tiles / 32u));
                    const uint32_t need = j.items;
                    add(jx, BT_SWEEP, sw, per, (tiles + per - 1) / per, 0);
                    tasks.back().need = need;
                }
            for (uint32_t jx : large) {
                BatchJob &j = jobs[jx];
                const uint32_t need = j.items, tiles = 1u << (j.n - K), per = std::min(8u, std::max(1u, tiles / 32u));
                j.part_off = (uint32_t)nparts;
                for (uint32_t p = 0; p < j.npasses; p++) {
                    const uint32_t parts = (tiles + per - 1) / per;
                    add(jx, BT_PASS, p, per, parts, j.nparts);
                    tasks.back().need = need;
                    j.nparts += parts;
                }
                if (j.nterms) {  // strings too wide for a tile: 2^K amplitudes per part
                    add(jx, BT_WIDE, 0, (uint32_t)K, tiles, j.nparts);
                    tasks.back().need = need;
                    j.nparts += tiles;
                }
                nparts += j.nparts;
            }
            for (uint32_t jx : small) add(jx, BT_WHOLE, 0, 0, 1, 0);
            round_items.push_back(items.size());
        }
    }
    if (items.size() > UINT32_MAX || nparts > UINT32_MAX) {
        set_error(KBWG_EINVAL, "batch circuits: more than 2^32 work items");
        return KBWG_EINVAL;
    }
    auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t jb = jobs.size() * sizeof(BatchJob), swb = std::max<size_t>(nsweeps, 1) * sizeof(BatchSweep),
                 pb = std::max<size_t>(nprog, 1) * sizeof(TileGate),
                 tb = std::max<size_t>(nterms, 1) * sizeof(BatchTerm), eb = circs.size() * sizeof(double),
                 pab = std::max<size_t>(npass, 1) * sizeof(BatchPass),
                 ttb = std::max<size_t>(ntt, 1) * sizeof(BatchTileTerm),
                 tkb = std::max<size_t>(tasks.size(), 1) * sizeof(BatchTask),
                 itb = std::max<size_t>(items.size(), 1) * sizeof(BatchItem),
                 ptb = std::max<size_t>((size_t)nparts, 1) * sizeof(double),
                 cb = (jobs.size() + round_items.size()) * sizeof(unsigned);
    const size_t o_sw = up(jb), o_p = o_sw + up(swb), o_t = o_p + up(pb), o_pa = o_t + up(tb), o_tt = o_pa + up(pab),
                 o_tk = o_tt + up(ttb), o_it = o_tk + up(tkb), o_pt = o_it + up(itb), o_e = o_pt + up(ptb),
                 o_c = o_e + up(eb), o_err = o_c + up(cb), o_s = o_err + 256;
    cudaStream_t st = nullptr;
    e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (e != cudaSuccess) return fail(e, "stream");
    char *dbuf = nullptr;
    size_t dcap = 0;
    e = batch_take(dev, o_s + (size_t)state_elems * sizeof(Mem), &dbuf, &dcap);
    if (e != cudaSuccess) {
        cudaStreamDestroy(st);
        return fail(e, "buffers");
    }
    BatchArgs a;
    memset(&a, 0, sizeof a);
    a.jobs = (const BatchJob *)dbuf;
    a.tasks = (const BatchTask *)(dbuf + o_tk);
    a.done = (unsigned *)(dbuf + o_c);
    a.partials = (double *)(dbuf + o_pt);
    a.sweeps = (const BatchSweep *)(dbuf + o_sw);
    a.prog = (const TileGate *)(dbuf + o_p);
    a.terms = (const BatchTerm *)(dbuf + o_t);
    a.energies = (double *)(dbuf + o_e);
    a.states = dbuf + o_s;
    a.err = (int *)(dbuf + o_err);
    a.passes = (const BatchPass *)(dbuf + o_pa);
    a.tterms = (const BatchTileTerm *)(dbuf + o_tt);
    int err_flag = 0;
    e = copy_async(dbuf, jobs.data(), jb, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess && nsweeps)
        e = copy_async(dbuf + o_sw, sweeps.get(), nsweeps * sizeof(BatchSweep), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess && nprog)
        e = copy_async(dbuf + o_p, prog.get(), nprog * sizeof(TileGate), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess && nterms)
        e = copy_async(dbuf + o_t, terms.get(), nterms * sizeof(BatchTerm), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess && npass)
        e = copy_async(dbuf + o_pa, passes.get(), npass * sizeof(BatchPass), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess && ntt)
        e = copy_async(dbuf + o_tt, tterms.get(), ntt * sizeof(BatchTileTerm), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = copy_async(dbuf + o_tk, tasks.data(), tasks.size() * sizeof(BatchTask), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = copy_async(dbuf + o_it, items.data(), items.size() * sizeof(BatchItem), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(dbuf + o_c, 0, up(cb) + 256, st);
    size_t i0 = 0;
    for (size_t r = 0; r < round_items.size() && e == cudaSuccess; r++) {
        a.items = (const BatchItem *)(dbuf + o_it) + i0;
        a.nitems = (uint32_t)(round_items[r] - i0);
        a.next = a.done + jobs.size() + r;
        i0 = round_items[r];
        if (a.nitems == 0) continue;
        const uint32_t grid = (uint32_t)std::min<size_t>(a.nitems, max_grid);
        k_batch_circuits<P, K, R><<<grid, BK::kThreads, BK::kSmem, st>>>(a);
        count_launch();
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = copy_async(energies, a.energies, eb, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = copy_async(&err_flag, a.err, sizeof(int), cudaMemcpyDeviceToHost, st);
    const cudaError_t es = cudaStreamSynchronize(st);  // (also after a failure: the buffer goes back idle)
    if (e == cudaSuccess) e = es;
    if (e == cudaSuccess) batch_give(dev, dbuf, dcap);
    else cudaFree(dbuf);
    cudaStreamDestroy(st);
    if (e != cudaSuccess) return fail(e, "run");
    if (err_flag) {
        set_error(KBWG_ETIMEOUT, "batch circuits: a bounded device-side wait ran out");
        return KBWG_ETIMEOUT;
    }
    return KBWG_OK;
}

constexpr uint32_t kBatchMaxQubits = 24;

int32_t batch_circuits(int precision, uint32_t flags, size_t ncirc, const uint32_t *num_qubits, const kbwg_gate *gates,
                       const uintptr_t *gate_offsets, const uint8_t *paulis, const uintptr_t *qubits,
                       const uintptr_t *term_offsets, const double *coefficients, const uintptr_t *ham_offsets,
                       double *energies) {
    std::vector<BatchCircuitIn> circs(ncirc);
    BatchWorkers workers((size_t)(gate_offsets[ncirc] > gate_offsets[0] ? gate_offsets[ncirc] - gate_offsets[0] : 0));
    workers.run(ncirc, [&](size_t c) {
        BatchCircuitIn &ci = circs[c];
        auto bad = [&](int32_t code, const char *msg) {
            ci.status = code;
            ci.error = msg;
        };
        const uint32_t n = num_qubits[c];
        if (n < 1 || n > kBatchMaxQubits) return bad(KBWG_EQUBITS, "batch circuits: every circuit needs 1..24 qubits");
        ci.n = n;
        if (gate_offsets[c + 1] < gate_offsets[c] || ham_offsets[c + 1] < ham_offsets[c])
            return bad(KBWG_EINVAL, "batch circuits: offsets must not decrease");
        ci.gates.reserve(gate_offsets[c + 1] - gate_offsets[c]);
        for (uintptr_t i = gate_offsets[c]; i < gate_offsets[c + 1]; i++) {
            const kbwg_gate &g = gates[i];
            if (g.kind > KBWG_RZ || g.target >= n || (g.control_mask >> n) || (g.control_mask & (1ull << g.target)))
                return bad(KBWG_EINVAL, "batch circuits: bad gate (kind, target or controls)");
            ci.gates.push_back(make_gate_desc(precision, g.kind, g.target, g.control_mask, g.angle));
        }
        ci.terms.reserve(ham_offsets[c + 1] - ham_offsets[c]);
        for (uintptr_t k = ham_offsets[c]; k < ham_offsets[c + 1]; k++) {
            BatchTerm t;
            memset(&t, 0, sizeof t);
            int ny = 0;
            if (term_offsets[k + 1] < term_offsets[k]) return bad(KBWG_EINVAL, "batch circuits: offsets must not decrease");
            for (uintptr_t i = term_offsets[k]; i < term_offsets[k + 1]; i++) {
                if (qubits[i] >= n || paulis[i] < 1 || paulis[i] > 3)
                    return bad(KBWG_EINVAL, "batch circuits: bad Pauli code or qubit");
                const uint64_t b = 1ull << qubits[i];
                if ((t.x | t.z) & b) return bad(KBWG_EINVAL, "batch circuits: a string names a qubit twice");
                if (paulis[i] == 1) t.x |= b;
                else if (paulis[i] == 2) t.x |= b, t.z |= b, ny++;
                else t.z |= b;
            }
            static const double re[4] = {1, 0, -1, 0}, im[4] = {0, 1, 0, -1};
            t.cr = coefficients[k] * re[ny & 3];
            t.ci = coefficients[k] * im[ny & 3];
            ci.terms.push_back(t);
        }
        std::stable_sort(ci.terms.begin(), ci.terms.end(),
                         [](const BatchTerm &x, const BatchTerm &y) { return x.x < y.x; });
    });
    for (const BatchCircuitIn &ci : circs)  // the first bad circuit's error
        if (ci.status != KBWG_OK) {
            set_error(ci.status, ci.error);
            return ci.status;
        }
    if (ncirc == 0) return KBWG_OK;
    if (precision == KBWG_C64) return batch_run<FastP, 12, 4>(ARITH_C64, workers, circs, energies);
    if (flags & KBWG_FLAG_FAST_C128) return batch_run<FF2B, 11, 3>(ARITH_FF, workers, circs, energies);
    return batch_run<Fast<double>, 11, 3>(ARITH_F64, workers, circs, energies);
}

}  // namespace kbwg
