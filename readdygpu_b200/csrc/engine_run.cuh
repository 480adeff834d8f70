// engine_run.cuh -- the pair-list steps of one rdgpu_step call in one launch.
//
// list_run_kernel advances a handle by up to nsteps steps: a cooperative grid
// (all blocks resident) steps every particle, meets at a grid barrier, and
// goes on with the next step; the list check of a step runs together with the
// next step, and the re-sort and list build run inside the same kernel when
// they are due.  Launched step by step (list_step_kernel, list_check_kernel
// and a conditional graph node per step), 8 to 40 us of every step went to
// launch gaps, the check's own launch and the conditional node: more than the
// step itself up to about a million particles.  Per step, launch by launch
// and in one launch (tuned, calls of 100 steps, rebuilds and the host's wait
// included): 1,000 particles FP64 20.5 and 5.8 us, 20,000 FP64 23.0 and 6.7,
// 250,000 (vesicle, FP32C) 52.4 and 30.5, 370,000 FP64 in 64 systems 53.5 and
// 33.2, 2.9 M in 512 systems 152 and 126 (there the step and the list build
// are bound by issue).
//
// The before-and-after figures at the parts below are of the builds in which
// each part was taken (skin 1.4), one after the other: they price the part,
// and are not the times of the kernel as it stands.
#pragma once
#include "engine_kernels.cuh"

namespace rdgpu {

// Control words of one launch, zero at its start.  A launch zeroes the next
// one's (two of them alternate), so no memset is queued per call.
struct RunCtl {
    unsigned long long bar[3];    // a grid barrier's arrivals and flags (run_sync), used in turn
    int nhot[3], err[3];          // per step attempt, used in turn
    int lerr, maxcnt;             // list build: EF_LIST*, longest list
};

// The launch's outcome, written to page-locked host memory by its last act.
struct RunOut {
    int err;        // EF_*: of step t (its input is intact), or of the build for step t's input
    int dead;       // a barrier wait ran out: the state is undefined
    int sel;        // the buffer that holds the input of step t
    int builds;     // list builds in this launch
    int maxcnt;     // longest list met by an overflowing build
    int pad;
    long long t;    // the next step to compute
};

constexpr int RUN_REBUILD = 1;
constexpr int RUN_REBUILD_INPUT = 2;   // the same, unless a.err says that the upload was rejected

template <class R> struct RunArgs {
    Args<R> a;
    ListArgs<R> v;
    RunCtl* ctl;
    RunCtl* next;      // the next launch's, zeroed by this one
    RunOut* out;
    int* tile_sum;     // one per scan tile (run_scan_tile cells each)
    long long ncells;
    long long t0;      // first step
    int nsteps;
    int sel0;          // the buffer that holds its input
    int rebuild;       // RUN_REBUILD: re-sort and build the lists first
};

// Threads per block, at most; one block per SM.  Its warps draw the SM's tiles
// from one counter, and 148 blocks arrive at the grid barrier: against 3 blocks
// of 384 (FP32C repulsion), 2 of 512 (FP32C) or 2 of 448 and 384 (FP64) 135 ->
// 130 us a step on 2.9 M particles in 512 systems, 39.4 -> 35.1 us on 250,000
// (vesicle), 36.0 -> 34.7 us on 370,000 FP64 in 64 systems and 25.9 -> 21.0 us
// on 60,000 FP64 (vesicle).  64 registers a thread FP32, 72 and 80 FP64.
template <class R, bool HREP, bool ALLPER> struct RunShape {
    static constexpr int BLOCK = sizeof(R) == 4 ? 1024 : (HREP && ALLPER ? 896 : 768);
};

// HOME > 0, for up to HOME tiles per SM (narrow lists): a warp keeps one tile
// for the whole launch, its particles' state and first list groups in
// registers, reads only partners from memory, and draws the next step's noise
// while the barrier completes; 3 or 4 more warps check the hot particles.  Per
// step, tiles read anew and kept: 1,000 particles FP64 9.8 and 7.3 us, FP32C
// 7.6 and 6.0, 20,000 FP64 11.2 and 8.6, 30,000 FP32C 8.7 and 7.4, 60,000 FP64
// (vesicle) 21.3 and 18.7 us.  Two sizes, 168 and 128 registers a thread: 13
// for all costs the small ones 2 to 5 %; 22 (80 registers) is no gain.
constexpr int RUN_HOME_FEW = 8;
constexpr int RUN_HOME_MANY = 13;
constexpr int run_home_block(int home) { return home == RUN_HOME_FEW ? 384 : 512; }
// HOME = RUN_RANK, for several tiles per warp and more than harmonic repulsion: a
// block takes its dearest tiles first, so that none of them is left for the end
// of the step.  Tiles of a vesicle's shell cost up to twice the mean: 250,000
// particles (FP32C) 31.9 -> 29.7 us a step.  With repulsion alone the costs are
// even and the neighbours in memory matter more: 2.9 M particles 125 -> 143 us.
constexpr int RUN_RANK = -1;
template <class R> constexpr int RUN_HOME_CHUNK = sizeof(R) == 4 ? 8 : 4;   // partners requested together

// a wait at the grid barrier gives up after this many polls (some seconds)
constexpr unsigned RUN_POLLS = 1u << 23;

constexpr int RUN_ORDER = 1024;       // tiles of a block that are ordered by cost, at most
constexpr int RUN_SCAN_PER = 8;       // cells per thread and scan tile

// dynamic shared memory: the squared list radii, list_build_one's scratch, then
// (HOME without HREP) the terms of the type pairs in use
extern __shared__ __align__(16) char run_dyn[];
template <class R> __host__ __device__ constexpr size_t run_dyn_bytes(int block)
{
    return MAXT * MAXT * sizeof(R) + (size_t)block * LB_BYTES;
}
template <class R> constexpr size_t run_term_bytes(int S)
{
    return (size_t)((S * S + 3) & ~3) * sizeof(int) + (size_t)S * S * MAX_TERMS * sizeof(PairTerm<R>);
}

__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long* p)
{
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void red_release(unsigned long long* p, unsigned long long v)
{
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" : : "l"(p), "l"(v) : "memory");
}

// what a block found since the last grid barrier
constexpr unsigned RF_HOT = 1;        // hot particles
constexpr unsigned RF_NEED = 2;       // a particle that moved too far
constexpr unsigned RF_FAIL = 4;       // a pair missing from the lists
constexpr unsigned RF_ERR = 8;        // an error (step or list build)

// block-wide words of list_run_kernel
struct RunShared {
    unsigned mine;    // RF_* of this block since the last barrier
    unsigned flags;   // RF_* of any block, as of the last barrier
    int dead;         // a barrier wait ran out
    int nhot, err;    // hot particles and errors of the attempt, read when flagged
    int next;         // next work item of the block
    int bars;         // grid barriers passed
    int warp[32];     // block scan
    int own;          // RANK: tiles of the block; ordered by cost; worth it
    int sorted, rankable;
};

// Grid barrier: everything written before it by any block is visible after it
// to plain loads of every block (release by the arriving thread after the
// block's barrier, acquire before the block's second one).  A block arrives
// with one addition that counts it and carries its flags in fields of their
// own (16 bits of arrivals, then 12 bits per flag), so that the poll that sees
// the last arrival has the flags too; the counter of the barrier after this
// one was last polled before this one's predecessor, and is cleared here.  The
// block's work counter restarts.  False when the wait ran out (every block then
// leaves the kernel).  Every thread calls meanwhile() between the block's
// arrival and the wait.  Against two fences, a 32-bit counter and four flags
// read after it, a step of 1,000 particles (FP64) 6.4 -> 5.9 us, of 20,000 7.4
// -> 6.8 us, of 100,000 (mixed, FP32C) 20.6 -> 19.1 us.
template <class F>
__device__ __forceinline__ bool run_sync(RunCtl* c, RunShared& sh, int slot, F&& meanwhile)
{
    const bool leader = threadIdx.x == blockDim.x - 32;      // of the last warp (HOME: without a tile)
    __syncthreads();
    const int k = sh.bars % 3;
    if (leader) {
        const unsigned f = sh.mine;
        if (blockIdx.x == 0) c->bar[k == 2 ? 0 : k + 1] = 0;
        red_release(&c->bar[k], 1ull | (unsigned long long)(f & 1u) << 16 | (unsigned long long)(f >> 1 & 1u) << 28 |
                                    (unsigned long long)(f >> 2 & 1u) << 40 | (unsigned long long)(f >> 3 & 1u) << 52);
    }
    meanwhile();
    if (leader) {
        unsigned polls = 0;
        unsigned long long v;
        while (((v = ld_acquire(&c->bar[k])) & 0xffffu) != gridDim.x && ++polls < RUN_POLLS) {}
        const unsigned f = ((v >> 16 & 0xfffu) ? RF_HOT : 0u) | ((v >> 28 & 0xfffu) ? RF_NEED : 0u) |
                           ((v >> 40 & 0xfffu) ? RF_FAIL : 0u) | ((v >> 52 & 0xfffu) ? RF_ERR : 0u);
        sh.flags = f;
        sh.nhot = (f & RF_HOT) ? *((volatile const int*)&c->nhot[slot]) : 0;
        sh.err = (f & RF_ERR) ? *((volatile const int*)&c->err[slot]) | *((volatile const int*)&c->lerr) : 0;
        sh.dead = polls >= RUN_POLLS;
        sh.mine = 0;
        sh.next = blockDim.x >> 5;
        ++sh.bars;
    }
    __syncthreads();
    return sh.dead == 0;
}
__device__ __forceinline__ bool run_sync(RunCtl* c, RunShared& sh, int slot)
{
    return run_sync(c, sh, slot, [] {});
}

// next work item of the calling warp within its block
__device__ __forceinline__ int run_next(RunShared& sh)
{
    int w = 0;
    if ((threadIdx.x & 31) == 0) w = atomicAdd(&sh.next, 1);
    return __shfl_sync(FULL, w, 0);
}

// The block's q-th tile of 32 particles: single tiles dealt to the blocks in
// turn, and drawn from the block's counter by its warps, so that systems of
// different density spread over all blocks (runs of 8 tiles, for partners
// shared in L1, measured 2 to 4 % slower from 250,000 particles up: the blocks
// then end apart by up to a fifth of a step).
__device__ __forceinline__ int run_tile(int q) { return q * (int)gridDim.x + (int)blockIdx.x; }

// Cell starts from the counts (cleared on the way), as scan_tiles_kernel and
// scan_apply_kernel do in two launches: tile sums, a grid barrier, then each
// tile's exclusive prefix.  A tile is RUN_SCAN_PER cells per thread.
__device__ __forceinline__ bool run_scan(RunCtl* c, RunShared& sh, int* counts, int* start, int* tile_sum,
                                         long long ncells, int slot)
{
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
    const long long per_tile = (long long)blockDim.x * RUN_SCAN_PER;
    const int ntiles = (int)((ncells + per_tile - 1) / per_tile);
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const long long base = tile * per_tile + tid;
        int sum = 0;
#pragma unroll
        for (int k = 0; k < RUN_SCAN_PER; ++k) {
            const long long q = base + (long long)k * blockDim.x;
            if (q < ncells) sum += counts[q];
        }
        sum = __reduce_add_sync(FULL, sum);
        if (lane == 0) sh.warp[wid] = sum;
        __syncthreads();
        if (tid == 0) {
            int tot = 0;
            for (int w = 0; w < nw; ++w) tot += sh.warp[w];
            tile_sum[tile] = tot;
        }
        __syncthreads();
    }
    if (!run_sync(c, sh, slot)) return false;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        int before = 0;
        for (int k = tid; k < tile; k += blockDim.x) before += tile_sum[k];
        // each thread scans RUN_SCAN_PER consecutive cells (32 bytes: whole sectors)
        const long long q0 = tile * per_tile + (long long)tid * RUN_SCAN_PER;
        alignas(16) int v[RUN_SCAN_PER];
        int sum = 0;
        const bool whole = q0 + RUN_SCAN_PER <= ncells;
        if (whole) {
            int4* c4 = reinterpret_cast<int4*>(counts + q0);
            reinterpret_cast<int4*>(v)[0] = c4[0];
            reinterpret_cast<int4*>(v)[1] = c4[1];
            c4[0] = c4[1] = make_int4(0, 0, 0, 0);
        } else {
#pragma unroll
            for (int k = 0; k < RUN_SCAN_PER; ++k) {
                v[k] = 0;
                if (q0 + k < ncells) {
                    v[k] = counts[q0 + k];
                    counts[q0 + k] = 0;
                }
            }
        }
#pragma unroll
        for (int k = 0; k < RUN_SCAN_PER; ++k) sum += v[k];
        const int incl = warp_incl_scan(sum, lane);
        before = __reduce_add_sync(FULL, before);
        if (lane == 31) sh.warp[wid] = incl + before;     // the tiles before, as the warps found them
        __syncthreads();
        // base of this warp: all tiles before (every warp's share) and the
        // warps before it in this tile
        const int mine = __shfl_sync(FULL, incl, 31);
        int all = 0;
        for (int w = 0; w < nw; ++w) {
            const int x = sh.warp[w];
            all += x;
        }
        __syncthreads();
        if (lane == 0) sh.warp[wid] = mine;
        __syncthreads();
        int inside = 0, upto = 0;
        for (int w = 0; w < nw; ++w) {
            const int x = sh.warp[w];
            inside += x;
            if (w < wid) upto += x;
        }
        int run = (all - inside) + upto + incl - sum;
        alignas(16) int o[RUN_SCAN_PER];
#pragma unroll
        for (int k = 0; k < RUN_SCAN_PER; ++k) {
            o[k] = run;
            run += v[k];
            if (q0 + k == ncells - 1) start[ncells] = run;
        }
        if (whole) {
            reinterpret_cast<int4*>(start + q0)[0] = reinterpret_cast<int4*>(o)[0];
            reinterpret_cast<int4*>(start + q0)[1] = reinterpret_cast<int4*>(o)[1];
        } else {
#pragma unroll
            for (int k = 0; k < RUN_SCAN_PER; ++k)
                if (q0 + k < ncells) start[q0 + k] = o[k];
        }
        __syncthreads();
    }
    return true;
}

// Re-sort by cell from src into dst and list build (list_count_kernel ..
// list_build_kernel in one go).  False: a barrier wait ran out.  An
// overflowing build leaves its flags in sh.err (the state in src is intact).
template <class R>
__device__ __noinline__ bool run_rebuild(const RunArgs<R>& p, RunShared& sh, int sel, int slot)
{
    R* s_rl2 = reinterpret_cast<R*>(run_dyn);
    char* scratch = run_dyn + MAXT * MAXT * sizeof(R);
    const Args<R>& a = p.a;
    const State<R> src = sel ? p.v.b1 : p.v.b0;
    const State<R> dst = sel ? p.v.b0 : p.v.b1;
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long first = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    for (long long i = first; i < a.ntot; i += stride) {
        const SysDev& s = a.sys[a.sys_of[i]];
        R x[3];
        int w;
        load_pos<true>(src, i, x, w);
        int c[3];
        cell_coords(s, x, c);
        const long long cell = s.cell_base + ((long long)c[2] * s.n[1] + c[1]) * s.n[0] + c[0];
        a.tslot[i] = atomicAdd(a.counts + cell, 1);
        a.tcell[i] = (int)cell;
    }
    for (int k = threadIdx.x; k < MAXT * MAXT; k += blockDim.x) s_rl2[k] = p.v.rl2t[k];
    if (!run_sync(p.ctl, sh, slot)) return false;
    if (!run_scan(p.ctl, sh, a.counts, const_cast<int*>(a.start), p.tile_sum, p.ncells, slot)) return false;
    if (!run_sync(p.ctl, sh, slot)) return false;
    for (long long i = first; i < a.ntot; i += stride) {
        const long long d = a.start[a.tcell[i]] + a.tslot[i];
        if constexpr (sizeof(R) == 4) {
            const float4 q = src.aux[i];
            dst.pos[d] = src.pos[i];
            dst.aux[d] = q;
            if (a.inv) a.inv[__float_as_int(q.w)] = (int)d;
        } else {
            const Rec64 r = src.rec[i];
            dst.rec[d] = r;
            if (a.inv) a.inv[r.id] = (int)d;
        }
    }
    if (!run_sync(p.ctl, sh, slot)) return false;
    const int lane = threadIdx.x & 31;
    const int tiles = (int)((a.ntot + 31) / 32);
    for (int q = threadIdx.x >> 5;; q = run_next(sh)) {
        const int tile = run_tile(q);
        if (tile >= tiles) break;
        const long long i = (long long)tile * 32 + lane;
        if (i < a.ntot) {
            int cnt;
            const int ef = list_build_one<R, true>(a, p.v, dst, (int)i, s_rl2, scratch, cnt);
            if (ef) {
                if (ef & EF_LISTOVF) atomicMax(&p.ctl->maxcnt, cnt);
                atomicOr(&p.ctl->lerr, ef);
                atomicOr(&sh.mine, RF_ERR);
            }
        }
        __syncwarp();
    }
    return run_sync(p.ctl, sh, slot);
}

// the check of one hot particle by a warp, in the state of buffer sel (for the
// warps without tiles; in the tile kernel, in line before the tiles, which
// measured 2 to 5 % faster there than this call)
template <class R> __device__ __noinline__ bool run_check(const RunArgs<R>& p, int sel, int h)
{
    return hot_pairs_listed<R, true>(p.a, p.v, sel ? p.v.b1 : p.v.b0, h, threadIdx.x & 31);
}

// Up to nsteps pair-list steps.  Step attempt n of the launch reads buffer
// sel and writes the other one; its flags are in slot n % 3 and its hot
// particles in half n & 1 of the hot list.  While it runs, warps check the
// hot particles of the step before it (the state in buffer sel) against the
// lists (list_check_kernel's test).  At the barrier that ends it every block
// takes the same decision:
//   - a pair was missing from the lists: attempt n is void (its input is
//     intact), the input is re-sorted, the lists are built and the step is
//     repeated;
//   - an error: the launch ends with that step's input intact;
//   - else the step stands; if it moved a particle too far (or made too many
//     hot) its result is re-sorted and the lists are built.
// So a step takes one grid barrier, and a pair that the lists miss costs a
// repeated step (about one in 20 to 50).  The forces a repeated step sees are
// those of a step after a separate check: the trajectory does not change.
template <class R, bool HREP, bool ALLPER, bool NARROW, int HOME>
__global__ void __launch_bounds__(HOME > 0 ? run_home_block(HOME) : RunShape<R, HREP, ALLPER>::BLOCK, 1)
    list_run_kernel(const __grid_constant__ RunArgs<R> p)
{
    __shared__ PairTables<R, HREP> s_pt;
    __shared__ __align__(16) char s_ext[HOME > 0 ? MAX_EXT * sizeof(ExtTerm<R>) : 16];
    __shared__ RunShared sh;
    const Args<R>& a = p.a;
    const ListArgs<R>& v = p.v;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int G = gridDim.x, bid = blockIdx.x;
    const int tiles = (int)((a.ntot + 31) / 32);
    if (bid == 0 && threadIdx.x < sizeof(RunCtl) / sizeof(int)) reinterpret_cast<int*>(p.next)[threadIdx.x] = 0;
    if (threadIdx.x == 0) {
        sh.bars = 0;
        sh.mine = 0;
        sh.next = blockDim.x >> 5;
    }
    s_pt.load(a.tab);
    // HOME: the terms of the type pairs in use and a single system's external
    // potentials too, since a barrier drops L1 and each step would wait for
    // them anew (60,000 particles FP64, vesicle: 18.1 -> 16.7 us a step; with
    // many tiles per warp the plain loads measured 2 to 6 % faster)
    const int S = a.tab->S;
    int* s_nterm = reinterpret_cast<int*>(run_dyn + run_dyn_bytes<R>(blockDim.x));
    PairTerm<R>* s_term = reinterpret_cast<PairTerm<R>*>(s_nterm + ((S * S + 3) & ~3));
    const ExtTerm<R>* ext1 = reinterpret_cast<const ExtTerm<R>*>(s_ext);
    if constexpr (HOME > 0) {
        if (!HREP)
            for (int q = threadIdx.x; q < S * S; q += blockDim.x) {
                const int k = (q / S) * MAXT + q % S;
                s_nterm[q] = a.tab->nterm[k];
                for (int m = 0; m < MAX_TERMS; ++m) s_term[q * MAX_TERMS + m] = a.tab->term[k * MAX_TERMS + m];
            }
        if (a.nsys == 1)
            for (int q = threadIdx.x; q < a.n_ext * (int)(sizeof(ExtTerm<R>) / 4); q += blockDim.x)
                reinterpret_cast<int*>(s_ext)[q] = reinterpret_cast<const int*>(a.ext)[q];
    }
    __syncthreads();
    long long t = p.t0;
    int sel = p.sel0, n = 0, slot = 0, builds = 0, nhot = 0, err = 0;
    bool alive = true;
    const long long tend = p.t0 + p.nsteps;
    // HOME: this thread's particle
    const int home_warps = (tiles + G - 1) / G;
    const int hi = (warp * G + bid) * 32 + lane;
    const bool home = HOME > 0 && warp < home_warps && hi < a.ntot;
    bool loaded = false;
    ListIn<R, NARROW, true> hin;
    SysDev hs;
    R hn[3];
    // RANK: the block's tiles by the clock over the first step after each list
    // build (all words in shared memory: the step has no register to spare)
    constexpr bool RANK = HOME == RUN_RANK;
    __shared__ unsigned short s_cost[RANK ? RUN_ORDER : 1], s_order[RANK ? RUN_ORDER : 1];
    __shared__ unsigned s_at[RANK ? 32 : 1];
    __shared__ int s_k[RANK ? 32 : 1];
    if (RANK && threadIdx.x == 0) {
        sh.own = tiles > bid ? (tiles - bid + G - 1) / G : 0;
        sh.sorted = 0;
        sh.rankable = sh.own > (int)(blockDim.x >> 5) && sh.own <= RUN_ORDER;
    }
    if (p.rebuild) {
        err = p.rebuild == RUN_REBUILD_INPUT ? *((volatile const int*)a.err) : 0;
        if (!err) {
            alive = run_rebuild<R>(p, sh, sel, 0);
            err = alive ? sh.err : 0;
            if (alive && !err) {
                sel ^= 1;
                ++builds;
            }
        }
    }
    while (t < tend && alive && !err) {
        const State<R> cur = sel ? v.b1 : v.b0;
        const State<R> nxt = sel ? v.b0 : v.b1;
        const int after = slot == 2 ? 0 : slot + 1;
        if (bid == 0 && threadIdx.x == 0) {
            p.ctl->nhot[after] = 0;
            p.ctl->err[after] = 0;
        }
        const int* hot_in = v.hot + ((n & 1) ^ 1) * v.hot_max;
        int* hot_out = v.hot + (n & 1) * v.hot_max;
        if constexpr (HOME > 0) {
            if (warp >= home_warps) {
                const int spare = (int)(blockDim.x >> 5) - home_warps;
                for (int h = (warp - home_warps) * G + bid; h < nhot; h += spare * G)
                    if (!run_check(p, sel, hot_in[h]) && lane == 0) atomicOr(&sh.mine, RF_FAIL);
            } else if (home) {
                if (!loaded) {
                    hin.load(a, v, cur, hi);
                    hin.q1 = head_count(hin.hd) > 8 ? v.nbr[hi + v.stride] : make_int4(0, 0, 0, 0);
                    hs = a.sys[hin.si];
                    bd_normals(hs.seed, t, (long long)hin.id, hn);
                }
                Acc<R> acc;
                acc.zero();
                list_pairs<R, HREP, NARROW, true, RUN_HOME_CHUNK<R>, true>(a, v, cur, hi, hin, hs, s_pt, s_nterm,
                                                                           s_term, S, acc);
                float dd;
                const int ef = list_move<R, ALLPER>(a, cur, nxt, hi, hin, hs, acc,
                                                    a.nsys == 1 ? ext1 : a.ext + (long long)hin.si * a.n_ext, [&](R* xn) {
                    xn[0] = hn[0]; xn[1] = hn[1]; xn[2] = hn[2];
                }, dd);
                const bool any = list_collect_hot(dd, v.thr2, hi, &p.ctl->nhot[slot], hot_out, v.hot_max);
                if (ef) atomicOr(&p.ctl->err[slot], ef);
                if (any || ef || dd > v.cap2)
                    atomicOr(&sh.mine, (any ? RF_HOT : 0u) | (ef ? RF_ERR : 0u) | (dd > v.cap2 ? RF_NEED : 0u));
            }
            loaded = true;
        } else {
            // work items of this block: its share of the hot particles to
            // check, then its tiles
            const int hb = nhot > bid ? (nhot - bid + G - 1) / G : 0;
            int w = warp;
            for (; w < hb; w = run_next(sh))
                if (!hot_pairs_listed<R, true>(a, v, cur, hot_in[w * G + bid], lane) && lane == 0)
                    atomicOr(&sh.mine, RF_FAIL);
            for (;; w = run_next(sh)) {
                int k = w - hb;
                if constexpr (RANK) {
                    if (sh.sorted) {
                        if (k >= sh.own) break;
                        k = s_order[k];
                    }
                    if (lane == 0) {
                        s_at[warp] = (unsigned)clock();
                        s_k[warp] = k;
                    }
                }
                const int tile = run_tile(k);
                if (tile >= tiles) break;
                const int i = tile * 32 + lane;
                if (i < a.ntot) {
                    ListIn<R, NARROW, true> in;
                    in.load(a, v, cur, i);
                    float dd;
                    const int ef = list_step_one<R, HREP, ALLPER, NARROW, true>(
                        a, v, cur, nxt, i, in, t, s_pt, a.tab->nterm, a.tab->term, MAXT,
                        a.ext + (long long)in.si * a.n_ext, dd);
                    const bool any = list_collect_hot(dd, v.thr2, i, &p.ctl->nhot[slot], hot_out, v.hot_max);
                    if (ef) atomicOr(&p.ctl->err[slot], ef);
                    if (any || ef || dd > v.cap2)
                        atomicOr(&sh.mine, (any ? RF_HOT : 0u) | (ef ? RF_ERR : 0u) | (dd > v.cap2 ? RF_NEED : 0u));
                }
                __syncwarp();
                if (RANK && lane == 0 && s_k[warp] < RUN_ORDER)
                    s_cost[s_k[warp]] = (unsigned short)min(((unsigned)clock() - s_at[warp]) >> 5, 65535u);
            }
        }
        alive = run_sync(p.ctl, sh, slot, [&] {
            if (HOME > 0 && home) bd_normals(hs.seed, t + 1, (long long)hin.id, hn);
        });
        if (!alive) break;
        if (RANK && sh.rankable && !sh.sorted) {
            const int own = sh.own;
            for (int k = threadIdx.x; k < own; k += blockDim.x) {
                const int c = s_cost[k];
                int r = 0;
                for (int o = 0; o < own; ++o) {
                    const int d = s_cost[o];
                    r += d > c || (d == c && o < k);
                }
                s_order[r] = (unsigned short)k;
            }
            __syncthreads();
            if (threadIdx.x == 0) sh.sorted = 1;
            __syncthreads();
        }
        const bool fail = (sh.flags & RF_FAIL) != 0, need = (sh.flags & RF_NEED) != 0;
        const int found = sh.nhot;
        err = sh.err;
        ++n;
        slot = after;
        nhot = 0;
        bool rebuild = fail;
        if (fail) {
            err = 0;
        } else {
            if (err) break;
            ++t;
            sel ^= 1;
            rebuild = need || found > v.hot_max;
            if (!rebuild) nhot = found;
        }
        if (!rebuild && t == tend && nhot > 0) {
            // the last step's hot particles
            hot_in = v.hot + ((n & 1) ^ 1) * v.hot_max;
            for (int h = warp * G + bid; h < nhot; h += G * (int)(blockDim.x >> 5))
                if (!run_check(p, sel, hot_in[h]) && lane == 0) atomicOr(&sh.mine, RF_FAIL);
            alive = run_sync(p.ctl, sh, slot);
            if (!alive) break;
            rebuild = (sh.flags & RF_FAIL) != 0;
        }
        if (rebuild) {
            nhot = 0;
            alive = run_rebuild<R>(p, sh, sel, slot);
            if (!alive) break;
            err = sh.err;
            if (err) break;
            sel ^= 1;
            loaded = false;
            if (RANK && threadIdx.x == 0) sh.sorted = 0;
            __syncthreads();
            ++builds;
        }
    }
    if (bid == 0 && threadIdx.x == 0) {
        volatile RunOut* o = p.out;
        o->err = err;
        o->dead = alive ? 0 : 1;
        o->sel = sel;
        o->builds = builds;
        o->maxcnt = *((volatile int*)&p.ctl->maxcnt);
        o->t = t;
    }
}

}  // namespace rdgpu
