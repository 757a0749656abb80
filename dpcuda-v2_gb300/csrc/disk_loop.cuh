// disk_loop.cuh -- the NVE and FIRE loops of a disk system as one resident
// grid: a cooperative launch whose blocks run many iterations, separated by
// grid barriers, instead of a CUDA graph with three kernels and two
// conditional nodes an iteration.
//
// What bounds the graph loop at 10^2 - 10^5 disks is neither memory nor
// arithmetic but its nodes: ~25 us of an iteration's 32 - 40 us pass between
// the kernels (measured: NVE of 1024 disks 38.6 us a step as a graph, 7.3 us
// here; of 10007 mixed 36 -> 7; FIRE of 16384 disks 71 -> 20 us an iteration).
// Here an NVE step costs one barrier (the kick that ends a step,
// the next step's kick and its drift run in the same pass, into the other of
// two position buffers) and a FIRE iteration two (its power decides the next
// move).  Per-particle arithmetic is that of the graph loop's kernels.
//
// Every block keeps a copy of the control state and takes the same decisions
// from the same totals (block partials summed in block order); block 0 writes
// the state back.  Block b owns the slots [b * chunk, (b + 1) * chunk).  Data
// that other blocks write is read with ordinary loads after a barrier (the
// acquire of the barrier's last poll, then __syncthreads); nothing here may be
// read through the non-coherent path.  The waits of the grid barrier through L2
// are bounded: a block whose barrier does not complete closes it, so that it
// fails for every block alike and none goes on with data that another has not
// written; all leave, and the call returns DPG_ERR_TIMEOUT.  A grid of one
// cluster uses the hardware's cluster barrier, which has no limit (its blocks
// are all resident or none is).
#pragma once
#include <cooperative_groups.h>

#include "disk_kernels.cuh"

namespace dpg {
namespace {

constexpr int kLoopMaxTPB = 512;
constexpr int kClusterMax = 16;      // blocks of a cluster at most
constexpr int kLoopBlocksMax = 160;  // blocks of a FIRE loop at most
constexpr int kBarPolls = 1 << 22;   // ~1 s of polls (DPG_LOOP_POLLS sets another limit)

struct LoopSync {
    unsigned long long ring[4];  // barrier k uses ring[k & 3]: arrivals and flag counts
    int err;                     // a barrier failed: read by block 0 as it leaves
    int max_count;               // longest neighbour row of the last list build
    int max_vcount;              // longest vertex row (rigid bodies)
};

// what a barrier carries besides the arrival count (bits 0 - 15): how many
// blocks raised each flag
constexpr unsigned long long kNeedList = 1ULL << 16, kNeedCell = 1ULL << 32, kFull = 1ULL << 48;
constexpr unsigned long long kClosed = 1ULL << 15;  // the barrier failed: above every count of arrivals
__device__ __forceinline__ bool raised(unsigned long long v, unsigned long long flag) {
    return (v / flag & 0xffff) != 0;
}

// Grid barrier k; flags of thread 0 are added to the arrival; polls: how often a
// wait looks (a launch argument, passed by value: kept beside k behind a reference
// it cost a FIRE iteration of 16384 disks 0.5 %).  Returns the
// completed word (arrivals and flag counts) on every thread, 0 if the barrier
// failed.  A block whose polls run out closes the word by compare-and-swap, which
// succeeds only while arrivals are missing, and a closed word stays so: a
// barrier completes for all blocks or fails for all.  Barrier k + 2's word is
// cleared by block 0 once barrier k is complete: every block has then left
// barrier k - 2, the word's last use, and reaches k + 2 only after block 0's
// arrival at k + 1.
// A grid of one thread-block cluster uses the cluster's barrier, the flags going
// to every block's shared memory before it (two sets in turn: a block that
// writes one again has passed a barrier that its readers entered later).
__device__ __forceinline__ unsigned long long grid_bar(LoopSync *ls, unsigned &k, int polls, unsigned long long flags) {
    __shared__ unsigned long long done, said[2][kClusterMax];
    const auto cluster = cooperative_groups::this_cluster();
    if (cluster.num_blocks() > 1) {
        const int nb = (int)cluster.num_blocks(), t = threadIdx.x;
        flags = __shfl_sync(0xffffffffu, flags, 0);
        if (t < nb) *cluster.map_shared_rank(&said[k & 1][cluster.block_rank()], t) = 1ULL + flags;
        cluster.sync();
        if (t < 32) {
            unsigned long long v = t < nb ? said[k & 1][t] : 0;
#pragma unroll
            for (int o = kClusterMax / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (t == 0) done = v;
        }
        __syncthreads();
        k++;
        return done;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long *w = &ls->ring[k & 3], v;
        __threadfence();
        atomicAdd(w, 1ULL + flags);
        int n = 0;
        do {
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(w) : "memory");
        } while ((v & 0xffff) < gridDim.x && ++n < polls);
        if ((v & 0xffff) != gridDim.x) {  // run out, or closed
            while ((v & 0xffff) < gridDim.x) {  // another arrival makes it look again
                const unsigned long long seen = atomicCAS(w, v, v | kClosed);
                v = seen == v ? v | kClosed : seen;
            }
            __threadfence();
            if (v & kClosed) {
                *(volatile int *)&ls->err = 1;
                v = 0;
            }
        }
        if (blockIdx.x == 0) {
            ls->ring[(k + 2) & 3] = 0;
            __threadfence();
        }
        done = v;
    }
    __syncthreads();
    k++;
    return done;
}

// Exclusive scan of n counts into start[0 .. n) by one block (the arithmetic of
// k_cell_scan).  Returns the total on every thread; a caller whose array holds
// n + 1 values stores it there itself.
__device__ __forceinline__ int scan_block(const int *cnt, int *start, int n) {
    __shared__ int wsum[32];
    __shared__ int carry_s;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int carry = 0;
    for (int base = 0; base < n; base += 4 * blockDim.x) {
        const int idx = base + 4 * threadIdx.x;
        int a[4];
#pragma unroll
        for (int k = 0; k < 4; k++) a[k] = idx + k < n ? cnt[idx + k] : 0;
        const int t = a[0] + a[1] + a[2] + a[3];
        int incl = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) wsum[wid] = incl;
        __syncthreads();
        if (wid == 0) {
            const int w = lane < nw ? wsum[lane] : 0;
            int wi = w;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, wi, o);
                if (lane >= o) wi += y;
            }
            wsum[lane] = wi - w;
            if (lane == 31) carry_s = wi;
        }
        __syncthreads();
        int ex = carry + wsum[wid] + incl - t;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (idx + k < n) start[idx + k] = ex;
            ex += a[k];
        }
        carry += carry_s;
        __syncthreads();
    }
    return carry;
}

// a block's slots and the tiles it walks them in: every thread runs the same
// number of tiles (G lanes per slot), `i < last` says whether its slot is real
struct Range {
    int first, last;
};

// neighbour row of particle i by the all-pairs methods, one thread
__device__ __forceinline__ int nlist_all_row(const DevSys *ds, int i) {
    const DevView &v = ds->v;
    const uint4 qi = v.q[i];
    int cnt = 0;
    for (int j = 0; j < ds->p.n; j++) {
        if (j == i || !within_cutoff(ds, v.pos, i, j, qi, v.q[j])) continue;
        if (cnt < ds->p.cap) v.nbr[(size_t)cnt * ds->p.n + i] = j;
        cnt++;
    }
    return cnt;
}

// The rebuild of the cell list (kind 2) and the neighbour list inside the
// loop: the kernels k_cell_index .. k_nlist_cell as phases between barriers.
// Returns false if the loop has to leave (a row longer than the capacity, or a
// barrier that ran out).
template <bool M>
__device__ bool loop_rebuild(DevSys *ds, LoopSync *ls, unsigned &bk, int polls, int kind, Range r) {
    const DevParams &p = ds->p;
    DevView &v = ds->v;
    DevState &s = ds->s;
    const int t = threadIdx.x, nt = blockDim.x;
    if (kind == 2) {
        for (int i = r.first + t; i < r.last; i += nt) {
            const double2 x = v.pos[i];
            const int c = cell_coord(x.x, p.cell_size, p.ncd) + cell_coord(x.y, p.cell_size, p.ncd) * p.ncd;
            ds->w.cell_raw[i] = c;
            atomicAdd(&ds->w.cell_cnt[c], 1);
        }
        if (!grid_bar(ls, bk, polls, 0)) return false;
        if (blockIdx.x == 0) {
            const int all = scan_block(ds->w.cell_cnt, ds->w.cell_start, p.ncells);
            if (t == 0) ds->w.cell_start[p.ncells] = all;
        }
        if (!grid_bar(ls, bk, polls, 0)) return false;
        for (int i = r.first + t; i < r.last; i += nt) {
            const int c = ds->w.cell_raw[i];
            ds->w.perm[ds->w.cell_start[c] + atomicAdd(&ds->w.cell_cur[c], 1)] = i;
        }
        if (!grid_bar(ls, bk, polls, 0)) return false;
        for (int c = blockIdx.x * nt + t; c < p.ncells; c += gridDim.x * nt) cell_sort_one(ds, c);
        if (!grid_bar(ls, bk, polls, 0)) return false;
        for (int i = r.first + t; i < r.last; i += nt) {
            const int o = ds->w.perm[i];
            const double2 x = v.pos[o];
            const double rad = v.rad[o];
            v.pos_t[i] = x;
            v.vel_t[i] = v.vel[o];
            v.frc_t[i] = v.frc[o];
            v.rad_t[i] = rad;
            v.mass_t[i] = v.mass[o];
            v.sidx_t[i] = v.sidx[o];
            v.q[i] = quant_of(p, x, rad);  // nothing reads q in this phase
            ds->w.cell_of[i] = ds->w.cell_raw[o];
            ds->w.pos_c[i] = x;
        }
        if (!grid_bar(ls, bk, polls, 0)) return false;
        if (t == 0) {
            swap_ptr(v.pos, v.pos_t);
            swap_ptr(v.vel, v.vel_t);
            swap_ptr(v.frc, v.frc_t);
            swap_ptr(v.rad, v.rad_t);
            swap_ptr(v.mass, v.mass_t);
            swap_ptr(v.sidx, v.sidx_t);
            swap_ptr(v.m1, v.m1_t);
            swap_ptr(v.m2, v.m2_t);
            s.n_cell_rebuilds++;
        }
        __syncthreads();
    } else if (M) {
        for (int i = r.first + t; i < r.last; i += nt) v.q[i] = quant_of(p, v.pos[i], v.rad[i]);
        if (!grid_bar(ls, bk, polls, 0)) return false;
    }
    int mx = 0;
    if (p.method == 0) {
        for (int b = r.first; b < r.last; b += nt / 8) {
            const int i = b + t / 8;
            const bool valid = i < r.last;
            const int cnt = nlist_row<8>(ds, i, valid);
            if (valid) mx = max(mx, cnt);
            if (valid && (t & 7) == 0) {
                const double2 x = v.pos[i];
                ds->w.count[i] = cnt;
                ds->w.pos_n[i] = x;
                if (M) v.pk[i] = mixed_pack(p, x, v.rad[i]);
            }
        }
    } else {
        for (int i = r.first + t; i < r.last; i += nt) {
            const int cnt = nlist_all_row(ds, i);
            mx = max(mx, cnt);
            const double2 x = v.pos[i];
            ds->w.count[i] = cnt;
            ds->w.pos_n[i] = x;
            if (M) v.pk[i] = mixed_pack(p, x, v.rad[i]);
        }
    }
    mx = (int)__reduce_max_sync(0xffffffffu, (unsigned)mx);
    __shared__ int bmx;
    if (t == 0) bmx = 0;
    __syncthreads();
    if ((t & 31) == 0) atomicMax(&bmx, mx);
    __syncthreads();
    if (t == 0) atomicMax(&ls->max_count, bmx);
    const unsigned long long w = grid_bar(ls, bk, polls, bmx > p.cap ? kFull : 0);
    if (!w) return false;
    if (t == 0) {
        s.n_rebuilds++;
        s.max_count = *(volatile int *)&ls->max_count;
        if (raised(w, kFull)) s.flags |= kOverflow;
    }
    __syncthreads();
    if (raised(w, kFull)) return false;
    // cleared for the next build, which starts only after another barrier
    if (blockIdx.x == 0 && t == 0) atomicExch(&ls->max_count, 0);
    return true;
}

// 3 d2 > thr for d2 >= 0, decided on the high words (lim: that of thr / 3) but
// for d2 next to the limit
__device__ __forceinline__ bool beyond(double d2, int lim, double thr) {
    const int h = __double2hiint(d2);
    if (h < lim - 1) return false;
    if (h > lim + 1 && h < 0x7ff00000) return true;
    return 3.0 * d2 > thr;
}

// per-particle displacements since the list builds as barrier flags
__device__ __forceinline__ unsigned long long move_flags(const DevParams &p, int lim_n, int lim_c, double nd2,
                                                         double cd2) {
    unsigned long long f = 0;
    if (p.method == 0 && beyond(cd2, lim_c, p.cthr2)) f |= kNeedCell;
    if (p.method != 2 && beyond(nd2, lim_n, p.nthr2)) f |= kNeedList;
    return f;
}

// the same without kept limits
__device__ __forceinline__ unsigned long long move_flags(const DevParams &p, double nd2, double cd2) {
    unsigned long long f = 0;
    if (p.method == 0 && 3.0 * cd2 > p.cthr2) f |= kNeedCell;
    if (p.method != 2 && 3.0 * nd2 > p.nthr2) f |= kNeedList;
    return f;
}

// thread 0's flags of the whole block
__device__ __forceinline__ unsigned long long block_flags(unsigned long long f) {
    const int cell = __syncthreads_or((f & kNeedCell) != 0), list = __syncthreads_or((f & kNeedList) != 0);
    return (cell ? kNeedCell : 0) | (list ? kNeedList : 0);
}

__device__ __forceinline__ int rebuild_kind(unsigned long long w) {
    return raised(w, kNeedCell) ? 2 : (raised(w, kNeedList) ? 1 : 0);
}

// The totals of a FIRE iteration over the grid: v[0], v[1] summed, the other
// K - 2 maxima; thread 0 gets them.  `nwr`: warps that hold values.  Two sums
// share each FP64 instruction (lanes 0 - 15 and 16 - 31): an instruction holds
// the pipe for a whole warp whatever its lanes.  The block partials are added
// in a fixed order, so every block gets the same bits.  false: the barrier ran
// out.  Every thread of the block calls it.
template <int K>
__device__ __forceinline__ void warp_totals(double &sum, double (&mx)[K - 2]) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o, 16);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < K - 2; k++) mx[k] = max_pos(mx[k], __shfl_down_sync(0xffffffffu, mx[k], o));
}
template <int K>
__device__ __forceinline__ bool grid_totals(double (&v)[K], int nwr, double *part, LoopSync *ls, unsigned &bk, int polls,
                                            double *sm) {
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5, nb = gridDim.x;
    double mx[K - 2], sum;
    if (wid < nwr) {
        const bool low = lane < 16;
        sum = low ? v[0] : v[1];
        sum += __shfl_xor_sync(0xffffffffu, low ? v[1] : v[0], 16);
#pragma unroll
        for (int k = 0; k < K - 2; k++) mx[k] = max_pos(0.0, v[2 + k]);
        warp_totals<K>(sum, mx);
        if ((lane & 15) == 0) sm[wid * K + (low ? 0 : 1)] = sum;
        if (lane == 0)
#pragma unroll
            for (int k = 0; k < K - 2; k++) sm[wid * K + 2 + k] = mx[k];
    }
    __syncthreads();
    if (t < K) {
        double a = sm[t];
        for (int w = 1; w < nwr; w++) a = t < 2 ? a + sm[w * K + t] : max_pos(a, sm[w * K + t]);
        part[t * nb + blockIdx.x] = a;
    }
    if (!grid_bar(ls, bk, polls, 0)) return false;
    if (wid == 0) {
        // all loads in flight at once (one trip to L2), then added in order
        const double *mine = part + (lane < 16 ? 0 : nb);
        constexpr int U = (kLoopBlocksMax + 15) / 16;
        double a[U], c[K - 2][U / 2];
#pragma unroll
        for (int q = 0; q < U; q++) a[q] = (lane & 15) + 16 * q < nb ? mine[(lane & 15) + 16 * q] : 0.0;
#pragma unroll
        for (int k = 0; k < K - 2; k++)
#pragma unroll
            for (int q = 0; q < U / 2; q++) c[k][q] = lane + 32 * q < nb ? part[(2 + k) * nb + lane + 32 * q] : 0.0;
        sum = a[0];
#pragma unroll
        for (int q = 1; q < U; q++)
            if (16 * q < nb) sum += a[q];
#pragma unroll
        for (int k = 0; k < K - 2; k++) {
            mx[k] = 0.0;
#pragma unroll
            for (int q = 0; q < U / 2; q++) mx[k] = max_pos(mx[k], c[k][q]);
        }
        warp_totals<K>(sum, mx);
        v[1] = __shfl_sync(0xffffffffu, sum, 16);
        v[0] = sum;
#pragma unroll
        for (int k = 0; k < K - 2; k++) v[2 + k] = mx[k];
    }
    return true;
}

// End of a resident loop: the displacement maxima of the last move (zero where
// a build followed), after every block has handed in its own.  True on thread 0
// of block 0, which then writes its copy of the system back.
__device__ __forceinline__ bool loop_exit(DevSys *L, LoopSync *ls, unsigned &bk, int polls, Range r, double *red) {
    const int t = threadIdx.x, nb = gridDim.x;
    double m[2] = {0.0, 0.0};
    for (int i = r.first + t; i < r.last; i += blockDim.x) {
        const double2 x = L->v.pos[i], a = L->w.pos_n[i], c = L->w.pos_c[i];
        const double dxn = x.x - a.x, dyn = x.y - a.y, dxc = x.x - c.x, dyc = x.y - c.y;
        m[0] = fmax(m[0], dxn * dxn + dyn * dyn);
        m[1] = fmax(m[1], dxc * dxc + dyc * dyc);
    }
    const int ops[2] = {1, 1};
    block_reduce<2>(m, ops, red);
    double *part = L->w.partials + 5 * nb;  // apart from the sums that a slower block may still read
    if (t == 0) {
        part[blockIdx.x] = m[0];
        part[nb + blockIdx.x] = m[1];
    }
    const bool all = grid_bar(ls, bk, polls, 0) != 0;
    if (blockIdx.x != 0) return false;
    m[0] = 0.0;
    m[1] = 0.0;
    if (all)
        for (int b = t; b < nb; b += blockDim.x) {
            m[0] = fmax(m[0], part[b]);
            m[1] = fmax(m[1], part[nb + b]);
        }
    block_reduce<2>(m, ops, red);
    if (t == 0) {
        L->s.max_nd2 = m[0];
        L->s.max_cd2 = m[1];
        L->s.rebuild = 0;
        // a barrier fails for every block alike: this thread has set err then
        if (!all || *(volatile int *)&ls->err) L->s.flags |= kError;
    }
    return t == 0;
}

// ---- one tile per block: a block's particles stay in its registers -----------
constexpr int kTileP = 128;      // particles per block at most
constexpr int kTileSlots = 32;   // list capacity at most: the rows are cached
constexpr int kTileStride = kTileSlots + 1;

// dynamic shared memory of a block of `np` particles
struct TileMem {
    double *rl;           // [np][kTileStride] radius of each listed neighbour
    double *res;          // [3][qw] terms of the queued pairs
    double *sum;          // [3][np] pair sums
    int *idx;             // [np][kTileStride] listed neighbours
    int *off;             // [np + 1] first queue entry of each particle
    unsigned short *ent;  // [qw] particle << 5 | slot
    int qw;
};
__host__ __device__ inline int tile_queue(int np) { return np * 10 < 256 ? 256 : np * 10; }
__host__ __device__ inline size_t tile_bytes(int np) {
    const int qw = tile_queue(np);
    return (size_t)8 * (np * kTileStride + 3 * qw + 3 * np) + (size_t)4 * (np * kTileStride + np + 1) + 2 * (size_t)qw;
}
__device__ __forceinline__ TileMem tile_mem(unsigned char *base, int np) {
    TileMem m;
    m.qw = tile_queue(np);
    m.rl = reinterpret_cast<double *>(base);
    m.res = m.rl + np * kTileStride;
    m.sum = m.res + 3 * m.qw;
    m.idx = reinterpret_cast<int *>(m.sum + 3 * np);
    m.off = m.idx + np * kTileStride;
    m.ent = reinterpret_cast<unsigned short *>(m.off + np + 1);
    return m;
}

// The loop for systems whose blocks hold their particles in one tile: thread t
// of a block owns particle first + t and keeps its position, velocity, force,
// mass, radius and last-build positions in registers across iterations; the
// neighbour rows (with the neighbours' radii) sit in shared memory.  An
// iteration then reads from L2 only what other blocks moved: one fixed-point
// position a listed neighbour and, prefetched beside it, the FP64 position of
// those that touch.  The contacts of the whole block form one queue (pair_sums
// with a block for a warp), so the FP64 instructions run on full warps, and the
// per-particle update runs on np / 32 warps whatever the lanes per neighbour
// row.  A particle's three sums run on three threads, which for few particles
// shares each addition among them; limits, kick factors and zeros are compared
// as integers and a kick's or a mix's quotient is a quick one: with few warps a
// block, every FP64 instruction of the update is ~64 clocks of the step (NVE of
// 1024 disks 8.2 -> 7.3 us, FIRE of 16384 20.6 -> 19.6).  Same arithmetic and
// order of sums as k_loop.
template <int KIND, int G, bool M>
__global__ void __launch_bounds__(kLoopMaxTPB, 1) k_tile(DevSys *ds, LoopSync *ls, double dt, int chunk,
                                                        long long iters, int polls) {
    extern __shared__ __align__(16) unsigned char loop_smem[];
    __shared__ DevSys L;
    __shared__ double red[32 * 3];
    __shared__ int wtot[kLoopMaxTPB / 32];
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5, nw = blockDim.x >> 5;
    const int g = t / G, sub = t & (G - 1), lead = lane - sub;
    if (t == 0) L = *ds;
    __syncthreads();
    // every block of a cluster runs before its shared memory is written to
    if (cooperative_groups::this_cluster().num_blocks() > 1) cooperative_groups::this_cluster().sync();
    const DevParams &p = L.p;
    DevView &v = L.v;
    DevState &s = L.s;
    const DevScratch &w = L.w;
    if (s.flags) return;  // the same for every block: nothing writes the state before a barrier
    const TileMem m = tile_mem(loop_smem, chunk);
    const int n = p.n;
    const Range r = {min((int)blockIdx.x * chunk, n), min(((int)blockIdx.x + 1) * chunk, n)};
    const int np = r.last - r.first, own = r.first + t;
    const bool mine = t < np;
    const double dt_half = 0.5 * dt;
    const int lim_n = __double2hiint(p.nthr2 / 3.0), lim_c = __double2hiint(p.cthr2 / 3.0);
    // the sums' threads: component t / np of particle t % np
    const int sum_k = np > 0 ? t / np : 3, sum_g = np > 0 ? t % np : 0;
    unsigned bk = 0;
    bool ok = true, stored = false;
    long long it = 0;

    double2 x = {0.0, 0.0}, u = {0.0, 0.0}, f = {0.0, 0.0}, xn = {0.0, 0.0}, xc = {0.0, 0.0};
    float rf = 0.f;
    double mass = 1.0, rad = 0.0, pe = 0.0, dtm = 0.0, dtm_of = 0.0;
    bool dtm_known = false;
    int gcnt = 0;  // row length of the group's particle
    auto load_own = [&]() {
        if (mine) {
            x = v.pos[own]; u = v.vel[own]; f = v.frc[own];
            xn = w.pos_n[own]; xc = w.pos_c[own];
            mass = v.mass[own]; rad = v.rad[own];
            rf = (float)rad;
        }
        dtm_known = false;
        gcnt = g < np ? min(w.count[r.first + g], p.cap) : 0;
        for (int k = sub; k < gcnt; k += G) {
            const int j = v.nbr[(size_t)k * n + r.first + g];
            m.idx[g * kTileStride + k] = j;
            m.rl[g * kTileStride + k] = v.rad[j];
        }
        __syncthreads();
    };
    auto store_own = [&]() {
        if (mine) {
            v.vel[own] = u;
            v.frc[own] = f;
        }
    };
    // (h / mass), kept while h is the same
    auto kick_factor = [&](double h) {
        if (!dtm_known || __double_as_longlong(h) != __double_as_longlong(dtm_of)) {
            dtm = over_mass(h, mass);
            dtm_of = h;
            dtm_known = true;
        }
        return dtm;
    };
    // the moved position into the given buffers; this particle's rebuild flags
    auto publish = [&](double2 *pos, float4 *pk, uint4 *q) -> unsigned long long {
        pos[own] = x;
        if (M) pk[own] = mixed_pack(p, x, rad);
        if (!M || (KIND == 0 && s.fp64_now)) q[own] = quant_of(p, x, rf);
        double d2[2];
        moved2(x, xn, xc, d2);
        return move_flags(p, lim_n, lim_c, d2[0], d2[1]);
    };
    auto nve_first = [&]() -> unsigned long long {
        if (!mine) return 0;
        const double h = kick_factor(dt_half);
        u.x = u.x + f.x * h;
        u.y = u.y + f.y * h;
        x.x = x.x + u.x * dt;
        x.y = x.y + u.y * dt;
        return publish(v.pos_t, v.pk_t, v.q_t);
    };
    // the barrier after a move, the buffer swap (NVE) and a rebuild if any
    // particle asks for one; false: leave
    auto after_move = [&](unsigned long long fl) {
        const unsigned long long bw = grid_bar(ls, bk, polls, block_flags(fl));
        if (!bw) return false;
        if (KIND == 1) {
            if (t == 0) {
                swap_ptr(v.pos, v.pos_t);
                if (M) swap_ptr(v.pk, v.pk_t);
                else swap_ptr(v.q, v.q_t);
            }
            __syncthreads();
        }
        const int kind = rebuild_kind(bw);
        if (!kind) return true;
        store_own();
        stored = true;
        if (!loop_rebuild<M>(&L, ls, bk, polls, kind, r)) return false;
        load_own();
        stored = false;
        return true;
    };

    load_own();
    if (KIND == 1) ok = after_move(nve_first());
    // the energy that the first iteration's is compared with, summed in the same order
    if (KIND == 0 && s.pe_diff_target > 0) {
        double tot[3] = {mine ? w.pe[own] : 0.0, 0.0, 0.0};
        ok = grid_totals<3>(tot, (np + 31) / 32, w.partials, ls, bk, polls, red);
        if (ok && t == 0) s.last_avg_pe = tot[0] / s.dof;
        __syncthreads();
    }
    while (ok) {
        if (KIND == 0) {
            // ---- move (k_fire_move)
            unsigned long long fl = 0;
            if (mine) {
                const double fdt = s.f_dt, alpha = s.f_alpha;
                if (s.fire_uphill) {
                    const double back = -fdt / 2.0;
                    x.x = x.x + u.x * back;
                    x.y = x.y + u.y * back;
                    u = make_double2(0.0, 0.0);
                }
                const double h = kick_factor(fdt / 2.0);
                u.x = u.x + f.x * h;
                u.y = u.y + f.y * h;
                u = fire_mix(u, f, alpha);
                x.x = x.x + u.x * fdt;
                x.y = x.y + u.y * fdt;
                fl = publish(v.pos, v.pk, v.q);
            }
            ok = after_move(fl);
            if (!ok) break;
        }
        // ---- pair sums
        double acc[3] = {0.0, 0.0, 0.0};
        const bool fp32 = M && !(KIND == 0 && s.fp64_now);
        const int most = (int)__reduce_max_sync(0xffffffffu, (unsigned)gcnt);
        if (fp32) {
            constexpr int R = 8 / G;
            const float e_c = (float)p.e_c, n_c = (float)p.n_c;
            const float4 a = v.pk[g < np ? r.first + g : r.first];
            double ax = 0.0, ay = 0.0, en = 0.0;
            for (int k0 = 0; k0 < most; k0 += 8) {  // mixed_sums<G>
                float fx[R], fy[R], e[R];
#pragma unroll
                for (int q = 0; q < R; q++) {
                    const int k = k0 + q * G + sub;
                    fx[q] = 0.f; fy[q] = 0.f; e[q] = 0.f;
                    if (k < gcnt) e[q] = mixed_pair(p, a, v.pk[m.idx[g * kTileStride + k]], e_c, n_c, fx[q], fy[q]);
                }
                float sx = 0.f, sy = 0.f, se = 0.f;
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    sx += __shfl_sync(0xffffffffu, fx[c / G], lead + c % G);
                    sy += __shfl_sync(0xffffffffu, fy[c / G], lead + c % G);
                    se += __shfl_sync(0xffffffffu, e[c / G], lead + c % G);
                }
                ax += (double)sx;
                ay += (double)sy;
                en += (double)se;
            }
            if (sub == 0 && g < np) {
                m.sum[g] = ax;
                m.sum[chunk + g] = ay;
                m.sum[2 * chunk + g] = en;
            }
        } else {
            double sum = 0.0;
            const uint4 qi = v.q[g < np ? r.first + g : r.first];
            unsigned bits = 0;
            for (int k0 = 0; k0 < most; k0 += 4 * G) {
                int j[4];
                uint4 qj[4];
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const int k = k0 + c * G + sub;
                    j[c] = k < gcnt ? m.idx[g * kTileStride + k] : r.first;
                }
#pragma unroll
                for (int c = 0; c < 4; c++) qj[c] = v.q[j[c]];
#pragma unroll
                for (int c = 0; c < 4; c++)
                    if (k0 + c * G + sub < gcnt) asm volatile("prefetch.global.L1 [%0];" ::"l"(v.pos + j[c]));
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const int k = k0 + c * G + sub;
                    const bool hit = k < gcnt && quant_touch(p.q_s[0], p.q_s[1], p.q_tol, qi, qj[c]);
                    const unsigned b = __ballot_sync(0xffffffffu, hit);
                    if (k0 + c * G < kTileSlots) bits |= ((b >> lead) & ((1u << G) - 1u)) << (k0 + c * G);
                }
            }
            // queue offsets over the block: warp scans, then the warps' totals
            const int c = __popc(bits);
            int incl = sub == 0 ? c : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            if (lane == 31) wtot[wid] = incl;
            __syncthreads();
            const int mine_w = lane < nw ? wtot[lane] : 0;
            const int before = __reduce_add_sync(0xffffffffu, lane < wid ? mine_w : 0);
            const int total = __reduce_add_sync(0xffffffffu, mine_w);
            const int end = __shfl_sync(0xffffffffu, incl, lead) + before, off = end - c;
            if (sub == 0 && g < np) m.off[g] = off;
            if (t == 0) m.off[np] = total;
            const PairArgs fa = pair_args(&L);
            for (int w0 = 0; w0 < total; w0 += m.qw) {
                const int w1 = min(total, w0 + m.qw);
                for (int k = sub; k < gcnt; k += G) {
                    const int at = off + __popc(bits & ((1u << k) - 1u));
                    if ((bits >> k & 1u) && at >= w0 && at < w1) m.ent[at - w0] = (unsigned short)(g << 5 | k);
                }
                __syncthreads();
                for (int e = t; e < w1 - w0; e += blockDim.x) {
                    const int ent = m.ent[e], o = ent >> 5, k = ent & 31, i = r.first + o;
                    const int j = m.idx[o * kTileStride + k];
                    double dx, dy, fx, fy;
                    const double ee = disk_pair_sum(fa, fa.pos[i], fa.rad[i], fa.pos[j],
                                                    m.rl[o * kTileStride + k], dx, dy, fx, fy);
                    m.res[e] = fx;
                    m.res[m.qw + e] = fy;
                    m.res[2 * m.qw + e] = ee;
                }
                __syncthreads();
                if (sum_k < 3) {
                    const int b0 = max(m.off[sum_g], w0) - w0, b1 = min(m.off[sum_g + 1], w1) - w0;
                    const double *res = m.res + sum_k * m.qw;
                    for (int b = b0; b < b1; b++) sum += res[b];
                }
                if (w1 < total) __syncthreads();
            }
            if (sum_k < 3) m.sum[sum_k * chunk + sum_g] = sum;
        }
        __syncthreads();
        if (mine)
#pragma unroll
            for (int k = 0; k < 3; k++) acc[k] = m.sum[k * chunk + t];
        // ---- kick (k_fire_force, k_nve_second)
        const bool last = KIND == 1 && (it + 1 >= iters || s.nve_steps_done + 1 >= s.max_steps);
        it++;
        if (KIND == 1) {
            unsigned long long fl = 0;
            if (mine) {
                f = nve_force(&L, own, u, acc[0], acc[1], acc[2], pe);
                const double h = kick_factor(dt_half);
                u.x = u.x + f.x * h;
                u.y = u.y + f.y * h;
                if (!last) fl = nve_first();
            }
            __syncthreads();  // every thread has read the state
            if (t == 0 && ++s.nve_steps_done >= s.max_steps) s.flags |= kDone;
            __syncthreads();
            if (last) break;
            ok = after_move(fl);
        } else {
            double tot[3] = {0.0, 0.0, 0.0};
            if (mine) {
                f = make_double2(acc[0], acc[1]);
                pe = acc[2];
                const double h = kick_factor(s.f_dt / 2.0);
                u.x = u.x + f.x * h;
                u.y = u.y + f.y * h;
                tot[0] = pe;
                tot[1] = f.x * u.x + f.y * u.y;
                tot[2] = f.x * f.x + f.y * f.y;
            }
            ok = grid_totals<3>(tot, (np + 31) / 32, w.partials, ls, bk, polls, red);
            if (!ok) break;
            if (t == 0) fire_epilogue<M>(s, tot);
            __syncthreads();
            if (s.flags || it >= iters) break;
        }
    }
    if (!stored) {
        store_own();
        if (mine) w.pe[own] = pe;
    }
    if (loop_exit(&L, ls, bk, polls, r, red)) {
        ds->v = v;
        ds->s = s;
    }
}

// Pair sums of slot i in the loop: FP64 with the queue, or FP32 (M) with G
// lanes sharing a run of 8 neighbours (disk_force_sum_mixed's sums)
template <int G, bool M>
__device__ __forceinline__ void loop_sums(const DevSys *ds, const PairArgs &f, int i, bool valid, bool fp32,
                                          ForceWarp *w, double &ax, double &ay, double &en) {
    const int cnt = valid ? min(ds->w.count[i], ds->p.cap) : 0;
    if (M && fp32) {
        mixed_sums<G>(ds->p, ds->v.pk, ds->v.nbr, valid ? i : 0, cnt, ax, ay, en);
    } else {
        double acc[3] = {0.0, 0.0, 0.0};
        pair_sums<G, 3>(f, valid ? i : 0, cnt, w[threadIdx.x >> 5], acc);
        ax = acc[0]; ay = acc[1]; en = acc[2];
    }
}

// kind 0: FIRE iterations (k_fire_move, rebuild, k_fire_force mode 0); kind 1:
// NVE steps (k_nve_first, rebuild, k_nve_second), until a flag is raised or
// `iters` iterations are done.
template <int KIND, int G, bool M>
__global__ void __launch_bounds__(kLoopMaxTPB, 1) k_loop(DevSys *ds, LoopSync *ls, double dt, int chunk,
                                                      long long iters, int polls) {
    extern __shared__ __align__(16) unsigned char loop_smem[];
    ForceWarp *fw = reinterpret_cast<ForceWarp *>(loop_smem);
    // the block's copy of the system: pointers, parameters and control state
    // without a trip to L2 after every barrier
    __shared__ DevSys L;
    __shared__ double red[32 * 3];
    const int t = threadIdx.x, nt = blockDim.x, tile = nt / G, sub = t & (G - 1);
    if (t == 0) L = *ds;
    __syncthreads();
    const DevParams &p = L.p;
    DevView &v = L.v;
    DevState &s = L.s;
    const DevScratch &w = L.w;
    if (s.flags) return;  // the same for every block: nothing writes the state before a barrier
    const int n = p.n;
    const Range r = {min((int)blockIdx.x * chunk, n), min(((int)blockIdx.x + 1) * chunk, n)};
    unsigned bk = 0;
    bool ok = true;
    long long it = 0;
    const double dt_half = 0.5 * dt;
    const int lim_n = __double2hiint(p.nthr2 / 3.0), lim_c = __double2hiint(p.cthr2 / 3.0);

    // NVE: the first half of a step, from the current into the other buffers
    auto drift_to_other = [&](int i, double2 u, double2 f, double dtm, unsigned long long &fl) {
        double2 x = v.pos[i];
        u.x = u.x + f.x * dtm;
        u.y = u.y + f.y * dtm;
        v.vel[i] = u;
        x.x = x.x + u.x * dt;
        x.y = x.y + u.y * dt;
        v.pos_t[i] = x;
        const double rad = v.rad[i];
        if (M) v.pk_t[i] = mixed_pack(p, x, rad);
        else v.q_t[i] = quant_of(p, x, rad);
        double d2[2];
        moved2(x, w.pos_n[i], w.pos_c[i], d2);
        fl |= move_flags(p, lim_n, lim_c, d2[0], d2[1]);
    };
    auto swap_moved = [&]() {
        if (t == 0) {
            swap_ptr(v.pos, v.pos_t);
            if (M) swap_ptr(v.pk, v.pk_t);
            else swap_ptr(v.q, v.q_t);
        }
        __syncthreads();
    };

    if (KIND == 1) {
        unsigned long long fl = 0;
        for (int i = r.first + t; i < r.last; i += nt)
            drift_to_other(i, v.vel[i], v.frc[i], over_mass(dt_half, v.mass[i]), fl);
        const unsigned long long bw = grid_bar(ls, bk, polls, block_flags(fl));
        ok = bw != 0;
        if (ok) {
            swap_moved();
            const int kind = rebuild_kind(bw);
            if (kind) ok = loop_rebuild<M>(&L, ls, bk, polls, kind, r);
        }
    }
    if (KIND == 0 && s.pe_diff_target > 0) {  // as in k_tile
        double tot[3] = {0.0, 0.0, 0.0};
        for (int i = r.first + t / G; i < r.last; i += tile)
            if (sub == 0) tot[0] += w.pe[i];
        ok = grid_totals<3>(tot, nt / 32, w.partials, ls, bk, polls, red);
        if (ok && t == 0) s.last_avg_pe = tot[0] / s.dof;
        __syncthreads();
    }
    while (ok) {
        if (KIND == 0) {
            // ---- move (k_fire_move)
            const double fdt = s.f_dt, alpha = s.f_alpha;
            const int up = s.fire_uphill;
            unsigned long long fl = 0;
            for (int i = r.first + t; i < r.last; i += nt) {
                double2 u = v.vel[i], x = v.pos[i];
                const double2 f = v.frc[i];
                if (up) {
                    const double back = -fdt / 2.0;
                    x.x = x.x + u.x * back;
                    x.y = x.y + u.y * back;
                    u = make_double2(0.0, 0.0);
                }
                const double dtm = over_mass(fdt / 2.0, v.mass[i]);
                u.x = u.x + f.x * dtm;
                u.y = u.y + f.y * dtm;
                u = fire_mix(u, f, alpha);
                v.vel[i] = u;
                x.x = x.x + u.x * fdt;
                x.y = x.y + u.y * fdt;
                v.pos[i] = x;
                const double rad = v.rad[i];
                if (M) v.pk[i] = mixed_pack(p, x, rad);
                if (!M || s.fp64_now) v.q[i] = quant_of(p, x, rad);
                double d2[2];
                moved2(x, w.pos_n[i], w.pos_c[i], d2);
                fl |= move_flags(p, lim_n, lim_c, d2[0], d2[1]);
            }
            const unsigned long long bw = grid_bar(ls, bk, polls, block_flags(fl));
            ok = bw != 0;
            if (!ok) break;
            const int kind = rebuild_kind(bw);
            if (kind) ok = loop_rebuild<M>(&L, ls, bk, polls, kind, r);
            if (!ok) break;
        }
        // ---- forces and kick (k_fire_force, k_nve_second); NVE: the next
        // step's first half too, unless this is the last step of the launch
        const PairArgs f = pair_args(&L);
        const bool fp32 = M && !(KIND == 0 && s.fp64_now);
        const bool last = KIND == 1 && (it + 1 >= iters || s.nve_steps_done + 1 >= s.max_steps);
        unsigned long long fl = 0;
        double tot[3] = {0.0, 0.0, 0.0};
        for (int b = r.first; b < r.last; b += tile) {
            const int i = b + t / G;
            const bool valid = i < r.last;
            double ax, ay, en;
            loop_sums<G, M>(&L, f, i, valid, fp32, fw, ax, ay, en);
            if (!valid || sub != 0) continue;
            double2 u = v.vel[i];
            if (KIND == 1) {
                double pe;
                const double2 frc = nve_force(&L, i, u, ax, ay, en, pe);
                v.frc[i] = frc;
                w.pe[i] = pe;
                const double dtm = over_mass(dt_half, v.mass[i]);
                u.x = u.x + frc.x * dtm;
                u.y = u.y + frc.y * dtm;
                if (last) v.vel[i] = u;
                else drift_to_other(i, u, frc, dtm, fl);
            } else {
                const double2 frc = make_double2(ax, ay);
                v.frc[i] = frc;
                w.pe[i] = en;
                const double dtm = over_mass(s.f_dt / 2.0, v.mass[i]);
                u.x = u.x + frc.x * dtm;
                u.y = u.y + frc.y * dtm;
                v.vel[i] = u;
                tot[0] += en;
                tot[1] += frc.x * u.x + frc.y * u.y;
                tot[2] = fmax(tot[2], frc.x * frc.x + frc.y * frc.y);
            }
        }
        it++;
        if (KIND == 1) {
            __syncthreads();  // every thread has read the state
            if (t == 0 && ++s.nve_steps_done >= s.max_steps) s.flags |= kDone;
            __syncthreads();
            if (last) break;
            const unsigned long long bw = grid_bar(ls, bk, polls, block_flags(fl));
            ok = bw != 0;
            if (!ok) break;
            swap_moved();
            const int kind = rebuild_kind(bw);
            if (kind) ok = loop_rebuild<M>(&L, ls, bk, polls, kind, r);
        } else {
            ok = grid_totals<3>(tot, nt / 32, w.partials, ls, bk, polls, red);
            if (!ok) break;
            if (t == 0) fire_epilogue<M>(s, tot);
            __syncthreads();
            if (s.flags || it >= iters) break;
        }
    }
    if (loop_exit(&L, ls, bk, polls, r, red)) {
        ds->v = v;
        ds->s = s;
    }
}

}  // namespace
}  // namespace dpg
