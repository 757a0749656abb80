// disk_kernels.cuh -- plain FP64 kernels for soft disks (the drop-in form).
//
// Compiled with --fmad=false: every multiply and add is rounded separately, in
// the reference's operation order, so per-particle results are bit-identical
// to the reference kernels (src/particles/base/kernels.cu,
// src/particles/disk/kernels.cu).  Explicit fma() calls appear only where the
// reference itself calls fma (Adam).
//
// Every kernel takes the device-resident DevSys and reads the current buffer
// pointers from it, so launch arguments never go stale inside a CUDA graph.
#pragma once
#include "dpg_device.cuh"

namespace dpg {
namespace {  // kernels have internal linkage: each translation unit owns its copy

constexpr int kMixed = 1;  // DevParams.precision of the mixed form (DPG_MIXED)

template <class T>
__device__ __forceinline__ void swap_ptr(T *&a, T *&b) {
    T *t = a;
    a = b;
    b = t;
}

__device__ __forceinline__ bool halted(const DevSys *ds) { return ds->s.flags != 0; }

// harmonic (power-law) contact of particle i with j, force on i:
// include/particles/base/kernels.cuh:154-183
__device__ __forceinline__ double disk_pair(double xi, double yi, double ri, double xj, double yj,
                                            double rj, double bx, double by, double e_c,
                                            double n_c, double &fx, double &fy) {
    double dx = pbc_dist(xi, xj, bx);
    double dy = pbc_dist(yi, yj, by);
    double rs = ri + rj;
    double d2 = dx * dx + dy * dy;
    if (d2 >= rs * rs) { fx = 0.0; fy = 0.0; return 0.0; }
    double d = sqrt(d2);
    double ov = 1.0 - (d / rs);
    double ovp, energy;
    if (n_c == 2.0) {  // pow(ov, 1) == ov, and x / 4 == x * 0.25 exactly
        ovp = ov;
        energy = e_c * ov * ovp * 0.25;
    } else {
        ovp = pow(ov, n_c - 1);
        energy = e_c * ov * ovp / (2.0 * n_c);
    }
    double fm = e_c * ovp / (rs * d);
    fx = fm * dx;
    fy = fm * dy;
    return energy;
}

// ---- FP64 pair sums of the particles of a warp ---------------------------------
// kernelCalcDiskForces (src/particles/disk/kernels.cu:11-57): per particle, the
// sum of its pair terms in neighbour-slot order.  Pairs that do not touch add
// +0.0, which leaves a sum that started at +0.0 unchanged, so only the
// contacts need FP64 work.  Bound: the FP64 pipe (2 lanes a clock on each SM;
// a contact is ~30 FP64 instructions), where an instruction costs the same with
// one active lane as with 32.  So a warp (32 / G particles, G lanes each) works in three steps: G lanes test
// a particle's slots by the fixed-point filter; the surviving pairs of all its
// particles are queued in shared memory, ordered by particle and slot, and
// evaluated 32 at a time, whoever they belong to; each particle then adds its
// own results in slot order, so the sums are those of the sequential loop, bit
// for bit, for every G.  A loop over slots instead runs as many FP64 rounds as
// the longest list of the warp has entries (~12 against ~4 queue rounds at 6.5
// neighbours and 3.3 contacts a particle).
// Measured at 2^20 disks of 3.3 contacts: k_nve_second 1219 -> 365 us; at 16384
// (2 lanes) k_fire_force 46 -> 32 us; k_stress of 131071 disks 262 -> 126 us.
constexpr int kSlotChunk = 16;   // slots filtered before the queue is worked off
constexpr int kPairWin = 160;    // queue entries evaluated before they are added up:
                                 // 32 particles with 5 contacts each
template <int K>
struct PairWarp {                // shared memory of one warp
    unsigned short ent[32 * kSlotChunk];  // owner lane << 5 | slot in the chunk
    double r[K][kPairWin];                // the terms of each entry
};
constexpr int kForceTPB = 256;   // threads per block of the force kernels
typedef PairWarp<3> ForceWarp;   // force x, force y, energy

// what the pair sums read (the caller may keep it in registers)
struct PairArgs {
    const double2 *pos;
    const double *rad;   // null: every radius is rv
    const int *nbr;
    const uint4 *q;
    int n;
    double bx, by, e_c, n_c;
    int l4x, l4y;
    float sx, sy, tol;
    double rv;
};

__device__ __forceinline__ PairArgs pair_args(const DevSys *ds) {
    return {ds->v.pos, ds->v.rad, ds->v.nbr, ds->v.q, ds->p.n, ds->p.box[0], ds->p.box[1], ds->p.e_c,
            ds->p.n_c, ds->p.q_l4[0], ds->p.q_l4[1], ds->p.q_s[0], ds->p.q_s[1], ds->p.q_tol, 0.0};
}

// The terms of a contact from its displacement for radius sum rs; inv: near
// 1 / rs where the caller keeps one (KEPT).  disk_pair's arithmetic and its bits, on 30 FP64
// instructions instead of 46 (displacement included) for harmonic contacts: an
// NVE step of 1048576 disks 362 -> 325 us, of 4096 bodies 60 -> 53 us.
template <bool KEPT>
__device__ __forceinline__ double contact_terms(double dx, double dy, double rs, double inv, double e_c,
                                                double n_c, double &fx, double &fy) {
    const double d2 = dx * dx + dy * dy;
    fx = 0.0;
    fy = 0.0;
    // constants compared as integers: FP64 compares take the FP64 pipe
    const bool square = __double2hiint(n_c) == 0x40000000 && __double2loint(n_c) == 0;
    const bool unit = __double2hiint(e_c) == 0x3ff00000 && __double2loint(e_c) == 0;
    if (square && middling(d2) && middling(rs) && middling(e_c)) {
        double y;
        const double d = root_near(d2, y);
        if (!KEPT) inv = rcp_near(rs);
        const double ov = 1.0 - div_near(d, rs, inv);
        // an overlap above 2^-40 needs no test
        if (__double2hiint(ov) < 0x3d700000 && d2 >= rs * rs) return 0.0;
        const double a = unit ? ov : e_c * ov;  // pow(ov, 1) == ov
        const double fm = div_near(a, rs * d, inv * y);
        fx = fm * dx;
        fy = fm * dy;
        return a * ov * 0.25;  // x / 4 == x * 0.25 exactly
    }
    if (d2 >= rs * rs) return 0.0;
    const double d = sqrt(d2);
    const double ov = 1.0 - (d / rs);
    double ovp, energy;
    if (square) {
        ovp = ov;
        energy = e_c * ov * ovp * 0.25;
    } else {
        ovp = pow(ov, n_c - 1);
        energy = e_c * ov * ovp / (2.0 * n_c);
    }
    const double fm = e_c * ovp / (rs * d);
    fx = fm * dx;
    fy = fm * dy;
    return energy;
}

// disk_pair for the sums (see pbc_dist_sum)
__device__ __forceinline__ double disk_pair_sum(const PairArgs &f, double2 pi, double ri, double2 pj,
                                                double rj, double &dx, double &dy, double &fx,
                                                double &fy) {
    dx = pbc_dist_sum(pi.x, pj.x, f.bx, f.l4x);
    dy = pbc_dist_sum(pi.y, pj.y, f.by, f.l4y);
    return contact_terms<false>(dx, dy, ri + rj, 0.0, f.e_c, f.n_c, fx, fy);
}

// Slots s0 .. s0 + kSlotChunk - 1 of the particle's list that may touch it, as
// bits (every lane of the group gets them).  cnt: its list length.  All lanes
// of the warp call it.
template <int G>
__device__ __forceinline__ unsigned touch_bits(const PairArgs &f, int i, uint4 qi, int s0, int cnt) {
    const int sub = threadIdx.x & (G - 1), lead = (threadIdx.x & 31) - sub;
    unsigned bits = 0;
    if (G == 1) {
#pragma unroll
        for (int u0 = 0; u0 < kSlotChunk; u0 += 4) {
            if (s0 + u0 >= cnt) break;
            int j[4];
            uint4 qj[4];
#pragma unroll
            for (int u = 0; u < 4; u++) j[u] = s0 + u0 + u < cnt ? f.nbr[(size_t)(s0 + u0 + u) * f.n + i] : i;
#pragma unroll
            for (int u = 0; u < 4; u++) qj[u] = f.q[j[u]];
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (s0 + u0 + u < cnt && quant_touch(f.sx, f.sy, f.tol, qi, qj[u])) bits |= 1u << (u0 + u);
        }
    } else {
        constexpr int R = kSlotChunk / G;
        int j[R];
        uint4 qj[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int k = s0 + r * G + sub;
            j[r] = k < cnt ? f.nbr[(size_t)k * f.n + i] : i;
        }
#pragma unroll
        for (int r = 0; r < R; r++) qj[r] = f.q[j[r]];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const bool hit = s0 + r * G + sub < cnt && quant_touch(f.sx, f.sy, f.tol, qi, qj[r]);
            const unsigned b = __ballot_sync(0xffffffffu, hit);
            bits |= ((b >> lead) & ((1u << G) - 1u)) << (r * G);
        }
    }
    return bits;
}

// Adds the terms of particle i's pairs (list length cnt; 0 for lanes past the
// last particle, whose i must still be a valid index) to acc: K = 3 force x,
// force y, energy; K = 4 the stress terms xx, xy, yx, yy
// (kernelCalcDiskStressTensor, src/particles/disk/kernels.cu:203-252).  Every
// lane of a group passes the same particle and gets its sums.  All lanes of
// the warp call it.
template <int G, int K>
__device__ __forceinline__ void pair_sums(const PairArgs &f, int i, int cnt, PairWarp<K> &w,
                                          double (&acc)[K]) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, sub = lane & (G - 1), lead = lane - sub;
    const uint4 qi = f.q[i];
    const int most = (int)__reduce_max_sync(kAll, (unsigned)cnt);
    for (int s0 = 0; s0 < most; s0 += kSlotChunk) {
        const unsigned bits = touch_bits<G>(f, i, qi, s0, cnt);
        const int c = __popc(bits);
        // queue offsets: exclusive scan of the particles' counts
        int incl = sub == 0 ? c : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kAll, incl, o);
            if (lane >= o) incl += y;
        }
        const int total = __shfl_sync(kAll, incl, 31);
        const int end = __shfl_sync(kAll, incl, lead), off = end - c;
        // lane sub of the group queues its slots sub, sub + G, ...
        if (G == 1) {
            int at = off;
            for (unsigned m = bits; m; m &= m - 1) w.ent[at++] = (unsigned short)(lane << 5 | (__ffs(m) - 1));
        } else {
#pragma unroll
            for (int r = 0; r < kSlotChunk / G; r++) {
                const int k = r * G + sub;
                if (bits >> k & 1u) w.ent[off + __popc(bits & ((1u << k) - 1u))] = (unsigned short)(lane << 5 | k);
            }
        }
        __syncwarp();
        for (int w0 = 0; w0 < total; w0 += kPairWin) {
            const int w1 = min(total, w0 + kPairWin);
            for (int e0 = w0; e0 < w1; e0 += 32) {
                const int e = e0 + lane;
                const int ent = e < w1 ? w.ent[e] : lane << 5;
                const int io = __shfl_sync(kAll, i, ent >> 5);
                if (e < w1) {
                    const int j = f.nbr[(size_t)(s0 + (ent & 31)) * f.n + io];
                    double dx, dy, fx, fy;
                    const double ri = f.rad ? f.rad[io] : f.rv, rj = f.rad ? f.rad[j] : f.rv;
                    const double ee = disk_pair_sum(f, f.pos[io], ri, f.pos[j], rj, dx, dy, fx, fy);
                    if (K == 3) {
                        w.r[0][e - w0] = fx;
                        w.r[1][e - w0] = fy;
                        w.r[2][e - w0] = ee;
                    } else {
                        w.r[0][e - w0] = dx * fx / 2;
                        w.r[1][e - w0] = dx * fy / 2;
                        w.r[2][e - w0] = dy * fx / 2;
                        w.r[K - 1][e - w0] = dy * fy / 2;
                    }
                }
            }
            __syncwarp();
            const int b0 = max(off, w0) - w0, b1 = min(end, w1) - w0;
            if (G >= K) {  // lanes 0 .. K - 1 of a group add one term each
                double s = acc[0];
#pragma unroll
                for (int k = 1; k < K; k++) s = sub == k ? acc[k] : s;
                if (sub < K)
                    for (int b = b0; b < b1; b++) s += w.r[sub][b];
#pragma unroll
                for (int k = 0; k < K; k++) acc[k] = __shfl_sync(kAll, s, lead + k);
            } else {
                for (int b = b0; b < b1; b++)
#pragma unroll
                    for (int k = 0; k < K; k++) acc[k] += w.r[k][b];
            }
            __syncwarp();
        }
    }
}

// The force sums of one thread's particle without the queue: the FP64
// refinement of a mixed system, whose FP32 kernels should not carry the
// queue's shared memory.
__device__ __forceinline__ void pair_sums_thread(const PairArgs &f, int i, int cnt, double &ax, double &ay,
                                                 double &en) {
    const uint4 qi = f.q[i];
    const double2 pi = f.pos[i];
    const double ri = f.rad[i];
    for (int s0 = 0; s0 < cnt; s0 += kSlotChunk) {
        for (unsigned m = touch_bits<1>(f, i, qi, s0, cnt); m; m &= m - 1) {
            const int j = f.nbr[(size_t)(s0 + __ffs(m) - 1) * f.n + i];
            double dx, dy, fx, fy;
            const double e = disk_pair_sum(f, pi, ri, f.pos[j], f.rad[j], dx, dy, fx, fy);
            ax += fx;
            ay += fy;
            en += e;
        }
    }
}

// Mixed form: FP32 pair forces from the packed offsets, summed in FP32 over
// runs of 8 neighbours and in FP64 across runs and for the particle total.  G
// lanes share a run's pairs (G = 1: the particle's own thread); its terms are
// added in slot order whatever G is.  cnt: the list length, 0 for lanes past
// the last particle.  All lanes of the warp call it.
template <int G>
__device__ __forceinline__ void mixed_sums(const DevParams &p, const float4 *pk, const int *nbr, int i,
                                           int cnt, double &ax, double &ay, double &en) {
    const int n = p.n;
    const float e_c = (float)p.e_c, n_c = (float)p.n_c;
    const float4 a = pk[i];
    ax = 0.0; ay = 0.0; en = 0.0;
    if constexpr (G == 1) {
        for (int k0 = 0; k0 < cnt; k0 += 8) {
            float sx = 0.f, sy = 0.f, se = 0.f;
            const int k1 = min(cnt, k0 + 8);
            for (int k = k0; k < k1; k++) {
                int j = nbr[(size_t)k * n + i];
                float fx, fy;
                se += mixed_pair(p, a, pk[j], e_c, n_c, fx, fy);
                sx += fx;
                sy += fy;
            }
            ax += (double)sx;
            ay += (double)sy;
            en += (double)se;
        }
    } else {
        constexpr int R = 8 / G;
        const int lane = threadIdx.x & 31, sub = lane & (G - 1), lead = lane - sub;
        const int most = (int)__reduce_max_sync(0xffffffffu, (unsigned)cnt);
        for (int k0 = 0; k0 < most; k0 += 8) {
            float fx[R], fy[R], e[R];
#pragma unroll
            for (int r = 0; r < R; r++) {
                const int k = k0 + r * G + sub;
                fx[r] = 0.f; fy[r] = 0.f; e[r] = 0.f;
                if (k < cnt) e[r] = mixed_pair(p, a, pk[nbr[(size_t)k * n + i]], e_c, n_c, fx[r], fy[r]);
            }
            float sx = 0.f, sy = 0.f, se = 0.f;
#pragma unroll
            for (int u = 0; u < 8; u++) {
                sx += __shfl_sync(0xffffffffu, fx[u / G], lead + u % G);
                sy += __shfl_sync(0xffffffffu, fy[u / G], lead + u % G);
                se += __shfl_sync(0xffffffffu, e[u / G], lead + u % G);
            }
            ax += (double)sx;
            ay += (double)sy;
            en += (double)se;
        }
    }
}

// Pair sum of particle i for a force kernel with G threads per particle.  The
// mixed instantiation (M, one thread per particle) uses FP32 pairs; only the
// FIRE force kernel (R) also carries the FP64 pairs of the refinement
// (DevState.fp64_now, clear outside dpg_fire_minimize): with both, the NVE
// kernel took 234 us at 2^20 disks, 160 with the FP32 pairs alone.  All lanes
// of the warp call it.
template <int G, bool M, bool R = false>
__device__ __forceinline__ void force_sum(const DevSys *ds, int i, bool valid, double &ax, double &ay,
                                          double &en) {
    ax = 0.0; ay = 0.0; en = 0.0;
    if constexpr (M) {
        if (!valid) return;
        const int cnt = min(ds->w.count[i], ds->p.cap);
        if (!R || !ds->s.fp64_now) mixed_sums<1>(ds->p, ds->v.pk, ds->v.nbr, i, cnt, ax, ay, en);
        else pair_sums_thread(pair_args(ds), i, cnt, ax, ay, en);
    } else {
        __shared__ ForceWarp w[kForceTPB / 32];
        const int cnt = valid ? min(ds->w.count[i], ds->p.cap) : 0;
        double acc[3] = {0.0, 0.0, 0.0};
        pair_sums<G, 3>(pair_args(ds), valid ? i : 0, cnt, w[threadIdx.x >> 5], acc);
        ax = acc[0]; ay = acc[1]; en = acc[2];
    }
}

// fixed-point positions of every particle from the current positions
__global__ void k_quant(DevSys *ds) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ds->p.n) return;
    ds->v.q[i] = quant_of(ds->p, ds->v.pos[i], ds->v.rad[i]);
}

// the same as the first kernel of a rebuild inside a loop whose move kernel
// does not keep them (mixed form)
__global__ void k_quant_rebuild(DevSys *ds) {
    if (ds->s.rebuild == 0) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ds->p.n) return;
    ds->v.q[i] = quant_of(ds->p, ds->v.pos[i], ds->v.rad[i]);
}

// mixed disk systems only (rigid-body systems keep their vertex offsets in
// BumpyExt and leave the body DevParams at FP64)
__device__ __forceinline__ void mixed_update(DevSys *ds, int i, double2 p) {
    if (ds->p.precision == kMixed && ds->v.pk) ds->v.pk[i] = mixed_pack(ds->p, p, ds->v.rad[i]);
}

// what the loops' move kernels keep current with the positions: the mixed
// form's packed offsets (its FP32 pairs read them), or the fixed-point
// positions (a mixed system's are refreshed when its lists are rebuilt, and on
// every move once its pairs are FP64)
__device__ __forceinline__ void moved_update(DevSys *ds, int i, double2 p) {
    const double r = ds->v.rad[i];
    if (ds->p.precision == kMixed) ds->v.pk[i] = mixed_pack(ds->p, p, r);
    if (ds->p.precision != kMixed || ds->s.fp64_now) ds->v.q[i] = quant_of(ds->p, p, r);
}

// Squared displacements since the last neighbour and cell lists, which have the
// same start as a rule (compared as integers).  The moves are bound by their
// FP64 instructions: with this, unit masses tested and maxima taken as integers
// some 20 instead of 50; k_nve_first of 2^20 disks 97 -> 53 us.
__device__ __forceinline__ void moved2(double2 p, double2 a, double2 c, double (&v)[2]) {
    const double dx = p.x - a.x, dy = p.y - a.y;
    v[0] = v[1] = dx * dx + dy * dy;
    if (__double_as_longlong(a.x) != __double_as_longlong(c.x) || __double_as_longlong(a.y) != __double_as_longlong(c.y)) {
        const double cx = p.x - c.x, cy = p.y - c.y;
        v[1] = cx * cx + cy * cy;
    }
}

// mixed form: offsets of every particle from the current positions
__global__ void k_mixed_refresh(DevSys *ds) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ds->p.n) return;
    ds->v.pk[i] = mixed_pack(ds->p, ds->v.pos[i], ds->v.rad[i]);
}

// device-side neighbour rebuild decision: checkForCellListUpdate /
// checkForVerletListUpdate (src/particles/base/particle.cu:1141-1161), tolerance 3
__device__ __forceinline__ int rebuild_decision(const DevSys *ds, double max_nd2, double max_cd2) {
    const double tol = 3.0;
    if (ds->p.method == 2) return 0;
    if (ds->p.method == 1) return (tol * max_nd2 > ds->p.nthr2) ? 1 : 0;
    if (tol * max_cd2 > ds->p.cthr2) return 2;
    if (tol * max_nd2 > ds->p.nthr2) return 1;
    return 0;
}

// ============================================================================
//  Single operations (drop-in path)
// ============================================================================

// kernelUpdateVelocities: src/particles/base/kernels.cu:117-139
__global__ void k_kick(DevSys *ds, double dt) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ds->p.n) return;
    double2 *vel = ds->v.vel;
    double2 v = vel[i], f = ds->v.frc[i];
    double dtm = dt / ds->v.mass[i];
    v.x = v.x + f.x * dtm;
    v.y = v.y + f.y * dtm;
    vel[i] = v;
}

// kernelUpdatePositions: src/particles/base/kernels.cu:48-81.  The reference's
// per-particle displacement arrays are only ever max-reduced, so the maxima
// are kept instead (grid reduction into DevState).
__global__ void k_drift(DevSys *ds, double dt) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    double v[2] = {0.0, 0.0};
    if (i < ds->p.n) {
        double2 *pos = ds->v.pos;
        double2 p = pos[i], u = ds->v.vel[i];
        p.x = p.x + u.x * dt;
        p.y = p.y + u.y * dt;
        pos[i] = p;
        double2 a = ds->w.pos_n[i], c = ds->w.pos_c[i];
        double dxn = p.x - a.x, dyn = p.y - a.y, dxc = p.x - c.x, dyc = p.y - c.y;
        v[0] = dxn * dxn + dyn * dyn;
        v[1] = dxc * dxc + dyc * dyc;
    }
    const int ops[2] = {1, 1};
    if (grid_reduce<2>(v, ops, ds)) { ds->s.max_nd2 = v[0]; ds->s.max_cd2 = v[1]; }
}

// kernelMixVelocitiesAndForces (per-particle FIRE mix): src/particles/base/kernels.cu:91-112
__device__ __forceinline__ double2 fire_mix(double2 v, double2 f, double alpha) {
    const double f2 = f.x * f.x + f.y * f.y, v2 = v.x * v.x + v.y * v.y;
    const bool nf = __double_as_longlong(f2) == 0, nv = __double_as_longlong(v2) == 0;
    double mix = 0.0;
    if ((nf || middling(f2)) && (nv || middling(v2))) {
        double yf, yv;
        const double fn = nf ? 0.0 : root_near(f2, yf);
        // |F| > 1e-16 by the high word, exactly where that is the same
        const int h = __double2hiint(fn);
        if (h > 0x3c9cd2b2 || (h == 0x3c9cd2b2 && fn > 1e-16)) {
            const double vn = root_near(v2, yv);
            mix = nv ? 0.0 : div_near(vn, fn, yf) * alpha;
        } else {
            v.x = 0.0; v.y = 0.0;
        }
    } else if (const double fn = sqrt(f2); fn > 1e-16) {
        mix = sqrt(v2) / fn * alpha;
    } else {
        v.x = 0.0; v.y = 0.0; mix = 0.0;
    }
    double2 o;
    o.x = v.x * (1 - alpha) + f.x * mix;
    o.y = v.y * (1 - alpha) + f.y * mix;
    return o;
}

__global__ void k_mix(DevSys *ds, double alpha) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ds->p.n) return;
    ds->v.vel[i] = fire_mix(ds->v.vel[i], ds->v.frc[i], alpha);
}

__global__ void k_zero_vel(DevSys *ds) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ds->p.n) return;
    ds->v.vel[i] = make_double2(0.0, 0.0);
}

// kernelZeroForceAndPotentialEnergy: src/particles/base/kernels.cu:150-161
__global__ void k_zero_force(DevSys *ds) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ds->p.n) return;
    ds->v.frc[i] = make_double2(0.0, 0.0);
    ds->w.pe[i] = 0.0;
}

// kernelCalcDiskForces (+= semantics): src/particles/disk/kernels.cu:11-57
template <int G, bool M>
__global__ void k_force_acc(DevSys *ds) {
    const int gid = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = gid / G;
    double ax, ay, en;
    force_sum<G, M>(ds, i, i < ds->p.n, ax, ay, en);
    if (i >= ds->p.n || (gid & (G - 1)) != 0) return;
    if (ds->w.count[i] == 0) return;
    double2 *frc = ds->v.frc;
    double2 f = frc[i];
    f.x += ax;
    f.y += ay;
    frc[i] = f;
    ds->w.pe[i] += en;
}

// ---- pair and Hessian dump -----------------------------------------------------
struct PairOut {
    double *d[16];  // see dpg_pair_dump in include/dpg.h for the order
    long long *this_id, *other_id;
};

// the fills of Disk::calculateForceDistancePairs (src/particles/disk/disk.cu:229-247)
__global__ void k_pair_fill(PairOut o, long long m) {
    long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= m) return;
    const double fill[16] = {-1, 0, 0, -1, -1, -1, -1, -1, 0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int k = 0; k < 16; k++)
        if (o.d[k]) o.d[k][q] = fill[k];
    o.this_id[q] = -1;
    o.other_id[q] = -1;
}

// kernelCalcDiskForceDistancePairs (src/particles/disk/kernels.cu:73-175):
// entry [slot * cap + k] for the k-th neighbour of the particle in slot i
__global__ void k_pair_dump(DevSys *ds, PairOut o) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = ds->p.n, cap = ds->p.cap;
    if (i >= n) return;
    int cnt = ds->w.count[i];
    if (cnt == 0) return;
    if (cnt > cap) cnt = cap;
    const double2 *pos = ds->v.pos;
    const double *rad = ds->v.rad;
    const double2 pi = pos[i];
    const double ri = rad[i];
    const double bx = ds->p.box[0], by = ds->p.box[1], e_c = ds->p.e_c, n_c = ds->p.n_c;
    for (int k = 0; k < cnt; k++) {
        const int j = ds->v.nbr[(size_t)k * n + i];
        const double2 pj = pos[j];
        const double rj = rad[j];
        double fx, fy;
        const double e = disk_pair(pi.x, pi.y, ri, pj.x, pj.y, rj, bx, by, e_c, n_c, fx, fy);
        const long long q = (long long)i * cap + k;
        const double dx = pbc_dist(pi.x, pj.x, bx), dy = pbc_dist(pi.y, pj.y, by);
        if (o.d[0]) o.d[0][q] = e;
        if (o.d[1]) o.d[1][q] = fx;
        if (o.d[2]) o.d[2][q] = fy;
        if (o.d[3]) o.d[3][q] = dx;
        if (o.d[4]) o.d[4][q] = dy;
        o.this_id[q] = ds->v.sidx[i];
        o.other_id[q] = ds->v.sidx[j];
        const double dist = sqrt(dx * dx + dy * dy);
        if (o.d[5]) o.d[5][q] = dist - (ri + rj);
        if (o.d[6]) o.d[6][q] = ri + rj;
        if (o.d[7]) o.d[7][q] = atan2(dy, dx);
        if (dist < ri + rj) {
            const double radsum = ri + rj;
            const double t_ij = -e_c / radsum * (1 - dist / radsum);
            const double c_ij = e_c / (radsum * radsum);
            double hij[4] = {0.0, 0.0, 0.0, 0.0}, hii[4] = {0.0, 0.0, 0.0, 0.0};
            for (int a = 0; a < 2; a++) {
                for (int b = 0; b < 2; b++) {
                    const double dia_x = 1 * (a == 0), dia_y = 1 * (a == 1);
                    const double djb_x = -1 * (b == 0), djb_y = -1 * (b == 1);
                    const double q_ia = dx * dia_x + dy * dia_y;
                    const double q_jb = dx * djb_x + dy * djb_y;
                    const double dia_q_jb = dia_x * djb_x + dx * 0.0 + dia_y * djb_y + dy * 0.0;
                    hij[a * 2 + b] += c_ij * (q_ia * q_jb) / (dist * dist) +
                                      t_ij * (dia_q_jb / dist - (q_ia * q_jb) / (dist * dist * dist));
                    const double dib_x = 1 * (b == 0), dib_y = 1 * (b == 1);
                    const double q_ib = dx * dib_x + dy * dib_y;
                    const double dia_q_ib = dia_x * dib_x + dx * 0.0 + dia_y * dib_y + dy * 0.0;
                    hii[a * 2 + b] += c_ij * (q_ia * q_ib) / (dist * dist) +
                                      t_ij * (dia_q_ib / dist - (q_ia * q_ib) / (dist * dist * dist));
                }
            }
#pragma unroll
            for (int c = 0; c < 4; c++) {
                if (o.d[8 + c]) o.d[8 + c][q] += hij[c];
                if (o.d[12 + c]) o.d[12 + c][q] += hii[c];
            }
        }
    }
}

// calcWallInteraction (include/particles/base/kernels.cuh:185-235): hard walls
// at 0 and L on both axes, terms in the reference's order (left, right,
// bottom, top); returns the energy, force in (fx, fy) summed from 0
__device__ __forceinline__ double wall_force(const DevParams &p, double2 x, double rad,
                                             double &fx, double &fy) {
    const double dist[4] = {x.x, p.box[0] - x.x, x.y, p.box[1] - x.y};
    const bool near[4] = {x.x < rad, x.x > p.box[0] - rad, x.y < rad, x.y > p.box[1] - rad};
    double en = 0.0;
    fx = 0.0;
    fy = 0.0;
#pragma unroll
    for (int w = 0; w < 4; w++) {
        if (!near[w]) continue;
        const double ov = rad - dist[w];
        if (!(ov > 0)) continue;
        const double q = ov / rad;
        const double ovp = p.n_c - 1 == 1.0 ? q : pow(q, p.n_c - 1);
        const double f = p.e_c * ovp / rad;
        if (w == 0) fx += f;
        else if (w == 1) fx -= f;
        else if (w == 2) fy += f;
        else fy -= f;
        en += p.e_c * ov * ovp / (p.n_c * rad);
    }
    return en;
}

// kernelCalcDiskWallForces (+= semantics): src/particles/disk/kernels.cu:59-71
__global__ void k_wall_force(DevSys *ds) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ds->p.n) return;
    double fx, fy;
    double en = wall_force(ds->p, ds->v.pos[i], ds->v.rad[i], fx, fy);
    double2 f = ds->v.frc[i];
    f.x += fx;
    f.y += fy;
    ds->v.frc[i] = f;
    ds->w.pe[i] += en;
}

// kernelCalculateDampedForces: src/particles/base/kernels.cu:83-89
__global__ void k_damp(DevSys *ds, double gamma) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ds->p.n) return;
    double2 f = ds->v.frc[i], u = ds->v.vel[i];
    f.x -= gamma * u.x;
    f.y -= gamma * u.y;
    ds->v.frc[i] = f;
}

// kernelGradDescStep: src/particles/base/kernels.cu:613-637, with the
// displacement maxima kept as in k_drift
__global__ void k_grad_desc(DevSys *ds, double alpha) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    double v[2] = {0.0, 0.0};
    if (i < ds->p.n) {
        double2 *pos = ds->v.pos;
        double2 p = pos[i], f = ds->v.frc[i];
        p.x = p.x + alpha * f.x;
        p.y = p.y + alpha * f.y;
        pos[i] = p;
        double2 a = ds->w.pos_n[i], c = ds->w.pos_c[i];
        double dxn = p.x - a.x, dyn = p.y - a.y, dxc = p.x - c.x, dyc = p.y - c.y;
        v[0] = dxn * dxn + dyn * dyn;
        v[1] = dxc * dxc + dyc * dyc;
    }
    const int ops[2] = {1, 1};
    if (grid_reduce<2>(v, ops, ds)) { ds->s.max_nd2 = v[0]; ds->s.max_cd2 = v[1]; }
}

// PE and KE totals (kernelCalculateTranslationalKineticEnergy + reductions,
// src/particles/base/kernels.cu:163-180, src/particles/base/particle.cu:1074-1080),
// FIRE power P = F.v (src/particles/base/particle.cu:993-1009), max|F|^2 and sum F.
__global__ void k_observables(DevSys *ds) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    double v[6] = {0, 0, 0, 0, 0, 0};
    if (i < ds->p.n) {
        double2 u = ds->v.vel[i], f = ds->v.frc[i];
        double m = ds->v.mass[i];
        double v2 = u.x * u.x + u.y * u.y;
        v[0] = ds->w.pe[i];
        v[1] = 0.5 * m * v2;
        v[2] = f.x * u.x + f.y * u.y;
        v[3] = f.x * f.x + f.y * f.y;
        v[4] = f.x;
        v[5] = f.y;
    }
    const int ops[6] = {0, 0, 0, 1, 0, 0};
    if (grid_reduce<6>(v, ops, ds)) {
        ds->s.pe = v[0]; ds->s.ke = v[1]; ds->s.power = v[2]; ds->s.fmax2 = v[3];
        ds->s.fsum_x = v[4]; ds->s.fsum_y = v[5];
    }
}

// kernelCalcDiskStressTensor: src/particles/disk/kernels.cu:203-252 (summed)
constexpr int kStressTPB = 128;
__global__ void __launch_bounds__(kStressTPB) k_stress(DevSys *ds) {
    __shared__ PairWarp<4> w[kStressTPB / 32];
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = ds->p.n;
    double v[4] = {0, 0, 0, 0};
    const bool valid = i < n;
    if (valid) {
        const double2 u = ds->v.vel[i];
        const double m = ds->v.mass[i];
        v[0] = m * u.x * u.x;
        v[1] = m * u.x * u.y;
        v[2] = v[1];
        v[3] = m * u.y * u.y;
    }
    pair_sums<1, 4>(pair_args(ds), valid ? i : 0, valid ? min(ds->w.count[i], ds->p.cap) : 0,
                    w[threadIdx.x >> 5], v);
    const double area = ds->p.box[0] * ds->p.box[1];
#pragma unroll
    for (int k = 0; k < 4; k++) v[k] = valid ? v[k] / area : 0.0;
    const int ops[4] = {0, 0, 0, 0};
    if (grid_reduce<4>(v, ops, ds))
        for (int k = 0; k < 4; k++) ds->s.stress[k] = v[k];
}

// kernelCountDiskContacts: src/particles/disk/kernels.cu:177-201 (summed); the
// fixed-point distance decides all pairs but those within 1e-5 of touching
__global__ void k_contacts(DevSys *ds) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    double v[1] = {0.0};
    const int n = ds->p.n;
    if (i < n) {
        const PairArgs f = pair_args(ds);
        const uint4 qi = f.q[i];
        int cnt = min(ds->w.count[i], ds->p.cap), c = 0;
        for (int k = 0; k < cnt; k++) {
            const int j = f.nbr[(size_t)k * n + i];
            const uint4 qj = f.q[j];
            const float rs = __uint_as_float(qi.z) + __uint_as_float(qj.z), d2 = quant_d2(f.sx, f.sy, qi, qj);
            const float lo = rs * 0.99999f - f.tol, hi = rs * 1.00001f + f.tol;
            if (d2 > hi * hi) continue;
            if (lo > 0.f && d2 < lo * lo && rs < INFINITY) { c++; continue; }
            const double2 pi = f.pos[i], pj = f.pos[j];
            const double dx = pbc_dist(pi.x, pj.x, f.bx), dy = pbc_dist(pi.y, pj.y, f.by);
            if (sqrt(dx * dx + dy * dy) < f.rad[i] + f.rad[j]) c++;
        }
        v[0] = (double)c;
    }
    const int ops[1] = {0};
    if (grid_reduce<1>(v, ops, ds)) ds->s.contacts = v[0];
}

// kernelAdamStep: src/particles/base/kernels.cu:550-611
__global__ void k_adam(DevSys *ds, double alpha, double b1, double b2, double c1, double c2,
                       double eps) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    double v[2] = {0.0, 0.0};
    if (i < ds->p.n) {
        double2 f = ds->v.frc[i], m1 = ds->v.m1[i], m2 = ds->v.m2[i];
        m1.x = fma(b1, m1.x, (b1 - 1) * f.x);
        m1.y = fma(b1, m1.y, (b1 - 1) * f.y);
        m2.x = fma(b2, m2.x, (1 - b2) * f.x * f.x);
        m2.y = fma(b2, m2.y, (1 - b2) * f.y * f.y);
        double mhx = m1.x / c1, mhy = m1.y / c1, vhx = m2.x / c2, vhy = m2.y / c2;
        double ux = -alpha * mhx / (sqrt(vhx) + eps);
        double uy = -alpha * mhy / (sqrt(vhy) + eps);
        double2 *pos = ds->v.pos;
        double2 p = pos[i];
        p.x += ux;
        p.y += uy;
        pos[i] = p;
        double2 a = ds->w.pos_n[i], c = ds->w.pos_c[i];
        double dxn = p.x - a.x, dyn = p.y - a.y, dxc = p.x - c.x, dyc = p.y - c.y;
        v[0] = dxn * dxn + dyn * dyn;
        v[1] = dxc * dxc + dyc * dyc;
        ds->v.m1[i] = m1;
        ds->v.m2[i] = m2;
    }
    const int ops[2] = {1, 1};
    if (grid_reduce<2>(v, ops, ds)) { ds->s.max_nd2 = v[0]; ds->s.max_cd2 = v[1]; }
}

// scalePositions / scalePositionsFull (src/particles/base/particle.cu:1066-1072)
__global__ void k_scale_pos(DevSys *ds, double f) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ds->p.n) return;
    double2 p = ds->v.pos[i];
    p.x *= f;
    p.y *= f;
    ds->v.pos[i] = p;
}

// ============================================================================
//  Neighbour rebuild (each kernel does nothing unless DevState.rebuild asks)
// ============================================================================

__global__ void k_set_rebuild(DevSys *ds, int kind) { ds->s.rebuild = kind; }

// host-independent decision from the stored displacement maxima
__global__ void k_decide_rebuild(DevSys *ds) {
    if (halted(ds)) { ds->s.rebuild = 0; return; }
    ds->s.rebuild = rebuild_decision(ds, ds->s.max_nd2, ds->s.max_cd2);
}

// kernelGetCellIndexForParticle (src/particles/base/kernels.cu:309-330) + counts
__global__ void k_cell_index(DevSys *ds) {
    if (ds->s.rebuild != 2) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ds->p.n) return;
    double2 p = ds->v.pos[i];
    const int ncd = ds->p.ncd;
    const double cs = ds->p.cell_size;
    int c = cell_coord(p.x, cs, ncd) + cell_coord(p.y, cs, ncd) * ncd;
    ds->w.cell_raw[i] = c;
    atomicAdd(&ds->w.cell_cnt[c], 1);
}

// exclusive scan of the per-cell counts into CSR starts (one block)
__global__ void __launch_bounds__(kScanTPB) k_cell_scan(DevSys *ds) {
    if (ds->s.rebuild != 2) return;
    __shared__ int wsum[kScanTPB / 32];
    __shared__ int carry_s;
    const int ncells = ds->p.ncells;
    const int *cnt = ds->w.cell_cnt;
    int *start = ds->w.cell_start;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int carry = 0;
    for (int base = 0; base < ncells; base += 4 * kScanTPB) {
        int idx = base + 4 * threadIdx.x;
        int a[4];
#pragma unroll
        for (int k = 0; k < 4; k++) a[k] = (idx + k < ncells) ? cnt[idx + k] : 0;
        int t = a[0] + a[1] + a[2] + a[3];
        int incl = t;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += y;
        }
        if (lane == 31) wsum[wid] = incl;
        __syncthreads();
        if (wid == 0) {
            int w = wsum[lane];
            int wi = w;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                int y = __shfl_up_sync(0xffffffffu, wi, off);
                if (lane >= off) wi += y;
            }
            wsum[lane] = wi - w;  // exclusive warp offsets
            if (lane == 31) carry_s = wi;
        }
        __syncthreads();
        int ex = carry + wsum[wid] + incl - t;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (idx + k < ncells) start[idx + k] = ex;
            ex += a[k];
        }
        carry += carry_s;
        __syncthreads();
    }
    if (threadIdx.x == 0) start[ncells] = carry;
}

__global__ void k_cell_scatter(DevSys *ds) {
    if (ds->s.rebuild != 2) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ds->p.n) return;
    int c = ds->w.cell_raw[i];
    int slot = ds->w.cell_start[c] + atomicAdd(&ds->w.cell_cur[c], 1);
    ds->w.perm[slot] = i;
}

// Within each cell, restore ascending particle order: the result is the
// permutation of a stable sort by cell (thrust::sort_by_key in
// src/particles/base/particle.cu:1293).  Also clears the counters.
__device__ __forceinline__ void cell_sort_one(DevSys *ds, int c) {
    int b = ds->w.cell_start[c], e = ds->w.cell_start[c + 1];
    int *perm = ds->w.perm;
    for (int k = b + 1; k < e; k++) {
        int key = perm[k];
        int j = k - 1;
        while (j >= b && perm[j] > key) { perm[j + 1] = perm[j]; j--; }
        perm[j + 1] = key;
    }
    ds->w.cell_cnt[c] = 0;
    ds->w.cell_cur[c] = 0;
}

__global__ void k_cell_sort(DevSys *ds) {
    if (ds->s.rebuild != 2) return;
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < ds->p.ncells) cell_sort_one(ds, c);
}

// kernelReorderParticleData (src/particles/base/kernels.cu:508-543) into the
// alternate buffers, then (last block) swap current/alternate on the device.
// The Adam moments are swapped with their twins without a gather, as the
// reference does (src/particles/base/particle.cu:1302-1303).
__global__ void k_reorder(DevSys *ds) {
    if (ds->s.rebuild != 2) return;
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < ds->p.n) {
        int o = ds->w.perm[s];
        const DevView &v = ds->v;
        double2 p = v.pos[o];
        v.pos_t[s] = p;
        v.vel_t[s] = v.vel[o];
        v.frc_t[s] = v.frc[o];
        v.rad_t[s] = v.rad[o];
        v.mass_t[s] = v.mass[o];
        v.sidx_t[s] = v.sidx[o];
        v.q[s] = quant_of(ds->p, p, v.rad[o]);  // nothing in this kernel reads q
        ds->w.cell_of[s] = ds->w.cell_raw[o];
        ds->w.pos_c[s] = p;
    }
    if (grid_last_block(ds)) {
        DevView &v = ds->v;
        swap_ptr(v.pos, v.pos_t);
        swap_ptr(v.vel, v.vel_t);
        swap_ptr(v.frc, v.frc_t);
        swap_ptr(v.rad, v.rad_t);
        swap_ptr(v.mass, v.mass_t);
        swap_ptr(v.sidx, v.sidx_t);
        swap_ptr(v.m1, v.m1_t);
        swap_ptr(v.m2, v.m2_t);
        ds->s.max_cd2 = 0.0;
        ds->s.n_cell_rebuilds++;
    }
}

__device__ __forceinline__ void finish_list_build(DevSys *ds, int cnt) {
    double v[1] = {(double)cnt};
    const int ops[1] = {1};
    if (grid_reduce<1>(v, ops, ds)) {
        int mx = (int)v[0];
        ds->s.max_count = mx;
        if (mx > ds->p.cap) ds->s.flags |= kOverflow;
        ds->s.max_nd2 = 0.0;
        ds->s.n_rebuilds++;
        ds->s.rebuild = 0;
    }
}

// d2 < cutoff2 for particles i and j, decided by the fixed-point distance where
// it can, by the FP64 test of the reference where it cannot
__device__ __forceinline__ bool within(const DevParams &p, const double2 *a, int i, const double2 *b, int j,
                                       uint4 qi, uint4 qj, float in2, float out2, double c2) {
    const float d2 = quant_d2(p.q_s[0], p.q_s[1], qi, qj);
    const bool marked = (qi.w | qj.w) != 0;
    if (!marked && d2 > out2) return false;
    if (!marked && d2 < in2) return true;
    const double2 pi = a[i], pj = b[j];
    const double dx = pbc_dist(pi.x, pj.x, p.box[0]), dy = pbc_dist(pi.y, pj.y, p.box[1]);
    return dx * dx + dy * dy < c2;
}
__device__ __forceinline__ bool within_cutoff(const DevSys *ds, const double2 *pos, int i, int j, uint4 qi,
                                              uint4 qj) {
    return within(ds->p, pos, i, pos, j, qi, qj, ds->p.q_in2, ds->p.q_out2, ds->p.cutoff2);
}

// The neighbour row of particle i from the 3x3 cells around its own
// (kernelUpdateCellNeighborList, src/particles/base/kernels.cu:440-505: dy
// outer, dx inner, ascending slot inside each cell), G lanes per particle.
// The three cells of a row hold consecutive slots (two ranges where the row
// wraps), so the group reads G neighbouring 16-byte entries at a time; ballots
// give each hit its place.  Returns the row's length (every lane of the group).
// Bound: the FP64 distance tests took 2.7 ms for 2^20 disks; the filter leaves
// one in ~1e5 of them and the pass runs on FP32 and L1: 209 us with one lane a
// particle, 106 -> 16 us for 16384 disks with eight.  All lanes of the warp
// call it, with valid = false past the last particle.
template <int G>
__device__ __forceinline__ int nlist_row(const DevSys *ds, int i, bool valid) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, sub = lane & (G - 1), lead = lane - sub;
    const int n = ds->p.n, ncd = ds->p.ncd, cap = ds->p.cap;
    const double2 *pos = ds->v.pos;
    const uint4 *q = ds->v.q;
    const int *cstart = ds->w.cell_start;
    int *nbr = ds->v.nbr;
    const int c = valid ? ds->w.cell_of[i] : 0, cx = c % ncd, cy = c / ncd;
    const uint4 qi = q[valid ? i : 0];
    int cnt = 0;
    for (int oy = -1; oy <= 1; oy++) {
        const int row = pmod(cy + oy, ncd) * ncd;
        // cells cx - 1, cx, cx + 1 in this order, as up to two slot ranges
        int b[2] = {0, 0}, e[2] = {0, 0};
        if (valid) {
            const int x0 = cx == 0 ? ncd - 1 : cx - 1;
            b[0] = cstart[row + x0];
            if (cx == 0) {
                e[0] = cstart[row + ncd];
                b[1] = cstart[row];
                e[1] = cstart[row + 2];
            } else if (cx == ncd - 1) {
                e[0] = cstart[row + ncd];
                b[1] = cstart[row];
                e[1] = cstart[row + 1];
            } else {
                e[0] = cstart[row + cx + 2];
            }
        }
#pragma unroll
        for (int g = 0; g < 2; g++) {
            if (G == 1) {
                for (int j = b[g]; j < e[g]; j++) {
                    if (j == i || !within_cutoff(ds, pos, i, j, qi, q[j])) continue;
                    if (cnt < cap) nbr[(size_t)cnt * n + i] = j;
                    cnt++;
                }
            } else {
                const int rounds = (int)__reduce_max_sync(kAll, (unsigned)((e[g] - b[g] + G - 1) / G));
                for (int r = 0; r < rounds; r++) {
                    const int j = b[g] + r * G + sub;
                    const bool hit = j < e[g] && j != i && within_cutoff(ds, pos, i, j, qi, q[j]);
                    const unsigned m = (__ballot_sync(kAll, hit) >> lead) & ((1u << G) - 1u);
                    const int at = cnt + __popc(m & ((1u << sub) - 1u));
                    if (hit && at < cap) nbr[(size_t)at * n + i] = j;
                    cnt += __popc(m);
                }
            }
        }
    }
    return cnt;
}

template <int G>
__global__ void k_nlist_cell(DevSys *ds) {
    if (ds->s.rebuild == 0) return;
    const int gid = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = gid / G;
    const bool valid = i < ds->p.n;
    const int cnt = nlist_row<G>(ds, i, valid);
    if (valid && (gid & (G - 1)) == 0) {
        const double2 pi = ds->v.pos[i];
        ds->w.count[i] = cnt;
        ds->w.pos_n[i] = pi;
        mixed_update(ds, i, pi);
    }
    finish_list_build(ds, valid ? cnt : 0);
}

// kernelUpdateNeighborList (all pairs, methods "verlet" / "all"):
// src/particles/base/kernels.cu:256-293.  j tiles staged in shared memory.
__global__ void k_nlist_all(DevSys *ds) {
    if (ds->s.rebuild == 0) return;
    __shared__ uint4 tile[kTPB];
    const int n = ds->p.n;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    const double2 *pos = ds->v.pos;
    const uint4 *q = ds->v.q;
    int *nbr = ds->v.nbr;
    const int cap = ds->p.cap;
    const uint4 qi = q[i < n ? i : 0];
    int cnt = 0;
    for (int base = 0; base < n; base += kTPB) {
        int j0 = base + threadIdx.x;
        if (j0 < n) tile[threadIdx.x] = q[j0];
        __syncthreads();
        int lim = min(kTPB, n - base);
        if (i < n) {
            for (int t = 0; t < lim; t++) {
                int j = base + t;
                if (j == i || !within_cutoff(ds, pos, i, j, qi, tile[t])) continue;
                if (cnt < cap) nbr[(size_t)cnt * n + i] = j;
                cnt++;
            }
        }
        __syncthreads();
    }
    if (i < n) {
        const double2 pi = pos[i];
        ds->w.count[i] = cnt;
        ds->w.pos_n[i] = pi;
        mixed_update(ds, i, pi);
    }
    finish_list_build(ds, cnt);
}

// ============================================================================
//  Fused loops
// ============================================================================

// NVE::step first half (src/integrator/nve.cu:16-17): kick dt/2, drift dt,
// displacement maxima and the rebuild decision.
__global__ void k_nve_first(DevSys *ds, double dt_half, double dt) {
    if (halted(ds)) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    double v[2] = {0.0, 0.0};
    if (i < ds->p.n) {
        double2 *vel = ds->v.vel, *pos = ds->v.pos;
        double2 u = vel[i], f = ds->v.frc[i], p = pos[i];
        const double dtm = over_mass(dt_half, ds->v.mass[i]);
        u.x = u.x + f.x * dtm;
        u.y = u.y + f.y * dtm;
        vel[i] = u;
        p.x = p.x + u.x * dt;
        p.y = p.y + u.y * dt;
        pos[i] = p;
        moved_update(ds, i, p);
        moved2(p, ds->w.pos_n[i], ds->w.pos_c[i], v);
    }
    if (grid_max<2>(v, ds)) {
        ds->s.max_nd2 = v[0];
        ds->s.max_cd2 = v[1];
        int rb = rebuild_decision(ds, v[0], v[1]);
        ds->s.rebuild = rb;
        if (ds->s.h_rb) cudaGraphSetConditional(ds->s.h_rb, rb != 0);
    }
}

// force and energy of particle i in an NVE step from its pair sums (ax, ay, en)
// and its velocity u, overwriting
__device__ __forceinline__ double2 nve_force(const DevSys *ds, int i, double2 u, double ax, double ay,
                                             double en, double &pe) {
    double2 f;
    const double g = ds->s.damping;
    pe = en;  // 0 + en: a sum that starts at +0 is never -0
    if (ds->s.walls) {
        // NVE::wall_step (src/integrator/nve.cu:33-35): zero, wall forces,
        // then += the pair sum unless the particle has no neighbours
        double wx, wy;
        const double ew = wall_force(ds->p, ds->v.pos[i], ds->v.rad[i], wx, wy);
        f = make_double2(0.0 + wx, 0.0 + wy);
        pe = 0.0 + ew;
        if (ds->w.count[i] != 0) { f.x += ax; f.y += ay; pe += en; }
    } else if (__double_as_longlong(g) << 1 != 0) {  // g != 0
        // DampedNVE::step (src/integrator/damped_nve.cu:22-23): F = 0 - g v,
        // then += the pair sum unless the particle has no neighbours
        f = make_double2(0.0 - g * u.x, 0.0 - g * u.y);
        if (ds->w.count[i] != 0) { f.x += ax; f.y += ay; }
    } else {
        f = make_double2(ax, ay);
    }
    return f;
}

// NVE::step second half (src/integrator/nve.cu:21-24): zero, forces, kick dt/2.
template <int G, bool M>
__global__ void k_nve_second(DevSys *ds, double dt_half) {
    if (halted(ds)) return;
    const int gid = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = gid / G;
    double ax, ay, en;
    force_sum<G, M>(ds, i, i < ds->p.n, ax, ay, en);
    if (i < ds->p.n && (gid & (G - 1)) == 0) {
        double2 *vel = ds->v.vel;
        double2 u = vel[i];
        double pe;
        const double2 f = nve_force(ds, i, u, ax, ay, en, pe);
        ds->v.frc[i] = f;
        ds->w.pe[i] = pe;
        const double dtm = over_mass(dt_half, ds->v.mass[i]);
        u.x = u.x + f.x * dtm;
        u.y = u.y + f.y * dtm;
        vel[i] = u;
    }
    if (grid_last_block(ds)) {
        if (++ds->s.nve_steps_done >= ds->s.max_steps) ds->s.flags |= kDone;
    }
}

// ---- FIRE -------------------------------------------------------------------

// Fire::step prologue (src/integrator/fire.cu:13-34): decide dt / alpha from
// the power of the state the next step starts from.
__device__ __forceinline__ void fire_decide(DevState &s, double power) {
    if (power > 0) {
        s.f_ngood++;
        s.f_nbad = 0;
        if (s.f_ngood > 5) {
            s.f_dt = fmin(s.f_dt * 1.1, s.f_dtmax);
            s.f_alpha *= 0.99;
        }
        s.fire_uphill = 0;
    } else {
        s.f_ngood = 0;
        s.f_nbad++;
        if (s.f_nbad > 10) {
            s.f_stopped = 1;
            s.fire_uphill = 0;
            s.flags |= kDone;
            return;
        }
        s.f_dt = fmax(s.f_dt * 0.5, s.f_dtmin);
        s.f_alpha = s.f_alpha0;
        s.fire_uphill = 1;
    }
}

// FIRE move: uphill rollback (x -= v dt/2, v = 0), kick dt/2, per-particle
// mix, drift dt (src/integrator/fire.cu:29-40), displacement maxima and the
// rebuild decision.
__global__ void k_fire_move(DevSys *ds) {
    if (halted(ds)) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    const double dt = ds->s.f_dt, alpha = ds->s.f_alpha;
    const int up = ds->s.fire_uphill;
    double v[2] = {0.0, 0.0};
    if (i < ds->p.n) {
        double2 *vel = ds->v.vel, *pos = ds->v.pos;
        double2 u = vel[i], f = ds->v.frc[i], p = pos[i];
        if (up) {
            double back = -dt / 2.0;
            p.x = p.x + u.x * back;
            p.y = p.y + u.y * back;
            u = make_double2(0.0, 0.0);
        }
        const double dtm = over_mass(dt / 2.0, ds->v.mass[i]);
        u.x = u.x + f.x * dtm;
        u.y = u.y + f.y * dtm;
        u = fire_mix(u, f, alpha);
        vel[i] = u;
        p.x = p.x + u.x * dt;
        p.y = p.y + u.y * dt;
        pos[i] = p;
        moved_update(ds, i, p);
        moved2(p, ds->w.pos_n[i], ds->w.pos_c[i], v);
    }
    if (grid_max<2>(v, ds)) {
        ds->s.max_nd2 = v[0];
        ds->s.max_cd2 = v[1];
        int rb = rebuild_decision(ds, v[0], v[1]);
        ds->s.rebuild = rb;
        if (ds->s.h_rb) cudaGraphSetConditional(ds->s.h_rb, rb != 0);
    }
}

// Mean energy of a FIRE iteration (s.pe) and whether it has stopped changing.
// Where no test reads it the FP64 division stays off the iteration's serial path
// (0: below no target).
__device__ __forceinline__ bool fire_energy(DevState &s, double &avg) {
    avg = 0.0;
    if (!s.pe_read) return false;
    avg = s.pe / s.dof;
    const bool still = s.pe_diff_target > 0 && fabs(avg / s.last_avg_pe - 1) < s.pe_diff_target;
    s.last_avg_pe = avg;
    return still;
}

// Mixed form: FP32 pairs until max|F| reaches switch_fmax, FIRE keeps going
// uphill, or max|F| stops falling within 100x of switch_fmax (FP32 noise
// floor); FP64 pairs after.  f2: max|F|^2 of the iteration.
__device__ __forceinline__ void fire_switch(DevState &s, double f2) {
    if (f2 < 0.81 * s.best_f2) { s.best_f2 = f2; s.best_it = s.iter; }
    bool go = s.f_nbad > 5;
    // above 100 switch_fmax (which may be 0, as may f2) the root is not needed to tell
    if (!go && !(f2 > 1.001e4 * s.switch_fmax * s.switch_fmax)) {
        const double fm = sqrt(f2);
        go = fm <= s.switch_fmax || (fm < 100.0 * s.switch_fmax && s.iter - s.best_it > 2000);
    }
    if (go) s.fp64_now = 1;
}

// End of a FIRE iteration, from its totals (PE, power, max|F|^2): the
// minimizeFire convergence tests (src/routines/minimization.cu:96-106) and the
// next step's Fire::step decision.
template <bool M>
__device__ __forceinline__ void fire_epilogue(DevState &s, const double (&v)[3]) {
    s.pe = v[0];
    s.power = v[1];
    s.fmax2 = v[2];
    double avg;
    const bool pe_still = fire_energy(s, avg);
    long long it = s.iter;
    // only an FP64 state may pass the PE-change and max|F| tests
    const bool fp64 = !M || s.fp64_now;
    if (!fp64) fire_switch(s, v[2]);
    if ((fp64 && pe_still) || avg < s.pe_target) {
        s.result_step = it; s.f_converged = 1; s.flags |= kDone; return;
    }
    if (fp64 && s.fmax_target > 0 && sqrt(v[2]) <= s.fmax_target) {
        s.result_step = it; s.f_converged = 1; s.flags |= kDone; return;
    }
    if (it + 1 >= s.max_steps) { s.result_step = s.max_steps; s.flags |= kDone; return; }
    s.iter = it + 1;
    fire_decide(s, v[1]);
    if (s.f_stopped) { s.result_step = it + 1; s.f_converged = 1; s.flags |= kDone; }
}

// FIRE force phase: forces (overwrite), kick dt/2, then on the last block
// fire_epilogue.  mode 0 = loop iteration, 1 = setup
// (forces only: minimizeFire's initial force call and last_avg_pe), 2 = a
// single Fire::step (no convergence test, decision for the next step only).
template <int G, bool M>
__global__ void k_fire_force(DevSys *ds, int mode) {
    if (halted(ds)) return;
    const int gid = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = gid / G;
    double v[3] = {0.0, 0.0, 0.0};
    double ax, ay, en;
    force_sum<G, M, true>(ds, i, i < ds->p.n, ax, ay, en);
    if (i < ds->p.n && (gid & (G - 1)) == 0) {
        double2 f = make_double2(0.0 + ax, 0.0 + ay);
        ds->v.frc[i] = f;
        ds->w.pe[i] = 0.0 + en;
        double2 *vel = ds->v.vel;
        double2 u = vel[i];
        if (mode != 1) {
            const double dtm = over_mass(ds->s.f_dt / 2.0, ds->v.mass[i]);
            u.x = u.x + f.x * dtm;
            u.y = u.y + f.y * dtm;
            vel[i] = u;
        }
        v[0] = 0.0 + en;
        v[1] = f.x * u.x + f.y * u.y;
        v[2] = f.x * f.x + f.y * f.y;
    }
    const int ops[3] = {0, 0, 1};
    if (!grid_reduce<3>(v, ops, ds)) return;
    DevState &s = ds->s;
    if (mode == 0) {
        fire_epilogue<M>(s, v);
        return;
    }
    s.pe = v[0];
    s.power = v[1];
    s.fmax2 = v[2];
    if (mode == 1) {
        s.last_avg_pe = v[0] / s.dof;
        fire_decide(s, v[1]);
        if (s.f_stopped) { s.result_step = 0; s.flags |= kDone; }
    }
}

// Fire::step prologue for a single step: P = F.v over the grid, then decide.
__global__ void k_fire_power_decide(DevSys *ds) {
    if (halted(ds)) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    double v[1] = {0.0};
    if (i < ds->p.n) {
        double2 u = ds->v.vel[i], f = ds->v.frc[i];
        v[0] = f.x * u.x + f.y * u.y;
    }
    const int ops[1] = {0};
    if (grid_reduce<1>(v, ops, ds)) {
        ds->s.power = v[0];
        fire_decide(ds->s, v[0]);
    }
}

// Last node of every WHILE body: continue only while no flag is raised and
// the iteration budget is not spent.  Guarantees the loop terminates.
__global__ void k_loop_guard(DevSys *ds) {
    DevState &s = ds->s;
    long long g = ++s.guard;
    int go = (s.flags == 0) && (g < s.guard_limit);
    if (!go && s.flags == 0) s.flags |= kError;
    if (s.h_loop) cudaGraphSetConditional(s.h_loop, go ? 1u : 0u);
}

// ============================================================================
//  State transfer (static order <-> sorted slots)
// ============================================================================

// which: 0 pos, 1 vel, 2 frc ; xy from separate x / y arrays in static order
__global__ void k_put_xy(DevSys *ds, int which, const double *x, const double *y) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ds->p.n) return;
    int k = ds->v.sidx[i];
    double2 *dst = which == 0 ? ds->v.pos : (which == 1 ? ds->v.vel : ds->v.frc);
    double2 o = dst[i];
    if (x) o.x = x[k];
    if (y) o.y = y[k];
    dst[i] = o;
}

// which: 0 rad, 1 mass
__global__ void k_put_scalar(DevSys *ds, int which, const double *a) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ds->p.n) return;
    int k = ds->v.sidx[i];
    (which == 0 ? ds->v.rad : ds->v.mass)[i] = a[k];
}

// which: 0 pos, 1 vel, 2 frc
__global__ void k_get_xy(DevSys *ds, int which, double *x, double *y) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ds->p.n) return;
    int k = ds->v.sidx[i];
    const double2 *src = which == 0 ? ds->v.pos : (which == 1 ? ds->v.vel : ds->v.frc);
    double2 o = src[i];
    if (x) x[k] = o.x;
    if (y) y[k] = o.y;
}

// which: 0 radii, 1 masses (static order out)
__global__ void k_get_scalar(DevSys *ds, int which, double *out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ds->p.n) return;
    out[ds->v.sidx[i]] = (which == 0 ? ds->v.rad : ds->v.mass)[i];
}

__global__ void k_get_pe(DevSys *ds, double *out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ds->p.n) return;
    out[ds->v.sidx[i]] = ds->w.pe[i];
}

__global__ void k_iota_sidx(DevSys *ds) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ds->p.n) return;
    ds->v.sidx[i] = i;
}

// neighbour rows in static indices, row-major [n][cap_out], -1 padded
__global__ void k_get_nbrs(DevSys *ds, int *list, int *counts, int cap_out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = ds->p.n;
    if (i >= n) return;
    const int *sidx = ds->v.sidx;
    int k = sidx[i];
    int cnt = ds->w.count[i];
    counts[k] = cnt;
    int lim = min(cnt, min(cap_out, ds->p.cap));
    for (int t = 0; t < cap_out; t++)
        list[(size_t)k * cap_out + t] = t < lim ? sidx[ds->v.nbr[(size_t)t * n + i]] : -1;
}

__global__ void k_get_cells(DevSys *ds, long long *cell_index, long long *cell_start,
                            long long *static_index) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < ds->p.n) {
        if (cell_index) cell_index[i] = ds->w.cell_of[i];
        if (static_index) static_index[i] = ds->v.sidx[i];
    }
    if (cell_start && i <= ds->p.ncells) {
        int b = ds->w.cell_start[i];
        if (i == ds->p.ncells) cell_start[i] = b;
        else cell_start[i] = (ds->w.cell_start[i + 1] > b) ? b : -1;
    }
}

// setLastState (dir = 0) / revertToLastStateVariables (dir = 1)
__global__ void k_snapshot(DevSys *ds, int dir) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ds->p.n) return;
    DevView &v = ds->v;
    DevScratch &w = ds->w;
    if (dir == 0) {
        w.s_pos[i] = v.pos[i]; w.s_vel[i] = v.vel[i]; w.s_frc[i] = v.frc[i];
        w.s_rad[i] = v.rad[i]; w.s_mass[i] = v.mass[i]; w.s_sidx[i] = v.sidx[i];
    } else {
        v.pos[i] = w.s_pos[i]; v.vel[i] = w.s_vel[i]; v.frc[i] = w.s_frc[i];
        v.rad[i] = w.s_rad[i]; v.mass[i] = w.s_mass[i]; v.sidx[i] = w.s_sidx[i];
    }
}

}  // namespace
}  // namespace dpg
