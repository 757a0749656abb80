// bumpy_kernels.cuh -- plain FP64 kernels for rigid bumpy bodies (rigid bodies
// made of vertex disks on a circle), the drop-in form of
// src/particles/rigid_bumpy/{rigid_bumpy.cu,kernels.cu}.
//
// Layout: BumpySys embeds the disk DevSys as its first member, with the BODIES
// in the disk slots (pos, vel, frc, rad, mass, sidx, body neighbour list, cell
// list), so the disk cell-list and body neighbour kernels run unchanged on the
// bodies.  BumpyExt adds the rotational body fields and the vertices; vertices
// of a body are contiguous ([start[b], start[b] + nvb[b])) and move as a block
// when bodies are re-sorted, like the reference.
//
// Vertex work runs warp-per-body: lane l owns vertices start + l, start + l +
// 32, ...; a body's force, torque and energy are summed over its vertices in
// vertex order with warp shuffles, which reproduces the reference's sequential
// per-body sum (kernelCalcRigidBumpyParticleForces1) bit for bit.
// Compiled with --fmad=false (reference operation order).
#pragma once
#include "disk_kernels.cuh"

namespace dpg {
namespace {  // kernels have internal linkage: each translation unit owns its copy

struct BumpyExt {
    int nv, capv, rotation, max_vcount;
    int max_nvb;             // most vertices of a body
    double rv, vcut2, vpcut2;
    double *w, *th, *tq, *I;  // angular velocity, angle, torque, moment of inertia
    int *nvb, *start;
    double *w_t, *th_t, *tq_t, *I_t;
    int *nvb_t, *start_t;
    double2 *vpos, *vpos_t;
    double *vmass, *vmass_t;
    int *vbody, *vbody_t, *svidx, *svidx_t;
    int *vnbr, *vcount;      // vertex neighbour list, column-major [capv][nv]
    float4 *vpk;             // mixed form: packed FP32 vertex offsets (see mixed_pack)
    uint4 *vq;               // fixed-point vertex positions (see Quant in dpg_device.cuh)
    float4 *vpk_t;           // the other buffers of vpk and vq (NVE in the resident grid)
    uint4 *vq_t;
    float vin2, vout2, vpin2, vpout2;  // filter limits of the two vertex-list cutoffs
    int mixed;               // 1: FP32 vertex pairs (the body DevParams stay FP64)
    long long vlist_built;   // n_rebuilds value at the last vertex-list build
    double tmax2, power_rot;
    // snapshot of the rotational state (setLastState)
    double *s_w, *s_th, *s_tq;
    double2 *s_vpos;
    int *s_nvb, *s_start, *s_vbody, *s_svidx;
    // per slot, never re-sorted (like the reference's angle_delta and angular
    // Adam moments): the last angle increment and the angular Adam moments
    double *adelta, *m1a, *m2a;
    // per-body results of the stress and contact passes (body-slot order)
    double *stress_b;   // [4][nb]: xx, xy, yx, yy
    int *ccount, *vccount;
    double vcontacts;
};

struct BumpySys {
    DevSys b;  // must stay first: BumpySys* is passed as DevSys* to the disk kernels
    BumpyExt x;
};

constexpr int kWarpsPerBlock = kTPB / 32;
constexpr int kMoveBodies = 32;  // bodies per block of the move kernels

// calcTorque: include/particles/base/kernels.cuh:237-241
__device__ __forceinline__ double torque_of(double fx, double fy, double px, double py, double cx,
                                           double cy) {
    double dx = px - cx, dy = py - cy;
    return fy * dx - fx * dy;
}

// ---- body kick: kernelUpdateRigidVelocities (kernels.cu:123-150) -----------
__device__ __forceinline__ void body_kick(BumpySys *bs, int b, double dt) {
    DevSys &d = bs->b;
    double2 v = d.v.vel[b], f = d.v.frc[b];
    double m = d.v.mass[b];
    double w = bs->x.w[b];
    if (bs->x.rotation) w += bs->x.tq[b] * dt / bs->x.I[b];
    else w = 0.0;
    v.x += f.x * dt / m;
    v.y += f.y * dt / m;
    d.v.vel[b] = v;
    bs->x.w[b] = w;
}

__global__ void kb_kick(BumpySys *bs, double dt) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= bs->b.p.n) return;
    body_kick(bs, b, dt);
}

// ---- body + vertex move: kernelUpdateRigidPositions + kernelTranslateAndRotateVertices1
// (kernels.cu:21-78,152-201) of the bodies [b0, b1) by a block.  The body part
// (kick, displacement, cosine and sine of the increment: some 130 FP64
// instructions, each of which holds an FP64 pipe for all 32 lanes whatever
// their number) runs on one thread a body; a warp a body spent them once per
// body.  The vertices then turn with one thread each.  kMoveBodies bodies at a
// time; every thread of the block calls it.
struct MoveMem {
    double2 p[kMoveBodies], n[kMoveBodies], cs[kMoveBodies];
};
// pre(b): what a body does before it moves (thread of the body); vpos, vpk, vq:
// where the moved vertices go, with what the pair loops read of them (see
// moved_update)
template <class F>
__device__ __forceinline__ void bodies_move(BumpySys *bs, int b0, int b1, double dt, MoveMem &m, F pre,
                                            double &nd2, double &cd2, double2 *vpos, float4 *vpk, uint4 *vq) {
    DevSys &d = bs->b;
    BumpyExt &x = bs->x;
    for (int base = b0; base < b1; base += kMoveBodies) {
        const int nbod = min(kMoveBodies, b1 - base);
        if (threadIdx.x < nbod) {
            const int b = base + threadIdx.x;
            pre(b);
            const double2 p = d.v.pos[b], u = d.v.vel[b];
            const double ang = x.th[b], w = x.w[b];
            const double ddx = u.x * dt, ddy = u.y * dt, dth = w * dt;
            const double nx = p.x + ddx, ny = p.y + ddy;
            d.v.pos[b] = make_double2(nx, ny);
            x.th[b] = ang + dth;
            x.adelta[b] = dth;
            const double2 a = d.w.pos_n[b], c = d.w.pos_c[b];
            const double a1 = nx - a.x, a2 = ny - a.y, c1 = nx - c.x, c2 = ny - c.y;
            nd2 = fmax(nd2, a1 * a1 + a2 * a2);
            cd2 = fmax(cd2, c1 * c1 + c2 * c2);
            m.p[threadIdx.x] = p;
            m.n[threadIdx.x] = make_double2(nx, ny);
            m.cs[threadIdx.x] = make_double2(cos(dth), sin(dth));
        }
        __syncthreads();
        const int v0 = x.start[base], last = base + nbod - 1, v1 = x.start[last] + x.nvb[last];
        for (int v = v0 + threadIdx.x; v < v1; v += blockDim.x) {
            const int k = x.vbody[v] - base;
            const double2 q = x.vpos[v], p = m.p[k], n = m.n[k], cs = m.cs[k];
            const double rx = q.x - p.x, ry = q.y - p.y;
            const double rxr = rx * cs.x - ry * cs.y, ryr = rx * cs.y + ry * cs.x;
            const double2 nq = make_double2(n.x + rxr, n.y + ryr);
            vpos[v] = nq;
            if (x.mixed) vpk[v] = mixed_pack(d.p, nq, x.rv);
            if (!x.mixed || d.s.fp64_now) vq[v] = quant_of(d.p, nq, x.rv);
        }
        __syncthreads();
    }
}

__global__ void kb_drift(BumpySys *bs, double dt) {
    __shared__ MoveMem m;
    const int b0 = blockIdx.x * kMoveBodies, b1 = min(b0 + kMoveBodies, bs->b.p.n);
    double v[2] = {0.0, 0.0};
    bodies_move(bs, b0, b1, dt, m, [](int) {}, v[0], v[1], bs->x.vpos, bs->x.vpk, bs->x.vq);
    const int ops[2] = {1, 1};
    if (grid_reduce<2>(v, ops, &bs->b)) { bs->b.s.max_nd2 = v[0]; bs->b.s.max_cd2 = v[1]; }
}

// ---- forces: kernelCalcRigidBumpyForces1 + kernelCalcRigidBumpyParticleForces1
// (kernels.cu:366-442) fused, one warp per body.  The vertex pairs run through
// the filter and the warp's queue (pair_sums); the body's force, torque and
// energy are then added over its vertices in vertex order by four lanes, one
// sum each, skipping the vertices without a term (+0.0 leaves such a sum as it
// is).  Lanes 0 - 3 return the force x, force y, torque and energy of the body.
// walls: kernelCalcRigidBumpyWallForces (kernels.cu:348-362) first, as
// NVE::wall_step calls it before the pairs, so a vertex carries (0 + wall) +
// pair sum.
__device__ __forceinline__ PairArgs vertex_args(const BumpySys *bs) {
    PairArgs f = pair_args(&bs->b);
    f.pos = bs->x.vpos;
    f.rad = nullptr;
    f.rv = bs->x.rv;
    f.nbr = bs->x.vnbr;
    f.q = bs->x.vq;
    f.n = bs->x.nv;
    return f;
}

__device__ __forceinline__ double body_forces(const BumpySys *bs, int b, bool walls, ForceWarp &fw) {
    const DevSys &d = bs->b;
    const BumpyExt &x = bs->x;
    const int lane = threadIdx.x & 31, capv = x.capv;
    const double rv = x.rv;
    const double2 c = d.v.pos[b];
    const int f = x.start[b], nvb = x.nvb[b];
    const bool mixed = x.mixed && !d.s.fp64_now;
    const PairArgs fa = vertex_args(bs);
    double sum = 0.0;
    for (int base = 0; base < nvb; base += 32) {
        const int k = base + lane, v = f + k;
        const bool real = k < nvb;
        const int cnt = real ? min(x.vcount[v], capv) : 0;
        double t[3] = {0.0, 0.0, 0.0};  // pair sums: force x, force y, energy
        if (mixed) {                    // FP32 vertex pairs; torque and body sums stay FP64
            if (real) {
                const float4 a = x.vpk[v];
                const float e_c = (float)d.p.e_c, n_c = (float)d.p.n_c;
                float sx = 0.f, sy = 0.f, se = 0.f;
                for (int q = 0; q < cnt; q++) {
                    float fx, fy;
                    se += mixed_pair(d.p, a, x.vpk[x.vnbr[(size_t)q * fa.n + v]], e_c, n_c, fx, fy);
                    sx += fx;
                    sy += fy;
                }
                t[0] = (double)sx;
                t[1] = (double)sy;
                t[2] = (double)se;
            }
        } else {
            pair_sums<1, 3>(fa, real ? v : f, cnt, fw, t);
        }
        double vf[4] = {0.0, 0.0, 0.0, 0.0};  // the vertex: force x, force y, torque, energy
        bool some = t[0] != 0.0 || t[1] != 0.0 || t[2] != 0.0;
        const double2 q = x.vpos[real ? v : f];
        if (walls && real) {
            double wx, wy;
            const double we = wall_force(d.p, q, rv, wx, wy);
            vf[0] = 0.0 + wx;
            vf[1] = 0.0 + wy;
            vf[2] = 0.0 + torque_of(wx, wy, q.x, q.y, c.x, c.y);
            vf[3] = 0.0 + we;
            some = true;
        }
        if (some) {
            vf[0] = vf[0] + t[0];
            vf[1] = vf[1] + t[1];
            vf[2] = vf[2] + torque_of(t[0], t[1], q.x, q.y, c.x, c.y);
            vf[3] = vf[3] + t[2];
        }
        __syncwarp();
        // the queue's result rows hold the four terms of 32 vertices
#pragma unroll
        for (int e = 0; e < 4; e++) fw.r[0][e * 32 + lane] = vf[e];
        __syncwarp();
        unsigned todo = __ballot_sync(0xffffffffu, some);
        if (lane < 4)
            for (; todo; todo &= todo - 1) sum += fw.r[0][lane * 32 + __ffs(todo) - 1];
        __syncwarp();
    }
    return sum;
}

// mixed form: packed offsets of every vertex from the current vertex positions
__global__ void kb_mixed_refresh(BumpySys *bs) {
    int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= bs->x.nv) return;
    bs->x.vpk[v] = mixed_pack(bs->b.p, bs->x.vpos[v], bs->x.rv);
}

// fixed-point positions of every vertex
__global__ void kb_vquant(BumpySys *bs) {
    int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= bs->x.nv) return;
    bs->x.vq[v] = quant_of(bs->b.p, bs->x.vpos[v], bs->x.rv);
}

// the same ahead of a vertex-list build, for the systems whose move kernels do
// not keep them
__global__ void kb_vquant_rebuild(BumpySys *bs) {
    if (bs->b.s.n_rebuilds == bs->x.vlist_built) return;
    int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= bs->x.nv) return;
    bs->x.vq[v] = quant_of(bs->b.p, bs->x.vpos[v], bs->x.rv);
}

// drop-in calculateForces (+= into the body arrays); walls = 1: calculateWallForces
// then calculateForces
__global__ void kb_force_acc(BumpySys *bs, int walls) {
    __shared__ ForceWarp fw[kWarpsPerBlock];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int b = blockIdx.x * kWarpsPerBlock + wid;
    if (b >= bs->b.p.n) return;
    const double sum = body_forces(bs, b, walls != 0, fw[wid]);
    if (lane == 0) bs->b.v.frc[b].x += sum;
    if (lane == 1) bs->b.v.frc[b].y += sum;
    if (lane == 2) bs->x.tq[b] += sum;
    if (lane == 3) bs->b.w.pe[b] += sum;
}

// zeroForceAndPotentialEnergy (rigid_bumpy.cu:1378-1381); vertex arrays are not kept
__global__ void kb_zero_force(BumpySys *bs) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= bs->b.p.n) return;
    bs->b.v.frc[b] = make_double2(0.0, 0.0);
    bs->x.tq[b] = 0.0;
    bs->b.w.pe[b] = 0.0;
}

// kernelMixRigidVelocitiesAndForces (kernels.cu:89-121)
__device__ __forceinline__ void body_mix(BumpySys *bs, int b, double alpha) {
    double2 f = bs->b.v.frc[b], v = bs->b.v.vel[b];
    double fn = sqrt(f.x * f.x + f.y * f.y), vn = sqrt(v.x * v.x + v.y * v.y), mix = 0.0;
    if (fn > 1e-16) mix = vn / fn * alpha;
    else { v.x = 0.0; v.y = 0.0; }
    double w = bs->x.w[b], t = bs->x.tq[b];
    double tn = fabs(t), wn = fabs(w), tmix = 0.0;
    if (tn > 1e-16) tmix = wn / tn * alpha;
    else { w = 0.0; tmix = 0.0; }
    double2 o;
    o.x = v.x * (1 - alpha) + f.x * mix;
    o.y = v.y * (1 - alpha) + f.y * mix;
    bs->b.v.vel[b] = o;
    bs->x.w[b] = w * (1 - alpha) + t * tmix;
}

__global__ void kb_mix(BumpySys *bs, double alpha) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= bs->b.p.n) return;
    body_mix(bs, b, alpha);
}

__global__ void kb_zero_vel(BumpySys *bs) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= bs->b.p.n) return;
    bs->b.v.vel[b] = make_double2(0.0, 0.0);
    bs->x.w[b] = 0.0;
}

// PE, KE (kernelCalculateTranslationalAndRotationalKineticEnergy, kernels.cu:254-269),
// FIRE power incl. the rotational part (rigid_bumpy.cu:1181-1190), max|F|^2, max tau^2
__global__ void kb_observables(BumpySys *bs) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    double v[5] = {0, 0, 0, 0, 0};
    if (b < bs->b.p.n) {
        double2 u = bs->b.v.vel[b], f = bs->b.v.frc[b];
        double m = bs->b.v.mass[b], w = bs->x.w[b], t = bs->x.tq[b];
        v[0] = bs->b.w.pe[b];
        v[1] = bs->x.rotation ? 0.5 * m * (u.x * u.x + u.y * u.y) + 0.5 * bs->x.I[b] * w * w
                              : 0.5 * m * (u.x * u.x + u.y * u.y);
        v[2] = f.x * u.x + f.y * u.y + t * w;
        v[3] = f.x * f.x + f.y * f.y;
        v[4] = t * t;
    }
    const int ops[5] = {0, 0, 0, 1, 1};
    if (grid_reduce<5>(v, ops, &bs->b)) {
        bs->b.s.pe = v[0]; bs->b.s.ke = v[1]; bs->b.s.power = v[2]; bs->b.s.fmax2 = v[3];
        bs->x.tmax2 = v[4];
    }
}

// ---- vertex neighbour list: kernelUpdateVertexNeighborList (kernels.cu:870-922):
// vertices within the vertex cutoff, over the body's neighbour bodies (those
// whose centre is within the body cutoff of the vertex) in list order, vertices
// ascending.  A warp takes 32 vertices of a body, one a lane.  For each listed
// body its lanes first load 32 of that body's vertices side by side and drop
// those out of reach of every vertex of their own body (triangle inequality
// over the body's centre); the few that are left go round the warp by shuffles.
// The fixed-point filter decides all but ~1e-5 of the tests.  `rows`: the
// warp's listed bodies [t0, t1); cnt: the row's length so far; write: entries
// are stored.  All lanes of the warp call it with the same body.
__device__ __forceinline__ void vlist_scan(BumpySys *bs, int b, int v, bool real, uint4 qv, float reach, int t0,
                                           int t1, bool write, int &cnt) {
    constexpr unsigned kAll = 0xffffffffu;
    const DevSys &d = bs->b;
    BumpyExt &x = bs->x;
    const DevParams &p = d.p;
    const int lane = threadIdx.x & 31, nb = p.n, nv = x.nv, capv = x.capv;
    const uint4 qb = d.v.q[b];
    for (int r0 = t0; r0 < t1; r0 += 32) {
        // the listed bodies, one a lane: all their loads in flight together, and
        // the next body's vertices while this one's are tested
        const int rows = min(32, t1 - r0);
        const int ob_l = lane < rows ? d.v.nbr[(size_t)(r0 + lane) * nb + b] : 0;
        const uint4 q_l = d.v.q[ob_l];
        const int of_l = x.start[ob_l], on_l = x.nvb[ob_l];
        auto vertex_of = [&](int r) {
            const int of = __shfl_sync(kAll, of_l, r), on = __shfl_sync(kAll, on_l, r);
            return x.vq[of + (lane < on ? lane : 0)];
        };
        uint4 next = vertex_of(0);
        for (int r = 0; r < rows; r++) {
            const int ob = __shfl_sync(kAll, ob_l, r), of = __shfl_sync(kAll, of_l, r), on = __shfl_sync(kAll, on_l, r);
            const uint4 qo = make_uint4(__shfl_sync(kAll, q_l.x, r), __shfl_sync(kAll, q_l.y, r), 0u,
                                        __shfl_sync(kAll, q_l.w, r));
            uint4 qu = next;
            if (r + 1 < rows) next = vertex_of(r + 1);
            const bool near = real && within(p, x.vpos, v, d.v.pos, ob, qv, qo, x.vpin2, x.vpout2, x.vpcut2);
            if (!__any_sync(kAll, near)) continue;
            for (int u0 = 0; u0 < on; u0 += 32) {
                const bool there = u0 + lane < on;
                if (u0) qu = x.vq[of + (there ? u0 + lane : 0)];
                const bool close = there && ((qu.w | qb.w) != 0 || !(quant_d2(p.q_s[0], p.q_s[1], qu, qb) > reach * reach));
                for (unsigned todo = __ballot_sync(kAll, close); todo; todo &= todo - 1) {
                    const int src = __ffs(todo) - 1, u = of + u0 + src;
                    const uint4 qw = make_uint4(__shfl_sync(kAll, qu.x, src), __shfl_sync(kAll, qu.y, src), 0u,
                                                __shfl_sync(kAll, qu.w, src));
                    if (near && within(p, x.vpos, v, x.vpos, u, qv, qw, x.vin2, x.vout2, x.vcut2)) {
                        if (write && cnt < capv) x.vnbr[(size_t)cnt * nv + v] = u;
                        cnt++;
                    }
                }
            }
        }
    }
}

// how far from its centre a vertex of another body can be and still be in the
// row of one of the warp's vertices (real lanes)
__device__ __forceinline__ float vlist_reach(const BumpySys *bs, uint4 qb, uint4 qv, bool real) {
    const DevParams &p = bs->b.p;
    const float d = real ? sqrtf(quant_d2(p.q_s[0], p.q_s[1], qv, qb)) : 0.f;
    const float most = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(d)));
    if (__any_sync(0xffffffffu, real && qv.w != 0)) return INFINITY;
    return (most + sqrtf(bs->x.vout2)) * 1.00001f + 2.f * p.q_tol;
}

// Runs only when the body list was rebuilt since the last vertex build; a warp
// a body.
__global__ void kb_vlist(BumpySys *bs) {
    if (bs->b.s.n_rebuilds == bs->x.vlist_built) return;
    BumpyExt &x = bs->x;
    const int lane = threadIdx.x & 31, b = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    int mx = 0;
    if (b < bs->b.p.n) {
        const int f = x.start[b], nvb = x.nvb[b], rows = min(bs->b.w.count[b], bs->b.p.cap);
        for (int base = 0; base < nvb; base += 32) {
            const bool real = base + lane < nvb;
            const int v = f + (real ? base + lane : 0);
            const uint4 qv = x.vq[v];
            int cnt = 0;
            vlist_scan(bs, b, v, real, qv, vlist_reach(bs, bs->b.v.q[b], qv, real), 0, rows, true, cnt);
            if (!real) continue;
            x.vcount[v] = cnt;
            if (x.mixed) x.vpk[v] = mixed_pack(bs->b.p, x.vpos[v], x.rv);
            mx = max(mx, cnt);
        }
    }
    double val[1] = {(double)mx};
    const int ops[1] = {1};
    if (grid_reduce<1>(val, ops, &bs->b)) {
        int m = (int)val[0];
        x.max_vcount = m;
        if (m > x.capv) bs->b.s.flags |= kOverflow;
        x.vlist_built = bs->b.s.n_rebuilds;
    }
}

// ---- re-sort of bodies and their vertex blocks:
// RigidBumpy::reorderParticleData (rigid_bumpy.cu:1303-1376, kernels.cu:796-868)
__device__ __forceinline__ void reorder_body(BumpySys *bs, int s) {
    DevSys &d = bs->b;
    BumpyExt &x = bs->x;
    int o = d.w.perm[s];
    double2 p = d.v.pos[o];
    d.v.pos_t[s] = p;
    d.v.vel_t[s] = d.v.vel[o];
    d.v.frc_t[s] = d.v.frc[o];
    d.v.rad_t[s] = d.v.rad[o];
    d.v.mass_t[s] = d.v.mass[o];
    d.v.sidx_t[s] = d.v.sidx[o];
    d.v.q[s] = quant_of(d.p, p, d.v.rad[o]);  // nothing in this kernel reads q
    x.w_t[s] = x.w[o];
    x.th_t[s] = x.th[o];
    x.tq_t[s] = x.tq[o];
    x.I_t[s] = x.I[o];
    x.nvb_t[s] = x.nvb[o];
    d.w.cell_of[s] = d.w.cell_raw[o];
    d.w.pos_c[s] = p;
}

__global__ void kb_reorder_bodies(BumpySys *bs) {
    if (bs->b.s.rebuild != 2) return;
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < bs->b.p.n) reorder_body(bs, s);
}

// exclusive scan of the re-sorted vertex counts into the new block starts (one block)
__global__ void __launch_bounds__(kScanTPB) kb_scan_starts(BumpySys *bs) {
    if (bs->b.s.rebuild != 2) return;
    __shared__ int wsum[kScanTPB / 32];
    __shared__ int carry_s;
    const int nb = bs->b.p.n;
    const int *cnt = bs->x.nvb_t;
    int *start = bs->x.start_t;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int carry = 0;
    for (int base = 0; base < nb; base += kScanTPB) {
        int idx = base + threadIdx.x;
        int a = idx < nb ? cnt[idx] : 0;
        int incl = a;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += y;
        }
        if (lane == 31) wsum[wid] = incl;
        __syncthreads();
        if (wid == 0) {
            int w = wsum[lane], wi = w;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                int y = __shfl_up_sync(0xffffffffu, wi, off);
                if (lane >= off) wi += y;
            }
            wsum[lane] = wi - w;
            if (lane == 31) carry_s = wi;
        }
        __syncthreads();
        if (idx < nb) start[idx] = carry + wsum[wid] + incl - a;
        carry += carry_s;
        __syncthreads();
    }
}

// move the vertex block of new body s to its new start, one warp
__device__ __forceinline__ void reorder_vertices(BumpySys *bs, int s, int lane) {
    BumpyExt &x = bs->x;
    int o = bs->b.w.perm[s];
    int of = x.start[o], nf = x.start_t[s], n = x.nvb_t[s];
    for (int k = lane; k < n; k += 32) {
        x.vpos_t[nf + k] = x.vpos[of + k];
        x.vmass_t[nf + k] = x.vmass[of + k];
        x.svidx_t[nf + k] = x.svidx[of + k];
        x.vbody_t[nf + k] = s;
    }
}

// after a re-sort: the sorted buffers become the current ones
__device__ __forceinline__ void swap_sorted(BumpySys *bs) {
    DevView &v = bs->b.v;
    BumpyExt &x = bs->x;
    swap_ptr(v.pos, v.pos_t); swap_ptr(v.vel, v.vel_t); swap_ptr(v.frc, v.frc_t);
    swap_ptr(v.rad, v.rad_t); swap_ptr(v.mass, v.mass_t); swap_ptr(v.sidx, v.sidx_t);
    swap_ptr(v.m1, v.m1_t); swap_ptr(v.m2, v.m2_t);
    swap_ptr(x.w, x.w_t); swap_ptr(x.th, x.th_t); swap_ptr(x.tq, x.tq_t); swap_ptr(x.I, x.I_t);
    swap_ptr(x.nvb, x.nvb_t); swap_ptr(x.start, x.start_t);
    swap_ptr(x.vpos, x.vpos_t); swap_ptr(x.vmass, x.vmass_t);
    swap_ptr(x.vbody, x.vbody_t); swap_ptr(x.svidx, x.svidx_t);
}

// the vertex blocks (warp per new body), then the swap (last block)
__global__ void kb_reorder_vertices(BumpySys *bs) {
    if (bs->b.s.rebuild != 2) return;
    const int s = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    if (s < bs->b.p.n) reorder_vertices(bs, s, threadIdx.x & 31);
    if (grid_last_block(&bs->b)) {
        swap_sorted(bs);
        bs->b.s.max_cd2 = 0.0;
        bs->b.s.n_cell_rebuilds++;
    }
}

// ---- fused loops ------------------------------------------------------------

// NVE::step first half with the rigid overrides: kick dt/2, move dt
__global__ void kb_nve_first(BumpySys *bs, double dt_half, double dt) {
    if (halted(&bs->b)) return;
    __shared__ MoveMem m;
    const int b0 = blockIdx.x * kMoveBodies, b1 = min(b0 + kMoveBodies, bs->b.p.n);
    double v[2] = {0.0, 0.0};
    bodies_move(bs, b0, b1, dt, m, [&](int b) { body_kick(bs, b, dt_half); }, v[0], v[1],
                bs->x.vpos, bs->x.vpk, bs->x.vq);
    const int ops[2] = {1, 1};
    if (grid_reduce<2>(v, ops, &bs->b)) {
        DevSys *ds = &bs->b;
        ds->s.max_nd2 = v[0];
        ds->s.max_cd2 = v[1];
        int rb = rebuild_decision(ds, v[0], v[1]);
        ds->s.rebuild = rb;
        if (ds->s.h_rb) cudaGraphSetConditional(ds->s.h_rb, rb != 0);
    }
}

// a body's new force, torque and energy (overwriting) from its sums, and the
// kick dt/2 that follows in an NVE step
__device__ __forceinline__ void body_nve_second(BumpySys *bs, int b, double fx, double fy, double tq,
                                                double pe, double dt_half) {
    const double g = bs->b.s.damping;
    if (g != 0.0) {
        // DampedNVE::step (src/integrator/damped_nve.cu:22-23) with
        // kernelCalculateRigidDampedForces (kernels.cu:80-87): body
        // F = 0 - g v, tau = 0 - g omega, then += the vertex sums
        const double2 u = bs->b.v.vel[b];
        const double w = bs->x.w[b];
        bs->b.v.frc[b] = make_double2((0.0 - g * u.x) + fx, (0.0 - g * u.y) + fy);
        bs->x.tq[b] = (0.0 - g * w) + tq;
    } else {
        bs->b.v.frc[b] = make_double2(0.0 + fx, 0.0 + fy);
        bs->x.tq[b] = 0.0 + tq;
    }
    bs->b.w.pe[b] = 0.0 + pe;
    body_kick(bs, b, dt_half);
}

// The sums of the bodies [b0, b1), a warp a body, into sm[body - b0][4], at
// most kWarpsPerBlock bodies; ends with a barrier.  The threads of the first
// b1 - b0 bodies then update them side by side.
__device__ __forceinline__ void block_forces(const BumpySys *bs, int b0, int b1, bool walls, ForceWarp *fw,
                                             double (*sm)[4]) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, b = b0 + wid;
    if (b < b1) {
        const double sum = body_forces(bs, b, walls, fw[wid]);
        if (lane < 4) sm[wid][lane] = sum;
    }
    __syncthreads();
}

// second half: forces (overwrite) + kick dt/2
__global__ void kb_nve_second(BumpySys *bs, double dt_half) {
    if (halted(&bs->b)) return;
    __shared__ ForceWarp fw[kWarpsPerBlock];
    __shared__ double sm[kWarpsPerBlock][4];
    const int b0 = blockIdx.x * kWarpsPerBlock, b1 = min(b0 + kWarpsPerBlock, bs->b.p.n), t = threadIdx.x;
    block_forces(bs, b0, b1, bs->b.s.walls != 0, fw, sm);
    if (t < b1 - b0) body_nve_second(bs, b0 + t, sm[t][0], sm[t][1], sm[t][2], sm[t][3], dt_half);
    if (grid_last_block(&bs->b)) {
        if (++bs->b.s.nve_steps_done >= bs->b.s.max_steps) bs->b.s.flags |= kDone;
    }
}

// FIRE move (src/integrator/fire.cu:29-40 with the rigid overrides)
__device__ __forceinline__ void bodies_fire_move(BumpySys *bs, int b0, int b1, MoveMem &m, double &nd2,
                                                 double &cd2) {
    DevSys *ds = &bs->b;
    const double dt = ds->s.f_dt, alpha = ds->s.f_alpha;
    const int up = ds->s.fire_uphill;
    if (up) {
        double t0 = 0.0, t1 = 0.0;
        bodies_move(bs, b0, b1, -dt / 2.0, m, [](int) {}, t0, t1, bs->x.vpos, bs->x.vpk, bs->x.vq);
    }
    bodies_move(bs, b0, b1, dt, m, [&](int b) {
        if (up) {
            ds->v.vel[b] = make_double2(0.0, 0.0);
            bs->x.w[b] = 0.0;
        }
        body_kick(bs, b, dt / 2.0);
        body_mix(bs, b, alpha);
    }, nd2, cd2, bs->x.vpos, bs->x.vpk, bs->x.vq);
}

__global__ void kb_fire_move(BumpySys *bs) {
    DevSys *ds = &bs->b;
    if (halted(ds)) return;
    __shared__ MoveMem m;
    const int b0 = blockIdx.x * kMoveBodies, b1 = min(b0 + kMoveBodies, ds->p.n);
    double v[2] = {0.0, 0.0};
    bodies_fire_move(bs, b0, b1, m, v[0], v[1]);
    const int ops[2] = {1, 1};
    if (grid_reduce<2>(v, ops, ds)) {
        ds->s.max_nd2 = v[0];
        ds->s.max_cd2 = v[1];
        int rb = rebuild_decision(ds, v[0], v[1]);
        ds->s.rebuild = rb;
        if (ds->s.h_rb) cudaGraphSetConditional(ds->s.h_rb, rb != 0);
    }
}

// a body's new force, torque and energy from its sums and the FIRE kick; adds
// its terms of the totals: PE, power, max|F|^2, max tau^2
__device__ __forceinline__ void body_fire_second(BumpySys *bs, int b, double fx, double fy, double tq,
                                                 double pe, bool kick, double (&v)[4]) {
    DevSys *ds = &bs->b;
    const double2 f = make_double2(0.0 + fx, 0.0 + fy);
    ds->v.frc[b] = f;
    bs->x.tq[b] = 0.0 + tq;
    ds->w.pe[b] = 0.0 + pe;
    if (kick) body_kick(bs, b, ds->s.f_dt / 2.0);
    const double2 u = ds->v.vel[b];
    const double w = bs->x.w[b], t = 0.0 + tq;
    v[0] += 0.0 + pe;
    v[1] += f.x * u.x + f.y * u.y + t * w;
    v[2] = fmax(v[2], f.x * f.x + f.y * f.y);
    v[3] = fmax(v[3], t * t);
}

// End of a FIRE iteration of rigid bodies (see fire_epilogue)
__device__ __forceinline__ void bumpy_fire_epilogue(BumpySys *bs, const double (&v)[4], double tmax_target) {
    DevState &s = bs->b.s;
    s.pe = v[0];
    s.power = v[1];
    s.fmax2 = v[2];
    bs->x.tmax2 = v[3];
    double avg;
    const bool pe_still = fire_energy(s, avg);
    long long it = s.iter;
    // mixed form: FP32 vertex pairs until the switch (as k_fire_force), then FP64
    const bool fp64 = !bs->x.mixed || s.fp64_now;
    if (!fp64) fire_switch(s, max_pos(v[2], v[3]));
    if ((fp64 && pe_still) || avg < s.pe_target) {
        s.result_step = it; s.f_converged = 1; s.flags |= kDone; return;
    }
    if (fp64 && s.fmax_target > 0 && sqrt(v[2]) <= s.fmax_target && sqrt(v[3]) <= tmax_target) {
        s.result_step = it; s.f_converged = 1; s.flags |= kDone; return;
    }
    if (it + 1 >= s.max_steps) { s.result_step = s.max_steps; s.flags |= kDone; return; }
    s.iter = it + 1;
    fire_decide(s, v[1]);
    if (s.f_stopped) { s.result_step = it + 1; s.f_converged = 1; s.flags |= kDone; }
}

// FIRE force phase (see k_fire_force for the modes); the stop test uses
// max|F_b| <= fmax_target and max|tau_b| <= tmax_target.
__global__ void kb_fire_force(BumpySys *bs, int mode, double tmax_target) {
    DevSys *ds = &bs->b;
    if (halted(ds)) return;
    __shared__ ForceWarp fw[kWarpsPerBlock];
    __shared__ double sm[kWarpsPerBlock][4];
    const int b0 = blockIdx.x * kWarpsPerBlock, b1 = min(b0 + kWarpsPerBlock, ds->p.n), t = threadIdx.x;
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    block_forces(bs, b0, b1, false, fw, sm);
    if (t < b1 - b0) body_fire_second(bs, b0 + t, sm[t][0], sm[t][1], sm[t][2], sm[t][3], mode != 1, v);
    const int ops[4] = {0, 0, 1, 1};
    if (!grid_reduce<4>(v, ops, ds)) return;
    if (mode == 0) {
        bumpy_fire_epilogue(bs, v, tmax_target);
        return;
    }
    DevState &s = ds->s;
    s.pe = v[0];
    s.power = v[1];
    s.fmax2 = v[2];
    bs->x.tmax2 = v[3];
    if (mode == 1) {
        s.last_avg_pe = v[0] / s.dof;
        fire_decide(s, v[1]);
    }
}

// FIRE power incl. rotation, then the Fire::step decision (single-step API)
__global__ void kb_fire_power_decide(BumpySys *bs) {
    DevSys *ds = &bs->b;
    if (halted(ds)) return;
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    double v[1] = {0.0};
    if (b < ds->p.n) {
        double2 u = ds->v.vel[b], f = ds->v.frc[b];
        v[0] = f.x * u.x + f.y * u.y + bs->x.tq[b] * bs->x.w[b];
    }
    const int ops[1] = {0};
    if (grid_reduce<1>(v, ops, ds)) {
        ds->s.power = v[0];
        fire_decide(ds->s, v[0]);
    }
}

// ---- initialisation and transfers -------------------------------------------

// kernelInitializeVerticesOnParticles (kernels.cu:1137-1162), warp per body
__global__ void kb_init_vertices(BumpySys *bs) {
    const int lane = threadIdx.x & 31;
    const int b = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    if (b >= bs->b.p.n) return;
    BumpyExt &x = bs->x;
    double2 c = bs->b.v.pos[b];
    double ang = x.th[b], r = bs->b.v.rad[b];
    int nvb = x.nvb[b], f = x.start[b];
    double inc = 2 * 3.14159265358979323846 / nvb;
    double ir = r - x.rv;
    for (int i = lane; i < nvb; i += 32) {
        double a = i * inc + ang;
        x.vpos[f + i] = make_double2(c.x + ir * cos(a), c.y + ir * sin(a));
    }
}

// vertex -> body index and block starts from the counts (host-computed starts)
__global__ void kb_index_vertices(BumpySys *bs) {
    const int lane = threadIdx.x & 31;
    const int b = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    if (b >= bs->b.p.n) return;
    BumpyExt &x = bs->x;
    int f = x.start[b], n = x.nvb[b];
    for (int k = lane; k < n; k += 32) {
        x.vbody[f + k] = b;
        x.svidx[f + k] = f + k;
    }
}

// RigidBumpy::setMass: vertex masses m/nv and I = sum m_v |v - c|^2
// (rigid_bumpy.cu:1068-1080, kernels.cu:1164-1189), warp per body
__global__ void kb_set_mass(BumpySys *bs, double mass) {
    const int lane = threadIdx.x & 31;
    const int b = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    if (b >= bs->b.p.n) return;
    BumpyExt &x = bs->x;
    int f = x.start[b], n = x.nvb[b];
    double2 c = bs->b.v.pos[b];
    if (lane == 0) bs->b.v.mass[b] = mass;
    double mv = mass / (double)n;
    for (int k = lane; k < n; k += 32) x.vmass[f + k] = mv;
    double acc = 0.0;
    for (int base = 0; base < n; base += 32) {
        int k = base + lane;
        double term = 0.0;
        if (k < n) {
            double2 q = x.vpos[f + k];
            double rx = q.x - c.x, ry = q.y - c.y;
            term = mv * (rx * rx + ry * ry);
        }
        int lim = min(32, n - base);
        for (int l = 0; l < lim; l++) acc += __shfl_sync(0xffffffffu, term, l);
    }
    if (lane == 0) x.I[b] = acc;
}

// radii, masses, vertex counts and vertex masses in static (vertex) order
__global__ void kb_get_static(BumpySys *bs, double *rad, double *mass, int *nvb, double *vmass) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < bs->b.p.n) {
        const int k = bs->b.v.sidx[i];
        if (rad) rad[k] = bs->b.v.rad[i];
        if (mass) mass[k] = bs->b.v.mass[i];
        if (nvb) nvb[k] = bs->x.nvb[i];
    }
    if (vmass && i < bs->x.nv) vmass[bs->x.svidx[i]] = bs->x.vmass[i];
}

// body masses, moments of inertia and vertex masses from static-order arrays
// (the values a state directory holds, as loadDataFromPath sets them)
__global__ void kb_put_mass(BumpySys *bs, const double *mass, const double *inertia,
                            const double *vmass) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < bs->b.p.n) {
        const int k = bs->b.v.sidx[i];
        bs->b.v.mass[i] = mass[k];
        bs->x.I[i] = inertia[k];
    }
    if (i < bs->x.nv) bs->x.vmass[i] = vmass[bs->x.svidx[i]];
}

// which: 0 angle, 1 angular velocity, 2 torque ; static order in/out
__global__ void kb_put_body_scalar(BumpySys *bs, int which, const double *a) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= bs->b.p.n) return;
    int k = bs->b.v.sidx[b];
    double *dst = which == 0 ? bs->x.th : (which == 1 ? bs->x.w : bs->x.tq);
    dst[b] = a[k];
}

__global__ void kb_get_body_scalar(BumpySys *bs, int which, double *a) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= bs->b.p.n) return;
    int k = bs->b.v.sidx[b];
    const double *src = which == 0 ? bs->x.th : (which == 1 ? bs->x.w : (which == 2 ? bs->x.tq : bs->x.I));
    a[k] = src[b];
}

__global__ void kb_put_vertices(BumpySys *bs, const double *px, const double *py) {
    int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= bs->x.nv) return;
    int k = bs->x.svidx[v];
    bs->x.vpos[v] = make_double2(px[k], py[k]);
}

__global__ void kb_get_vertices(BumpySys *bs, double *px, double *py) {
    int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= bs->x.nv) return;
    int k = bs->x.svidx[v];
    double2 q = bs->x.vpos[v];
    if (px) px[k] = q.x;
    if (py) py[k] = q.y;
}

__global__ void kb_get_vnbrs(BumpySys *bs, int *list, int *counts, int cap_out) {
    int v = blockIdx.x * blockDim.x + threadIdx.x;
    const int nv = bs->x.nv;
    if (v >= nv) return;
    const int *svidx = bs->x.svidx;
    int k = svidx[v];
    int cnt = bs->x.vcount[v];
    counts[k] = cnt;
    int lim = min(cnt, min(cap_out, bs->x.capv));
    for (int t = 0; t < cap_out; t++)
        list[(size_t)k * cap_out + t] = t < lim ? svidx[bs->x.vnbr[(size_t)t * nv + v]] : -1;
}

// scalePositionsFull: kernelScalePositions (kernels.cu:1308-1333), warp per body
__global__ void kb_scale(BumpySys *bs, double f) {
    const int lane = threadIdx.x & 31;
    const int b = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    if (b >= bs->b.p.n) return;
    double2 p = bs->b.v.pos[b];
    double nx = p.x * f, ny = p.y * f;
    __syncwarp();
    if (lane == 0) bs->b.v.pos[b] = make_double2(nx, ny);
    int s0 = bs->x.start[b], n = bs->x.nvb[b];
    for (int k = lane; k < n; k += 32) {
        double2 q = bs->x.vpos[s0 + k];
        q.x += (nx - p.x);
        q.y += (ny - p.y);
        bs->x.vpos[s0 + k] = q;
    }
}

// ---- kernelCalculateRigidDampedForces (kernels.cu:80-87) ---------------------
__global__ void kb_damp(BumpySys *bs, double g) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= bs->b.p.n) return;
    double2 f = bs->b.v.frc[b], u = bs->b.v.vel[b];
    f.x -= g * u.x;
    f.y -= g * u.y;
    bs->b.v.frc[b] = f;
    bs->x.tq[b] -= g * bs->x.w[b];
}

// ---- calculateWallForces_onlyWallContacts (rigid_bumpy.cu:1495-1499): the wall
// terms of every vertex (kernelCalcRigidBumpyWallForces, kernels.cu:348-362)
// summed per body in vertex order (kernelCalcRigidBumpyParticleForces1), += into
// the body arrays; one warp per body
__global__ void kb_wall_only(BumpySys *bs) {
    const int lane = threadIdx.x & 31;
    const int b = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    if (b >= bs->b.p.n) return;
    const DevSys &d = bs->b;
    const BumpyExt &x = bs->x;
    const double2 c = d.v.pos[b];
    const int f = x.start[b], nvb = x.nvb[b];
    double bfx = 0.0, bfy = 0.0, btq = 0.0, bpe = 0.0;
    for (int base = 0; base < nvb; base += 32) {
        int k = base + lane;
        double vfx = 0.0, vfy = 0.0, vtq = 0.0, vpe = 0.0;
        if (k < nvb) {
            const double2 q = x.vpos[f + k];
            double wx, wy;
            const double we = wall_force(d.p, q, x.rv, wx, wy);
            vfx = 0.0 + wx;
            vfy = 0.0 + wy;
            vtq = 0.0 + torque_of(wx, wy, q.x, q.y, c.x, c.y);
            vpe = 0.0 + we;
        }
        int lim = min(32, nvb - base);
        for (int l = 0; l < lim; l++) {
            bfx += __shfl_sync(0xffffffffu, vfx, l);
            bfy += __shfl_sync(0xffffffffu, vfy, l);
            btq += __shfl_sync(0xffffffffu, vtq, l);
            bpe += __shfl_sync(0xffffffffu, vpe, l);
        }
    }
    if (lane == 0) {
        double2 g = bs->b.v.frc[b];
        g.x += bfx;
        g.y += bfy;
        bs->b.v.frc[b] = g;
        bs->x.tq[b] += btq;
        bs->b.w.pe[b] += bpe;
    }
}

// ---- RigidBumpy::updatePositionsAdam: kernelRigidBumpyAdamStep then
// kernelTranslateAndRotateVertices1 (rigid_bumpy.cu:1473-1486, kernels.cu:1004-1093,
// 152-201), one warp per body.  The translational moments live in DevView (m1,
// m2: swapped with their twins on a re-sort, never gathered), the angular ones
// stay with the slot.  With rotation off the angle is left alone and the
// vertices turn by the slot's last angle increment, as the reference's stale
// angle_delta does (0 after any kick, which zeroes omega without rotation).
__global__ void kb_adam(BumpySys *bs, double alpha, double b1, double b2, double c1, double c2,
                        double eps) {
    const int lane = threadIdx.x & 31;
    const int b = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    double v[2] = {0.0, 0.0};
    if (b < bs->b.p.n) {
        DevSys &d = bs->b;
        BumpyExt &x = bs->x;
        const double2 f = d.v.frc[b], p = d.v.pos[b];
        double2 m1 = d.v.m1[b], m2 = d.v.m2[b];
        const double t = x.tq[b], ang = x.th[b], adel = x.adelta[b];
        double m1a = x.m1a[b], m2a = x.m2a[b];
        m1.x = fma(b1, m1.x, (b1 - 1) * f.x);
        m1.y = fma(b1, m1.y, (b1 - 1) * f.y);
        m1a = fma(b1, m1a, (b1 - 1) * t);
        m2.x = fma(b2, m2.x, (1 - b2) * f.x * f.x);
        m2.y = fma(b2, m2.y, (1 - b2) * f.y * f.y);
        m2a = fma(b2, m2a, (1 - b2) * t * t);
        const double ux = -alpha * (m1.x / c1) / (sqrt(m2.x / c2) + eps);
        const double uy = -alpha * (m1.y / c1) / (sqrt(m2.y / c2) + eps);
        const double ua = -alpha * (m1a / c1) / (sqrt(m2a / c2) + eps);
        const double nx = p.x + ux, ny = p.y + uy;
        const double dth = x.rotation ? ua : adel;
        __syncwarp();
        if (lane == 0) {
            d.v.pos[b] = make_double2(nx, ny);
            if (x.rotation) {
                x.th[b] = ang + ua;
                x.adelta[b] = ua;
            }
            d.v.m1[b] = m1;
            d.v.m2[b] = m2;
            x.m1a[b] = m1a;
            x.m2a[b] = m2a;
            const double2 a = d.w.pos_n[b], c = d.w.pos_c[b];
            const double a1 = nx - a.x, a2 = ny - a.y, e1 = nx - c.x, e2 = ny - c.y;
            v[0] = a1 * a1 + a2 * a2;
            v[1] = e1 * e1 + e2 * e2;
        }
        const double ca = cos(dth), sa = sin(dth);
        const int f0 = x.start[b], nvb = x.nvb[b];
        for (int k = lane; k < nvb; k += 32) {
            const double2 q = x.vpos[f0 + k];
            const double rx = q.x - p.x, ry = q.y - p.y;
            const double rxr = rx * ca - ry * sa, ryr = rx * sa + ry * ca;
            const double2 nq = make_double2(nx + rxr, ny + ryr);
            x.vpos[f0 + k] = nq;
            if (x.mixed) x.vpk[f0 + k] = mixed_pack(d.p, nq, x.rv);
        }
    }
    const int ops[2] = {1, 1};
    if (grid_reduce<2>(v, ops, &bs->b)) { bs->b.s.max_nd2 = v[0]; bs->b.s.max_cd2 = v[1]; }
}

// ---- rigid gradient descent (no reference kernel: the reference's GradDesc on
// rigid bodies runs the disk kernelGradDescStep, src/particles/base/kernels.cu:
// 613-637, on the body centres only).  x += alpha F as that kernel, theta +=
// alpha tau with rotation, vertices translated and rotated with the body as in
// kernelTranslateAndRotateVertices1; one warp per body.
__global__ void kb_grad_desc(BumpySys *bs, double alpha) {
    const int lane = threadIdx.x & 31;
    const int b = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    double v[2] = {0.0, 0.0};
    if (b < bs->b.p.n) {
        DevSys &d = bs->b;
        BumpyExt &x = bs->x;
        const double2 f = d.v.frc[b], p = d.v.pos[b];
        const double ang = x.th[b];
        const double nx = p.x + alpha * f.x, ny = p.y + alpha * f.y;
        const double dth = x.rotation ? alpha * x.tq[b] : 0.0;
        __syncwarp();
        if (lane == 0) {
            d.v.pos[b] = make_double2(nx, ny);
            if (x.rotation) x.th[b] = ang + dth;
            const double2 a = d.w.pos_n[b], c = d.w.pos_c[b];
            const double a1 = nx - a.x, a2 = ny - a.y, e1 = nx - c.x, e2 = ny - c.y;
            v[0] = a1 * a1 + a2 * a2;
            v[1] = e1 * e1 + e2 * e2;
        }
        const double ca = cos(dth), sa = sin(dth);
        const int f0 = x.start[b], nvb = x.nvb[b];
        for (int k = lane; k < nvb; k += 32) {
            const double2 q = x.vpos[f0 + k];
            const double rx = q.x - p.x, ry = q.y - p.y;
            const double2 nq = make_double2(nx + (rx * ca - ry * sa), ny + (rx * sa + ry * ca));
            x.vpos[f0 + k] = nq;
            if (x.mixed) x.vpk[f0 + k] = mixed_pack(d.p, nq, x.rv);
        }
    }
    const int ops[2] = {1, 1};
    if (grid_reduce<2>(v, ops, &bs->b)) { bs->b.s.max_nd2 = v[0]; bs->b.s.max_cd2 = v[1]; }
}

// ---- kernelCalcRigidBumpyStressTensor (kernels.cu:705-789): one thread per
// body in the reference's accumulation order (per vertex: the kinetic term with
// omega x r through atan2 / sin / cos when omega != 0, then half the virial of
// each listed vertex of another body), divided by the box area.  Per-body
// values go to stress_b, the component sums to DevState.stress.
__global__ void kb_stress(BumpySys *bs) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    const DevSys &d = bs->b;
    const BumpyExt &x = bs->x;
    const int nb = d.p.n;
    if (b < nb) {
        const int nv = x.nv, capv = x.capv;
        const double bx = d.p.box[0], by = d.p.box[1], e_c = d.p.e_c, n_c = d.p.n_c, rv = x.rv;
        const double2 c = d.v.pos[b], u = d.v.vel[b];
        const double w = x.w[b];
        double axx = 0.0, axy = 0.0, ayx = 0.0, ayy = 0.0;
        const int f0 = x.start[b], nvb = x.nvb[b];
        for (int k = 0; k < nvb; k++) {
            const int vv = f0 + k;
            const double2 q = x.vpos[vv];
            const double mv = x.vmass[vv];
            const double rx = q.x - c.x, ry = q.y - c.y;
            const double prad = sqrt(rx * rx + ry * ry);
            double wx = u.x, wy = u.y;
            if (w != 0.0) {
                const double a = atan2(ry, rx);
                wx -= sin(a) * w * prad;
                wy += cos(a) * w * prad;
            }
            axx += mv * wx * wx;
            axy += mv * wx * wy;
            ayx += mv * wy * wx;
            ayy += mv * wy * wy;
            const int cnt = min(x.vcount[vv], capv);
            for (int t = 0; t < cnt; t++) {
                const int o = x.vnbr[(size_t)t * nv + vv];
                if (o == vv || x.vbody[o] == b) continue;
                const double2 op = x.vpos[o];
                const double dx = pbc_dist(q.x, op.x, bx), dy = pbc_dist(q.y, op.y, by);
                double fx, fy;
                disk_pair(q.x, q.y, rv, op.x, op.y, rv, bx, by, e_c, n_c, fx, fy);
                axx += dx * fx / 2;
                axy += dx * fy / 2;
                ayx += dy * fx / 2;
                ayy += dy * fy / 2;
            }
        }
        const double area = bx * by;
        v[0] = axx / area;
        v[1] = axy / area;
        v[2] = ayx / area;
        v[3] = ayy / area;
        for (int k = 0; k < 4; k++) x.stress_b[(size_t)k * nb + b] = v[k];
    }
    const int ops[4] = {0, 0, 0, 0};
    if (grid_reduce<4>(v, ops, &bs->b))
        for (int k = 0; k < 4; k++) bs->b.s.stress[k] = v[k];
}

// ---- kernelCountRigidBumpyContacts (kernels.cu:924-997): per body, the
// neighbour bodies with at least one overlapping vertex pair, and per such
// neighbour the overlapping partners of the first vertex (in body vertex
// order) that has one.  Totals (getContactCount and the vertex count) go to
// DevState.contacts and BumpyExt.vcontacts.
__global__ void kb_contacts(BumpySys *bs) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    double v[2] = {0.0, 0.0};
    const DevSys &d = bs->b;
    const BumpyExt &x = bs->x;
    const int nb = d.p.n;
    if (b < nb) {
        const int nv = x.nv, capv = x.capv;
        const double bx = d.p.box[0], by = d.p.box[1], rs = 2 * x.rv;
        const int nn = min(d.w.count[b], d.p.cap), f0 = x.start[b], nvb = x.nvb[b];
        int nc = 0, nvc = 0;
        for (int k = 0; k < nn; k++) {
            const int ob = d.v.nbr[(size_t)k * nb + b];
            if (ob == b) continue;
            bool contact = false;
            for (int i = 0; i < nvb; i++) {
                const int vv = f0 + i;
                const double2 q = x.vpos[vv];
                const int cnt = min(x.vcount[vv], capv);
                for (int t = 0; t < cnt; t++) {
                    const int o = x.vnbr[(size_t)t * nv + vv];
                    if (o == vv || x.vbody[o] != ob) continue;
                    const double2 op = x.vpos[o];
                    const double dx = pbc_dist(q.x, op.x, bx), dy = pbc_dist(q.y, op.y, by);
                    if (sqrt(dx * dx + dy * dy) < rs) {
                        if (!contact) nc++;
                        nvc++;
                        contact = true;
                    }
                }
                if (contact) break;
            }
        }
        x.ccount[b] = nc;
        x.vccount[b] = nvc;
        v[0] = (double)nc;
        v[1] = (double)nvc;
    }
    const int ops[2] = {0, 0};
    if (grid_reduce<2>(v, ops, &bs->b)) {
        bs->b.s.contacts = v[0];
        bs->x.vcontacts = v[1];
    }
}

// ---- RigidBumpy::calculateForceDistancePairs (rigid_bumpy.cu:1383-1459) with
// kernelCalcRigidBumpyForceDistancePairs (kernels.cu:482-703): one thread per
// body in the reference's order; entry [slot * cap + k] for the k-th listed
// neighbour body.  Array order: see dpg_bumpy_pair_dump in include/dpg.h.
constexpr int kBumpyPairArrays = 30;
constexpr double kPi = 3.14159265358979323846;

struct BumpyPairOut {
    double *d[kBumpyPairArrays];
    long long *this_id, *other_id, *vcount;
};

__global__ void kb_pair_fill(BumpyPairOut o, long long m) {
    long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= m) return;
    // the resizeAndFill values of calculateForceDistancePairs
#pragma unroll
    for (int k = 0; k < kBumpyPairArrays; k++) {
        const double f = (k == 0 || (k >= 3 && k <= 10)) ? -1.0 : 0.0;
        if (o.d[k]) o.d[k][q] = f;
    }
    o.this_id[q] = -1;
    o.other_id[q] = -1;
    o.vcount[q] = -1;
}

__global__ void kb_pair_dump(BumpySys *bs, BumpyPairOut o) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    const DevSys &d = bs->b;
    const BumpyExt &x = bs->x;
    const int nb = d.p.n, cap = d.p.cap;
    if (b >= nb) return;
    const int nn = min(d.w.count[b], cap);
    if (nn == 0) return;
    const int nv = x.nv, capv = x.capv;
    const double bx = d.p.box[0], by = d.p.box[1], e_c = d.p.e_c, n_c = d.p.n_c, rv = x.rv;
    const double rs = rv * 2.0;
    const double2 c = d.v.pos[b];
    const double thi = x.th[b], rad = d.v.rad[b];
    const int f0 = x.start[b], nvb = x.nvb[b];
    for (int k = 0; k < nn; k++) {
        const int ob = d.v.nbr[(size_t)k * nb + b];
        if (ob == b) continue;
        const double2 oc = d.v.pos[ob];
        const double thj = x.th[ob], orad = d.v.rad[ob];
        const int of = x.start[ob], onvb = x.nvb[ob];
        double fx = 0.0, fy = 0.0, en = 0.0, vov = 0.0;
        long long vci = 0;
        double hij[9], hii[9];
#pragma unroll
        for (int e = 0; e < 9; e++) { hij[e] = 0.0; hii[e] = 0.0; }
        for (int u = 0; u < nvb; u++) {
            const int v = f0 + u;
            const double2 q = x.vpos[v];
            const double phu = (double)(u * 2) * kPi / (double)nvb;
            const double rdx = q.x - c.x, rdy = q.y - c.y;
            const double Ri = sqrt(rdx * rdx + rdy * rdy);
            bool contact = false;
            const int cnt = min(x.vcount[v], capv);
            for (int t = 0; t < cnt; t++) {
                const int w = x.vnbr[(size_t)t * nv + v];
                if (w == v || x.vbody[w] != ob) continue;
                const double2 wp = x.vpos[w];
                const int iv = w - of;
                const double phv = (double)(iv * 2) * kPi / (double)onvb;
                const double odx = wp.x - oc.x, ody = wp.y - oc.y;
                const double Rj = sqrt(odx * odx + ody * ody);
                double tfx, tfy;
                const double te = disk_pair(q.x, q.y, rv, wp.x, wp.y, rv, bx, by, e_c, n_c, tfx, tfy);
                en += te;
                fx += tfx;
                fy += tfy;
                if (te > 0.0) {
                    contact = true;
                    const double dx = pbc_dist(q.x, wp.x, bx), dy = pbc_dist(q.y, wp.y, by);
                    vov += rs - sqrt(dx * dx + dy * dy);
                    const double dist = sqrt(dx * dx + dy * dy);
                    const double tij = -e_c / rs * (1 - dist / rs);
                    const double cij = e_c / (rs * rs);
                    const double si = sin(thi + phu), ci = cos(thi + phu);
                    const double sj = sin(thj + phv), cj = cos(thj + phv);
                    for (int a = 0; a < 3; a++) {
                        for (int cc = 0; cc < 3; cc++) {
                            const double dia_x = (double)(a == 0) - Ri * si * (double)(a == 2);
                            const double dia_y = (double)(a == 1) + Ri * ci * (double)(a == 2);
                            const double djb_x = -1.0 * ((double)(cc == 0) - Rj * sj * (double)(cc == 2));
                            const double djb_y = -1.0 * ((double)(cc == 1) + Rj * cj * (double)(cc == 2));
                            const double qia = dx * dia_x + dy * dia_y;
                            const double qjb = dx * djb_x + dy * djb_y;
                            const double dqjb = (dia_x * djb_x + dia_y * djb_y) / dist;
                            hij[a * 3 + cc] += cij * qia * qjb / (dist * dist) +
                                               tij * (dqjb - qia * qjb / (dist * dist * dist));
                            const double dib_x = (double)(cc == 0) - Ri * si * (double)(cc == 2);
                            const double dib_y = (double)(cc == 1) + Ri * ci * (double)(cc == 2);
                            const double d2x = -Ri * ci * (double)(a == 2) * (double)(cc == 2);
                            const double d2y = -Ri * si * (double)(a == 2) * (double)(cc == 2);
                            const double qib = dx * dib_x + dy * dib_y;
                            const double dqib = (dia_x * dib_x + dx * d2x + dia_y * dib_y + dy * d2y) / dist;
                            hii[a * 3 + cc] += cij * qia * qib / (dist * dist) +
                                               tij * (dqib - qia * qib / (dist * dist * dist));
                        }
                    }
                }
            }
            if (contact) vci++;
        }
        const long long qi = (long long)b * cap + k;
        const double xd = pbc_dist(c.x, oc.x, bx), yd = pbc_dist(c.y, oc.y, by);
        const double dist = sqrt(xd * xd + yd * yd);
        double fric = 0.0;
        if (fx != 0.0 || fy != 0.0) {
            const double nfx = fx * xd / dist, nfy = fy * yd / dist;
            const double nf = sqrt(nfx * nfx + nfy * nfy);
            const double tfx = fx - nfx, tfy = fy - nfy;
            fric = sqrt(tfx * tfx + tfy * tfy) / nf;
        }
        const double vals[12] = {en, fx, fy, xd, yd, dist - (rad + orad), rad + orad,
                                 atan2(yd, xd), thi, thj, fric, vov};
#pragma unroll
        for (int e = 0; e < 12; e++)
            if (o.d[e]) o.d[e][qi] = vals[e];
#pragma unroll
        for (int e = 0; e < 9; e++) {
            if (o.d[12 + e]) o.d[12 + e][qi] += hij[e];
            if (o.d[21 + e]) o.d[21 + e][qi] += hii[e];
        }
        o.this_id[qi] = d.v.sidx[b];
        o.other_id[qi] = d.v.sidx[ob];
        o.vcount[qi] = vci;
    }
}

// per-body stress components [4][nb] and contact counts in static order
__global__ void kb_get_stress_contacts(BumpySys *bs, double *stress, int *cc, int *vcc) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    const int nb = bs->b.p.n;
    if (b >= nb) return;
    const int k = bs->b.v.sidx[b];
    if (stress)
        for (int c = 0; c < 4; c++) stress[(size_t)c * nb + k] = bs->x.stress_b[(size_t)c * nb + b];
    if (cc) cc[k] = bs->x.ccount[b];
    if (vcc) vcc[k] = bs->x.vccount[b];
}

// ---- RigidBumpy::setLastState (dir 0) / revertToLastStateVariables (dir 1)
// (rigid_bumpy.cu:1144-1179 over particle.cu:956-985): slot-by-slot copies of
// the body and vertex arrays the reference keeps; moments of inertia, vertex
// masses, Adam moments and cell arrays are not part of the snapshot.
__global__ void kb_snapshot(BumpySys *bs, int dir) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    DevView &v = bs->b.v;
    DevScratch &w = bs->b.w;
    BumpyExt &x = bs->x;
    if (i < bs->b.p.n) {
        if (dir == 0) {
            w.s_pos[i] = v.pos[i]; w.s_vel[i] = v.vel[i]; w.s_frc[i] = v.frc[i];
            w.s_rad[i] = v.rad[i]; w.s_mass[i] = v.mass[i]; w.s_sidx[i] = v.sidx[i];
            x.s_w[i] = x.w[i]; x.s_th[i] = x.th[i]; x.s_tq[i] = x.tq[i];
            x.s_nvb[i] = x.nvb[i]; x.s_start[i] = x.start[i];
        } else {
            v.pos[i] = w.s_pos[i]; v.vel[i] = w.s_vel[i]; v.frc[i] = w.s_frc[i];
            v.rad[i] = w.s_rad[i]; v.mass[i] = w.s_mass[i]; v.sidx[i] = w.s_sidx[i];
            x.w[i] = x.s_w[i]; x.th[i] = x.s_th[i]; x.tq[i] = x.s_tq[i];
            x.nvb[i] = x.s_nvb[i]; x.start[i] = x.s_start[i];
        }
    }
    if (i < x.nv) {
        if (dir == 0) {
            x.s_vpos[i] = x.vpos[i]; x.s_vbody[i] = x.vbody[i]; x.s_svidx[i] = x.svidx[i];
        } else {
            x.vpos[i] = x.s_vpos[i]; x.vbody[i] = x.s_vbody[i]; x.svidx[i] = x.s_svidx[i];
        }
    }
}

}  // namespace
}  // namespace dpg
