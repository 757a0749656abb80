// bumpy_loop.cuh -- the NVE and FIRE loops of rigid bumpy bodies as one
// resident cooperative grid (see disk_loop.cuh: barriers, decisions and the
// write-back are the same).  Block b owns the bodies [b * chunk, (b + 1) *
// chunk) and their vertices, which are contiguous.  An NVE step costs one
// barrier: the moved vertices go into the other of two buffers; a FIRE
// iteration costs two.
#pragma once
#include "bumpy_kernels.cuh"
#include "disk_loop.cuh"

namespace dpg {
namespace {

constexpr int kLoopBodies = 64;  // bodies per block at most
constexpr int kVlistParts = 4;   // warps that share a body in the list build at most

// The rebuild inside the loop: the kernels k_cell_index .. kb_vlist as phases
// between barriers.  Returns false if the loop has to leave.
__device__ __forceinline__ bool bumpy_rebuild(BumpySys *bs, LoopSync *ls, unsigned &bk, int kind, Range r) {
    DevSys &d = bs->b;
    BumpyExt &x = bs->x;
    const DevParams &p = d.p;
    DevView &v = d.v;
    DevState &s = d.s;
    const int t = threadIdx.x, nt = blockDim.x;
    auto vertices = [&](int &v0, int &v1) {
        v0 = r.first < r.last ? x.start[r.first] : 0;
        v1 = r.first < r.last ? x.start[r.last - 1] + x.nvb[r.last - 1] : 0;
    };
    int v0, v1;
    if (kind == 2) {
        for (int i = r.first + t; i < r.last; i += nt) {
            const double2 c = v.pos[i];
            const int cell = cell_coord(c.x, p.cell_size, p.ncd) + cell_coord(c.y, p.cell_size, p.ncd) * p.ncd;
            d.w.cell_raw[i] = cell;
            atomicAdd(&d.w.cell_cnt[cell], 1);
        }
        if (!grid_bar(ls, bk, 0)) return false;
        if (blockIdx.x == 0) cell_scan_block(d.w.cell_cnt, d.w.cell_start, p.ncells);
        if (!grid_bar(ls, bk, 0)) return false;
        for (int i = r.first + t; i < r.last; i += nt) {
            const int c = d.w.cell_raw[i];
            d.w.perm[d.w.cell_start[c] + atomicAdd(&d.w.cell_cur[c], 1)] = i;
        }
        if (!grid_bar(ls, bk, 0)) return false;
        for (int c = blockIdx.x * nt + t; c < p.ncells; c += gridDim.x * nt) cell_sort_one(&d, c);
        if (!grid_bar(ls, bk, 0)) return false;
        for (int i = r.first + t; i < r.last; i += nt) reorder_body(bs, i);
        if (!grid_bar(ls, bk, 0)) return false;
        if (blockIdx.x == 0) cell_scan_block(x.nvb_t, x.start_t, p.n);
        if (!grid_bar(ls, bk, 0)) return false;
        for (int i = r.first + t / 32; i < r.last; i += nt / 32) reorder_vertices(bs, i, t & 31);
        if (!grid_bar(ls, bk, 0)) return false;
        if (t == 0) {
            swap_sorted(bs);
            s.n_cell_rebuilds++;
        }
        __syncthreads();
        vertices(v0, v1);
        for (int u = v0 + t; u < v1; u += nt) x.vq[u] = quant_of(p, x.vpos[u], x.rv);
    } else {
        for (int i = r.first + t; i < r.last; i += nt) v.q[i] = quant_of(p, v.pos[i], v.rad[i]);
        vertices(v0, v1);
        if (x.mixed)
            for (int u = v0 + t; u < v1; u += nt) x.vq[u] = quant_of(p, x.vpos[u], x.rv);
    }
    if (!grid_bar(ls, bk, 0)) return false;
    __shared__ int bmx[2];
    if (t < 2) bmx[t] = 0;
    __syncthreads();
    int mx = 0;
    for (int b = r.first; b < r.last; b += nt / 8) {
        const int i = b + t / 8;
        const bool valid = i < r.last;
        int cnt = 0;
        if (p.method == 0) cnt = nlist_row<8>(&d, i, valid);
        else if (valid && (t & 7) == 0) cnt = nlist_all_row(&d, i);
        if (valid && (t & 7) == 0) {
            mx = max(mx, cnt);
            d.w.count[i] = cnt;
            d.w.pos_n[i] = v.pos[i];
        }
    }
    if (mx) atomicMax(&bmx[0], mx);
    __syncthreads();  // the rows of the block's bodies, which its vertices read
    // vertex rows: a warp a body; where the block has warps to spare, `parts`
    // warps share a body's listed bodies: they count their part, then write it
    // behind the parts before theirs
    mx = 0;
    const int lane = t & 31, wid = t >> 5, nw = nt >> 5, np = r.last - r.first;
    const int parts = np > 0 ? min(nw / np > 0 ? nw / np : 1, kVlistParts) : 1, slot = wid / parts, part = wid % parts;
    __shared__ int pcnt[kLoopMaxTPB];
    for (int g0 = 0; g0 < np; g0 += nw / parts) {
        const bool on = slot < nw / parts && g0 + slot < np;  // this warp has a body
        const int b = r.first + (on ? g0 + slot : 0);
        const int f = x.start[b], nvb = x.nvb[b], rows = min(d.w.count[b], p.cap);
        const int t0 = rows * part / parts, t1 = on ? rows * (part + 1) / parts : t0;
        for (int base = 0; base < x.max_nvb; base += 32) {
            const bool real = on && base + lane < nvb;
            const int u = f + (real ? base + lane : 0);
            const uint4 qv = x.vq[u];
            const float reach = vlist_reach(bs, v.q[b], qv, real);
            int cnt = 0;
            if (parts > 1) {
                vlist_scan(bs, b, u, real, qv, reach, t0, t1, false, cnt);
                pcnt[t] = cnt;
                __syncthreads();
                cnt = 0;
                for (int q = 0; q < part; q++) cnt += pcnt[(slot * parts + q) * 32 + lane];
                __syncthreads();
            }
            vlist_scan(bs, b, u, real, qv, reach, t0, t1, true, cnt);
            if (!real || part != parts - 1) continue;
            mx = max(mx, cnt);
            x.vcount[u] = cnt;
            if (x.mixed) x.vpk[u] = mixed_pack(p, x.vpos[u], x.rv);
        }
    }
    if (mx) atomicMax(&bmx[1], mx);
    __syncthreads();
    if (t < 2) atomicMax(t == 0 ? &ls->max_count : &ls->max_vcount, bmx[t]);
    const unsigned long long w = grid_bar(ls, bk, bmx[0] > p.cap || bmx[1] > x.capv ? kFull : 0);
    if (!w) return false;
    if (t == 0) {
        s.n_rebuilds++;
        s.max_count = *(volatile int *)&ls->max_count;
        x.max_vcount = *(volatile int *)&ls->max_vcount;
        x.vlist_built = s.n_rebuilds;
        if (raised(w, kFull)) s.flags |= kOverflow;
    }
    __syncthreads();
    if (raised(w, kFull)) return false;
    // cleared for the next build, which starts only after another barrier
    if (blockIdx.x == 0 && t < 2) atomicExch(t == 0 ? &ls->max_count : &ls->max_vcount, 0);
    return true;
}

// ---- the loop kernel ----------------------------------------------------------
// An FP64 instruction holds an SM quarter's pipe for ~64 clocks whatever the
// number of its lanes, so the kernel counts FP64 instructions per warp:
//  - the body part runs in four roles, 64 threads each, on different quarters:
//    role 0 / 1 the x / y components, role 2 the angle and the cosine of its
//    increment, role 3 the sine (role 2's arithmetic once more); a thread keeps
//    its component's position, velocity, force, mass (or angle, angular
//    velocity, torque, inertia) and last-build position in registers;
//  - the vertices of the block keep their positions in shared memory and turn
//    one thread each;
//  - the vertex pairs that the filter lets through form one queue per block,
//    evaluated on full warps; only the vertices that have a term compute a
//    torque and enter the body sums (in vertex order, one thread a sum).
constexpr int kBodyVerts = 2048;  // vertices per block at most
constexpr int kVertQueue = 2048;  // queued vertex pairs evaluated at a time
constexpr int kVertSlots = 32;    // vertex-list capacity at most

struct BodyMem {
    double2 vpos[kBodyVerts];           // current vertex positions
    double res[3][kVertQueue];          // terms of the queued pairs
    double term[4][kBodyVerts];         // terms of the vertices that have one
    double2 p[kLoopBodies], n[kLoopBodies], cs[kLoopBodies];  // a move: from, to, cosine and sine
    double sum[4][kLoopBodies];         // force x, force y, torque, energy
    double xa[4][kLoopBodies], xb[4][kLoopBodies];  // exchanged between the roles
    int ej[kVertQueue];                 // queue: other vertex,
    unsigned ent[kVertQueue];           //        vertex << 6 | sure << 5 | slot
    int off[kBodyVerts + 1];            // first queue entry of each term vertex
    unsigned short tv[kBodyVerts];      // its vertex
    int first[kLoopBodies + 1];         // first term vertex of each body
    int vfirst[kLoopBodies + 1];        // first vertex of each body (block-local)
    unsigned char vb[kBodyVerts];       // body of each vertex (block-local)
};

// vertex contact: disk_pair_sum with one radius sum, its square and its reciprocal
struct VertConst {
    double rs, rs2, inv;
};
__device__ __forceinline__ double vertex_pair(const PairArgs &f, const VertConst &c, bool sure, double2 a,
                                              double2 b, double &fx, double &fy) {
    const double dx = pbc_dist_sum(a.x, b.x, f.bx, f.l4x), dy = pbc_dist_sum(a.y, b.y, f.by, f.l4y);
    return contact_terms(dx, dy, c.rs, c.rs2, c.inv, sure, f.e_c, f.n_c, fx, fy);
}

// The queue in windows, for a block with more contacts than the queue holds
// (far above any packing): the entries are found again from the lists, each
// window's terms added to the term vertices in order.
__device__ __noinline__ void vertex_windows(BodyMem &m, const BumpySys &L, const PairArgs &fa,
                                            const VertConst &vc, int terms, int entries, int v0) {
    const int t = threadIdx.x, nt = blockDim.x;
    for (int q = t; q < terms; q += nt) m.term[0][q] = m.term[1][q] = m.term[3][q] = 0.0;
    for (int w0 = 0; w0 < entries; w0 += kVertQueue) {
        const int w1 = min(entries, w0 + kVertQueue);
        __syncthreads();
        for (int q = t; q < terms; q += nt) {
            if (m.off[q + 1] <= w0 || m.off[q] >= w1) continue;
            const int k = m.tv[q], vg = v0 + k, cnt = min(L.x.vcount[vg], L.x.capv);
            const uint4 qi = L.x.vq[vg];
            int at = m.off[q];
            for (int c = 0; c < cnt; c++) {
                const int j = L.x.vnbr[(size_t)c * fa.n + vg];
                if (!quant_contact(fa.sx, fa.sy, fa.tol, qi, L.x.vq[j])) continue;
                if (at >= w0 && at < w1) {
                    m.ent[at - w0] = (unsigned)k << 6 | (unsigned)c;
                    m.ej[at - w0] = j;
                }
                at++;
            }
        }
        __syncthreads();
        for (int e = t; e < w1 - w0; e += nt) {
            double fx, fy;
            const double ee = vertex_pair(fa, vc, false, m.vpos[m.ent[e] >> 6], fa.pos[m.ej[e]], fx, fy);
            m.res[0][e] = fx;
            m.res[1][e] = fy;
            m.res[2][e] = ee;
        }
        __syncthreads();
        for (int q = t; q < terms; q += nt)
            for (int e = max(m.off[q], w0); e < min(m.off[q + 1], w1); e++) {
                m.term[0][q] += m.res[0][e - w0];
                m.term[1][q] += m.res[1][e - w0];
                m.term[3][q] += m.res[2][e - w0];
            }
    }
    __syncthreads();
}

template <int KIND>
__global__ void __launch_bounds__(kLoopMaxTPB, 1) kb_loop(BumpySys *bs, LoopSync *ls, double dt, double tmax,
                                                         int chunk, long long iters) {
    extern __shared__ __align__(16) unsigned char loop_smem[];
    BodyMem &m = *reinterpret_cast<BodyMem *>(loop_smem);
    __shared__ BumpySys L;
    __shared__ double red[32 * 4];
    __shared__ int wtot[kLoopMaxTPB / 32];
    const int t = threadIdx.x, nt = blockDim.x, lane = t & 31, wid = t >> 5, nw = nt >> 5;
    if (t == 0) L = *bs;
    __syncthreads();
    DevState &s = L.b.s;
    DevView &v = L.b.v;
    BumpyExt &x = L.x;
    const DevParams &p = L.b.p;
    if (s.flags) return;  // the same for every block: nothing writes the state before a barrier
    const int n = p.n;
    const Range r = {min((int)blockIdx.x * chunk, n), min(((int)blockIdx.x + 1) * chunk, n)};
    const int np = r.last - r.first;
    const int role = t / kLoopBodies, lb = t % kLoopBodies, own = r.first + lb;
    const bool mine = role < 4 && lb < np;
    unsigned bk = 0;
    bool ok = true, stored = false;
    long long it = 0;
    const double dt_half = 0.5 * dt;
    const double rv = x.rv;
    const VertConst vc = {rv + rv, (rv + rv) * (rv + rv), 1.0 / (rv + rv)};
    int v0 = 0, nv = 0;  // the block's first vertex and their number

    double a = 0.0, u = 0.0, f = 0.0, mass = 1.0, xn = 0.0, xc = 0.0, da = 0.0, pe = 0.0;
    double kick = 0.0, kick_h = 0.0;  // (f h) / mass for h = kick_h, if known
    bool kick_known = false;
    const bool moves = x.rotation != 0;
    auto load_own = [&]() {
        if (mine) {
            if (role < 2) {
                const double2 q = v.pos[own], w = v.vel[own], g = v.frc[own], qn = L.b.w.pos_n[own],
                              qc = L.b.w.pos_c[own];
                a = role ? q.y : q.x; u = role ? w.y : w.x; f = role ? g.y : g.x;
                xn = role ? qn.y : qn.x; xc = role ? qc.y : qc.x;
                mass = v.mass[own];
                (&m.n[lb].x)[role] = a;  // the centre that the torques refer to
            } else {
                a = x.th[own]; u = x.w[own]; f = x.tq[own]; mass = x.I[own];
                da = x.adelta[own];
            }
        }
        kick_known = false;
        v0 = np > 0 ? x.start[r.first] : 0;
        nv = np > 0 ? x.start[r.last - 1] + x.nvb[r.last - 1] - v0 : 0;
        for (int k = t; k < nv; k += nt) {
            m.vpos[k] = x.vpos[v0 + k];
            m.vb[k] = (unsigned char)(x.vbody[v0 + k] - r.first);
        }
        if (t < np) m.vfirst[t] = x.start[r.first + t] - v0;
        if (t == 0) m.vfirst[np] = nv;
        __syncthreads();
    };
    auto store_own = [&]() {
        if (!mine) return;
        if (role < 2) {
            double *q = &v.pos[own].x + role, *w = &v.vel[own].x + role, *g = &v.frc[own].x + role;
            *q = a; *w = u; *g = f;
        } else if (role == 2) {
            x.th[own] = a; x.w[own] = u; x.tq[own] = f; x.adelta[own] = da;
        }
    };
    // body_kick: u += f h / mass (components and rotation alike)
    auto kick_by = [&](double h) {
        if (!kick_known || h != kick_h) {
            kick = f * h / mass;
            kick_h = h;
            kick_known = true;
        }
        if (role < 2 || moves) u += kick;
        else u = 0.0;
    };
    // the bodies' move by h and their vertices into the given buffers
    auto move_by = [&](double h, double2 *vpos, float4 *vpk, uint4 *vq) {
        if (mine) {
            const double d = u * h;
            if (role < 2) {
                const double q = a + d, dn = q - xn, dc = q - xc;
                (&m.p[lb].x)[role] = a;
                (&m.n[lb].x)[role] = q;
                m.xa[role][lb] = dn * dn;
                m.xb[role][lb] = dc * dc;
                a = q;
            } else {
                da = d;
                a = a + d;
                if (role == 2) m.cs[lb].x = cos(d);
                else m.cs[lb].y = sin(d);
            }
        }
        __syncthreads();
        for (int k = t; k < nv; k += nt) {
            const int b = m.vb[k];
            const double2 q = m.vpos[k], c = m.p[b], o = m.n[b], cs = m.cs[b];
            const double rx = q.x - c.x, ry = q.y - c.y;
            const double rxr = rx * cs.x - ry * cs.y, ryr = rx * cs.y + ry * cs.x;
            const double2 nq = make_double2(o.x + rxr, o.y + ryr);
            m.vpos[k] = nq;
            vpos[v0 + k] = nq;
            if (x.mixed) vpk[v0 + k] = mixed_pack(p, nq, rv);
            if (!x.mixed || s.fp64_now) vq[v0 + k] = quant_of(p, nq, rv);
        }
    };
    // the barrier after a move and a rebuild if any body asks for one
    auto after_move = [&]() {
        unsigned long long fl = 0;
        if (t < np) fl = move_flags(p, m.xa[0][t] + m.xa[1][t], m.xb[0][t] + m.xb[1][t]);
        const unsigned long long bw = grid_bar(ls, bk, block_flags(fl));
        if (!bw) return false;
        if (KIND == 1) {
            if (t == 0) {
                swap_ptr(x.vpos, x.vpos_t);
                if (x.mixed) swap_ptr(x.vpk, x.vpk_t);
                else swap_ptr(x.vq, x.vq_t);
            }
            __syncthreads();
        }
        const int kind = rebuild_kind(bw);
        if (!kind) return true;
        store_own();
        stored = true;
        __syncthreads();
        if (!bumpy_rebuild(&L, ls, bk, kind, r)) return false;
        load_own();
        stored = false;
        return true;
    };
    auto nve_first = [&]() {
        if (mine) kick_by(dt_half);
        move_by(dt, x.vpos_t, x.vpk_t, x.vq_t);
        return after_move();
    };

    load_own();
    if (KIND == 1) ok = nve_first();
    while (ok) {
        if (KIND == 0) {
            // ---- move (src/integrator/fire.cu:29-40 with the rigid overrides)
            const double fdt = s.f_dt, alpha = s.f_alpha;
            if (s.fire_uphill) {
                move_by(-fdt / 2.0, x.vpos, x.vpk, x.vq);
                u = 0.0;
                __syncthreads();
            }
            if (mine) kick_by(fdt / 2.0);
            // body_mix: |F| and |v| on two roles, the torque's part on its own
            if (mine && role < 2) {
                m.xa[role][lb] = f * f;
                m.xb[role][lb] = u * u;
            }
            __syncthreads();
            if (mine && role == 0) m.sum[0][lb] = sqrt(m.xa[0][lb] + m.xa[1][lb]);
            if (mine && role == 1) m.sum[1][lb] = sqrt(m.xb[0][lb] + m.xb[1][lb]);
            __syncthreads();
            if (mine) {
                const double fn = role < 2 ? m.sum[0][lb] : fabs(f), un = role < 2 ? m.sum[1][lb] : fabs(u);
                double mix = 0.0;
                if (fn > 1e-16) mix = un / fn * alpha;
                else u = 0.0;
                u = u * (1 - alpha) + f * mix;
            }
            move_by(fdt, x.vpos, x.vpk, x.vq);
            ok = after_move();
            if (!ok) break;
        }
        // ---- vertex forces
        const bool walls = KIND == 1 && s.walls != 0;
        const bool fp32 = x.mixed && !s.fp64_now;
        const PairArgs fa = vertex_args(&L);
        int entries = 0, terms = 0;  // queue entries and term vertices before this tile
        for (int k0 = 0; k0 < nv; k0 += nt) {
            const int k = k0 + t, vg = v0 + k;
            const bool real = k < nv;
            const int cnt = real ? min(x.vcount[vg], x.capv) : 0;
            unsigned bits = 0, sure = 0;
            double ax = 0.0, ay = 0.0, en = 0.0;
            if (fp32) {
                if (real) {
                    const float4 pa = x.vpk[vg];
                    const float e_c = (float)p.e_c, n_c = (float)p.n_c;
                    float sx = 0.f, sy = 0.f, se = 0.f;
                    for (int q = 0; q < cnt; q++) {
                        float fx, fy;
                        se += mixed_pair(p, pa, x.vpk[x.vnbr[(size_t)q * fa.n + vg]], e_c, n_c, fx, fy);
                        sx += fx;
                        sy += fy;
                    }
                    ax = (double)sx;
                    ay = (double)sy;
                    en = (double)se;
                }
            } else {
                const uint4 qi = x.vq[real ? vg : v0];
                for (int q0 = 0; q0 < cnt; q0 += 4) {
                    int j[4];
                    uint4 qj[4];
#pragma unroll
                    for (int c = 0; c < 4; c++) j[c] = q0 + c < cnt ? x.vnbr[(size_t)(q0 + c) * fa.n + vg] : vg;
#pragma unroll
                    for (int c = 0; c < 4; c++) qj[c] = x.vq[j[c]];
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        if (q0 + c >= cnt) break;
                        const int hit = quant_contact(fa.sx, fa.sy, fa.tol, qi, qj[c]);
                        if (hit) {
                            bits |= 1u << (q0 + c);
                            asm volatile("prefetch.global.L1 [%0];" ::"l"(x.vpos + j[c]));
                        }
                        if (hit == 2) sure |= 1u << (q0 + c);
                    }
                }
            }
            // places in the queue and among the term vertices: one block scan of both
            const bool some = real && (walls || bits != 0 || ax != 0.0 || ay != 0.0 || en != 0.0);
            const int c = __popc(bits);
            int incl = c | (some ? 1 << 16 : 0);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            if (lane == 31) wtot[wid] = incl;
            __syncthreads();
            const int w_l = lane < nw ? wtot[lane] : 0;
            const int before = (int)__reduce_add_sync(0xffffffffu, (unsigned)(lane < wid ? w_l : 0));
            const int tile = (int)__reduce_add_sync(0xffffffffu, (unsigned)w_l);
            const int ex = incl + before - (c | (some ? 1 << 16 : 0));
            const int off = entries + (ex & 0xffff), rank = terms + (ex >> 16);
            if (real && m.vfirst[m.vb[k]] == k) m.first[m.vb[k]] = rank;
            if (some) {
                m.tv[rank] = (unsigned short)k;
                m.off[rank] = off;
                if (fp32) {
                    m.term[0][rank] = ax;
                    m.term[1][rank] = ay;
                    m.term[3][rank] = en;
                }
            }
            // entries past the queue's end are queued again window by window below
            int at = off;
            for (unsigned b = bits; b; b &= b - 1, at++) {
                const int q = __ffs(b) - 1;
                if (at >= kVertQueue) break;
                m.ent[at] = (unsigned)k << 6 | (sure >> q & 1u) << 5 | (unsigned)q;
                m.ej[at] = x.vnbr[(size_t)q * fa.n + vg];
            }
            entries += tile & 0xffff;
            terms += tile >> 16;
            __syncthreads();  // wtot is rewritten by the next tile
        }
        if (t == 0) {
            m.off[terms] = entries;
            m.first[np] = terms;
        }
        __syncthreads();
        if (entries > kVertQueue) {  // the same on every thread: too many at once
            vertex_windows(m, L, fa, vc, terms, entries, v0);
        } else if (!fp32) {
            for (int e = t; e < entries; e += nt) {
                const unsigned ent = m.ent[e];
                double fx, fy;
                const double ee = vertex_pair(fa, vc, ent >> 5 & 1u, m.vpos[ent >> 6], fa.pos[m.ej[e]], fx, fy);
                m.res[0][e] = fx;
                m.res[1][e] = fy;
                m.res[2][e] = ee;
            }
            __syncthreads();
        }
        for (int q = t; q < terms; q += nt) {
            double ax = 0.0, ay = 0.0, en = 0.0;
            if (fp32 || entries > kVertQueue) {
                ax = m.term[0][q]; ay = m.term[1][q]; en = m.term[3][q];
            } else {
                for (int e = m.off[q]; e < m.off[q + 1]; e++) {
                    ax += m.res[0][e];
                    ay += m.res[1][e];
                    en += m.res[2][e];
                }
            }
            const int k = m.tv[q], b = m.vb[k];
            const double2 c = m.n[b], pv = m.vpos[k];
            double t0 = torque_of(ax, ay, pv.x, pv.y, c.x, c.y);
            if (walls) {
                double wx, wy;
                const double we = wall_force(p, pv, rv, wx, wy);
                t0 = (0.0 + torque_of(wx, wy, pv.x, pv.y, c.x, c.y)) + t0;
                ax = (0.0 + wx) + ax;
                ay = (0.0 + wy) + ay;
                en = (0.0 + we) + en;
            }
            m.term[0][q] = ax;
            m.term[1][q] = ay;
            m.term[2][q] = t0;
            m.term[3][q] = en;
        }
        __syncthreads();
        if (mine) {
            double acc = 0.0;
            for (int q = m.first[lb]; q < m.first[lb + 1]; q++) acc += m.term[role][q];
            m.sum[role][lb] = acc;
        }
        __syncthreads();
        // ---- new forces and the kick
        it++;
        if (mine) {
            f = m.sum[role == 3 ? 2 : role][lb];
            pe = m.sum[3][lb];
            kick_known = false;
        }
        if (KIND == 1) {
            if (mine) {
                if (s.damping != 0.0) f = (0.0 - s.damping * u) + f;  // (see body_nve_second)
                kick_by(dt_half);
            }
            const bool last = it >= iters || s.nve_steps_done + 1 >= s.max_steps;
            __syncthreads();  // every thread has read the state
            if (t == 0 && ++s.nve_steps_done >= s.max_steps) s.flags |= kDone;
            __syncthreads();
            if (last) break;
            ok = nve_first();
        } else {
            if (mine) {
                kick_by(s.f_dt / 2.0);
                m.xa[role][lb] = f * u;
                m.xb[role][lb] = f * f;
            }
            __syncthreads();
            double tot[4] = {0.0, 0.0, 0.0, 0.0};
            if (t < np) {
                tot[0] = pe;
                tot[1] = m.xa[0][t] + m.xa[1][t] + m.xa[2][t];
                tot[2] = m.xb[0][t] + m.xb[1][t];
                tot[3] = m.xb[2][t];
            }
            ok = grid_totals<4>(tot, (np + 31) / 32, L.b.w.partials, ls, bk, red);
            if (!ok) break;
            if (t == 0) bumpy_fire_epilogue(&L, tot, tmax);
            __syncthreads();
            if (s.flags || it >= iters) break;
        }
    }
    if (!stored) {
        store_own();
        if (mine && role == 3) L.b.w.pe[own] = pe;
    }
    __syncthreads();
    if (loop_exit(&L.b, ls, bk, r, red)) *bs = L;
}

}  // namespace
}  // namespace dpg
