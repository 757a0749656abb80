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
__device__ __forceinline__ bool bumpy_rebuild(BumpySys *bs, LoopSync *ls, unsigned &bk, int polls, int kind, Range r) {
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
        if (!grid_bar(ls, bk, polls, 0)) return false;
        if (blockIdx.x == 0) {
            const int all = scan_block(d.w.cell_cnt, d.w.cell_start, p.ncells);
            if (t == 0) d.w.cell_start[p.ncells] = all;
        }
        if (!grid_bar(ls, bk, polls, 0)) return false;
        for (int i = r.first + t; i < r.last; i += nt) {
            const int c = d.w.cell_raw[i];
            d.w.perm[d.w.cell_start[c] + atomicAdd(&d.w.cell_cur[c], 1)] = i;
        }
        if (!grid_bar(ls, bk, polls, 0)) return false;
        for (int c = blockIdx.x * nt + t; c < p.ncells; c += gridDim.x * nt) cell_sort_one(&d, c);
        if (!grid_bar(ls, bk, polls, 0)) return false;
        for (int i = r.first + t; i < r.last; i += nt) reorder_body(bs, i);
        if (!grid_bar(ls, bk, polls, 0)) return false;
        if (blockIdx.x == 0) scan_block(x.nvb_t, x.start_t, p.n);  // starts only: the array has no n + 1st
        if (!grid_bar(ls, bk, polls, 0)) return false;
        for (int i = r.first + t / 32; i < r.last; i += nt / 32) reorder_vertices(bs, i, t & 31);
        if (!grid_bar(ls, bk, polls, 0)) return false;
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
    if (!grid_bar(ls, bk, polls, 0)) return false;
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
    const unsigned long long w = grid_bar(ls, bk, polls, bmx[0] > p.cap || bmx[1] > x.capv ? kFull : 0);
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
constexpr int kBodyVerts = 1536;      // vertices per block at most
constexpr int kBodyVertsSmall = 256;  // ... of a block of 256 threads, two of which share an SM,
                                      // so that two small systems run side by side: 301 bodies
                                      // on two streams, 2000 steps each, 67.3 -> 35.7 ms
constexpr int kVertSlots = 32;        // vertex-list capacity at most

template <int V>  // vertices at most
struct BodyMem {
    static constexpr int kRows = V == kBodyVerts ? 6144 : 2048;   // list entries kept on chip (more are read from memory)
    static constexpr int kQueue = V == kBodyVerts ? 2048 : 1024;  // queued vertex pairs evaluated at a time
    double2 vpos[V];                    // current vertex positions
    double res[3][kQueue];              // terms of the queued pairs
    double term[4][V];                  // terms of the vertices that have one
    double2 p[kLoopBodies], n[kLoopBodies], cs[kLoopBodies];  // a move: from, to, cosine and sine
    double sum[4][kLoopBodies];         // force x, force y, torque, energy
    double xa[4][kLoopBodies], xb[4][kLoopBodies];  // exchanged between the roles
    // the vertex rows of the block as one list: entry e belongs to vertex k for
    // row[k] <= e < row[k + 1]
    int row[V + 1];
    int other[kRows];               // the other vertex
    unsigned short of[kRows];       // k
    // a force pass: which entries may touch (bit e), and how many before each
    // word: the queue position of entry e is rank(e)
    unsigned touch[V + 1];
    int count[V], before[V + 1];
    unsigned short ent[kQueue];     // entry at each queue position
    unsigned vmask[V / 32];    // vertices that have a term
    unsigned short tv[V];      // the term vertices
    int first[kLoopBodies + 1];         // first term vertex of each body
    int vfirst[kLoopBodies + 1];        // first vertex of each body (block-local)
    unsigned char vb[V];       // body of each vertex (block-local)
    __device__ __forceinline__ int rank(int e) const {
        return before[e >> 5] + __popc(touch[e >> 5] & ((1u << (e & 31)) - 1u));
    }
};

// vertex and other vertex of entry e: from the chip, or by a search of the rows
// and a load
template <int V>
__device__ __forceinline__ void entry_of(const BodyMem<V> &m, const BumpySys &L, int nv, int v0, int e, int &k, int &j) {
    if (m.row[nv] <= m.kRows) {
        k = m.of[e];
        j = m.other[e];
        return;
    }
    int lo = 0, hi = nv;  // row[lo] <= e < row[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (m.row[mid] <= e) lo = mid;
        else hi = mid;
    }
    k = lo;
    j = L.x.vnbr[(size_t)(e - m.row[k]) * L.x.nv + v0 + k];
}

// vertex contact: disk_pair_sum with one radius sum and its reciprocal
struct VertConst {
    double rs, inv;
};
__device__ __forceinline__ double vertex_pair(const PairArgs &f, const VertConst &c, double2 a, double2 b,
                                              double &fx, double &fy) {
    const double dx = pbc_dist_sum(a.x, b.x, f.bx, f.l4x), dy = pbc_dist_sum(a.y, b.y, f.by, f.l4y);
    return contact_terms<true>(dx, dy, c.rs, c.inv, f.e_c, f.n_c, fx, fy);
}

template <int KIND, int V>
__global__ void __launch_bounds__(kLoopMaxTPB, 1) kb_loop(BumpySys *bs, LoopSync *ls, double dt, double tmax,
                                                         int chunk, long long iters, int polls) {
    extern __shared__ __align__(16) unsigned char loop_smem[];
    BodyMem<V> &m = *reinterpret_cast<BodyMem<V> *>(loop_smem);
    constexpr int kQueue = BodyMem<V>::kQueue;
    __shared__ BumpySys L;
    __shared__ double red[32 * 4];
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
    const VertConst vc = {rv + rv, 1.0 / (rv + rv)};
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
            m.count[k] = min(x.vcount[v0 + k], x.capv);
        }
        if (t < np) m.vfirst[t] = x.start[r.first + t] - v0;
        if (t == 0) m.vfirst[np] = nv;
        __syncthreads();
        const int rows = scan_block(m.count, m.row, nv);
        if (t == 0) m.row[nv] = rows;
        __syncthreads();
        if (m.row[nv] <= m.kRows)
            for (int k = t; k < nv; k += nt)
                for (int q = 0; q < m.count[k]; q++) {
                    m.other[m.row[k] + q] = x.vnbr[(size_t)q * x.nv + v0 + k];
                    m.of[m.row[k] + q] = (unsigned short)k;
                }
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
        const unsigned long long bw = grid_bar(ls, bk, polls, block_flags(fl));
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
        if (!bumpy_rebuild(&L, ls, bk, polls, kind, r)) return false;
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
    if (KIND == 0 && s.pe_diff_target > 0) {  // as in k_tile
        double tot[4] = {t < np ? L.b.w.pe[r.first + t] : 0.0, 0.0, 0.0, 0.0};
        ok = grid_totals<4>(tot, (np + 31) / 32, L.b.w.partials, ls, bk, polls, red);
        if (ok && t == 0) s.last_avg_pe = tot[0] / s.dof;
        __syncthreads();
    }
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
        const int rows = nv > 0 ? m.row[nv] : 0, words = (rows + 31) / 32;
        const float e_cf = (float)p.e_c, n_cf = (float)p.n_c;
        // which entries touch: a word a warp, four words in flight
        for (int w0 = wid; w0 < words; w0 += 4 * nw) {
            int k[4], j[4];
            bool on[4];
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const int e = (w0 + c * nw) * 32 + lane;
                on[c] = e < rows;
                k[c] = 0;
                j[c] = v0;
                if (on[c]) entry_of(m, L, nv, v0, e, k[c], j[c]);
            }
            bool hit[4] = {false, false, false, false};
            if (fp32) {
                float4 o[4];
#pragma unroll
                for (int c = 0; c < 4; c++) o[c] = x.vpk[j[c]];
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    float fx, fy;
                    const float e = mixed_pair(p, x.vpk[v0 + k[c]], o[c], e_cf, n_cf, fx, fy);
                    hit[c] = on[c] && (e != 0.f || fx != 0.f || fy != 0.f);
                }
            } else {
                uint4 o[4];
#pragma unroll
                for (int c = 0; c < 4; c++) o[c] = x.vq[j[c]];
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    hit[c] = on[c] && quant_touch(fa.sx, fa.sy, fa.tol, x.vq[v0 + k[c]], o[c]);
                    if (hit[c]) asm volatile("prefetch.global.L1 [%0];" ::"l"(x.vpos + j[c]));
                }
            }
#pragma unroll
            for (int c = 0; c < 4; c++) {
                if (w0 + c * nw >= words) break;
                const unsigned any = __ballot_sync(0xffffffffu, hit[c]);
                if (lane == 0) {
                    m.touch[w0 + c * nw] = any;
                    m.count[w0 + c * nw] = __popc(any);
                }
            }
        }
        __syncthreads();
        const int entries = scan_block(m.count, m.before, words);
        if (t == 0) {  // rank(rows) reads these words
            m.before[words] = entries;
            if ((rows & 31) == 0) m.touch[words] = 0;
        }
        __syncthreads();
        // the vertices that have a term
        const int vwords = (nv + 31) / 32;
        for (int w = wid; w < vwords; w += nw) {
            const int k = w * 32 + lane;
            const bool some = k < nv && (walls || m.rank(m.row[k + 1]) > m.rank(m.row[k]));
            const unsigned b = __ballot_sync(0xffffffffu, some);
            if (lane == 0) m.vmask[w] = b;
        }
        // evaluate the queue, a window at a time (one, but far above any packing)
        for (int q0 = 0; q0 < entries || q0 == 0; q0 += kQueue) {
            const int q1 = min(entries, q0 + kQueue);
            for (int w = wid; w < words; w += nw) {
                const int at = m.before[w] + __popc(m.touch[w] & ((1u << lane) - 1u)) - q0;
                if ((m.touch[w] >> lane & 1u) && at >= 0 && at < kQueue) m.ent[at] = (unsigned short)(w * 32 + lane);
            }
            __syncthreads();
            if (q0 == 0) {  // the term vertices, their bodies' first
                for (int w = wid; w < vwords; w += nw) {
                    const int pre = (int)__reduce_add_sync(0xffffffffu, (unsigned)((lane < w ? __popc(m.vmask[lane]) : 0) +
                                                                                  (lane + 32 < w ? __popc(m.vmask[lane + 32]) : 0)));
                    const int k = w * 32 + lane, at = pre + __popc(m.vmask[w] & ((1u << lane) - 1u));
                    if (m.vmask[w] >> lane & 1u) m.tv[at] = (unsigned short)k;
                    if (k < nv && m.vfirst[m.vb[k]] == k) m.first[m.vb[k]] = at;
                    if (k == nv - 1) m.first[np] = at + (m.vmask[w] >> lane & 1u);
                }
            }
            for (int q = t; q < q1 - q0; q += nt) {
                const int e = m.ent[q];
                int k, j;
                entry_of(m, L, nv, v0, e, k, j);
                if (fp32) {
                    float *rf = reinterpret_cast<float *>(&m.res[0][0]);
                    float fx, fy;
                    rf[2 * kQueue + q] = mixed_pair(p, x.vpk[v0 + k], x.vpk[j], e_cf, n_cf, fx, fy);
                    rf[q] = fx;
                    rf[kQueue + q] = fy;
                } else {
                    double fx, fy;
                    const double ee = vertex_pair(fa, vc, m.vpos[k], fa.pos[j], fx, fy);
                    m.res[0][q] = fx;
                    m.res[1][q] = fy;
                    m.res[2][q] = ee;
                }
            }
            __syncthreads();
            const int terms = np > 0 ? m.first[np] : 0;
            for (int q = t; q < terms; q += nt) {
                const int k = m.tv[q], a0 = m.rank(m.row[k]), a1 = m.rank(m.row[k + 1]);
                const int b0 = max(a0, q0), b1 = min(a1, q1);
                double ax = 0.0, ay = 0.0, en = 0.0;
                if (fp32) {
                    const float *rf = reinterpret_cast<const float *>(&m.res[0][0]);
                    float sx = 0.f, sy = 0.f, se = 0.f;
                    if (a0 < q0 && b0 < b1) {  // carried over from the window before
                        sx = (float)m.term[0][q]; sy = (float)m.term[1][q]; se = (float)m.term[3][q];
                    }
                    for (int e = b0; e < b1; e++) {
                        sx += rf[e - q0];
                        sy += rf[kQueue + e - q0];
                        se += rf[2 * kQueue + e - q0];
                    }
                    ax = (double)sx; ay = (double)sy; en = (double)se;
                } else {
                    if (a0 < q0 && b0 < b1) { ax = m.term[0][q]; ay = m.term[1][q]; en = m.term[3][q]; }
                    for (int e = b0; e < b1; e++) {
                        ax += m.res[0][e - q0];
                        ay += m.res[1][e - q0];
                        en += m.res[2][e - q0];
                    }
                }
                if (a1 > q1) {  // goes on in the next window
                    if (b0 < b1) { m.term[0][q] = ax; m.term[1][q] = ay; m.term[3][q] = en; }
                    continue;
                }
                if (a1 <= q0 && q0 > 0) continue;  // done in an earlier window
                const int b = m.vb[k];
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
            if (q1 < entries) __syncthreads();
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
            ok = grid_totals<4>(tot, (np + 31) / 32, L.b.w.partials, ls, bk, polls, red);
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
    if (loop_exit(&L.b, ls, bk, polls, r, red)) *bs = L;
}

}  // namespace
}  // namespace dpg
