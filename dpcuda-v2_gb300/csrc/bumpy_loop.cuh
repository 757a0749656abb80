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

struct BumpyLoopMem {
    MoveMem move;
    double sum[kLoopBodies][4];
};

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
    mx = 0;
    for (int b = v0; b < v1; b += nt / kVlistLanes) {
        const int u = b + t / kVlistLanes;
        const bool real = u < v1;
        const int cnt = vlist_row<kVlistLanes>(bs, u, real);
        if (real && t % kVlistLanes == 0) {
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

template <int KIND>
__global__ void __launch_bounds__(kLoopMaxTPB, 1) kb_loop(BumpySys *bs, LoopSync *ls, double dt, double tmax,
                                                         int chunk, long long iters) {
    extern __shared__ __align__(16) unsigned char loop_smem[];
    ForceWarp *fw = reinterpret_cast<ForceWarp *>(loop_smem);
    __shared__ BumpySys L;
    __shared__ BumpyLoopMem m;
    __shared__ double red[32 * 3];
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5, nw = blockDim.x >> 5;
    if (t == 0) L = *bs;
    __syncthreads();
    DevState &s = L.b.s;
    BumpyExt &x = L.x;
    if (s.flags) return;  // the same for every block: nothing writes the state before a barrier
    const int n = L.b.p.n;
    const Range r = {min((int)blockIdx.x * chunk, n), min(((int)blockIdx.x + 1) * chunk, n)};
    const int np = r.last - r.first;
    unsigned bk = 0;
    bool ok = true;
    long long it = 0;
    const double dt_half = 0.5 * dt;

    // the barrier after a move and a rebuild if any body asks for one
    auto after_move = [&](double nd2, double cd2) {
        const unsigned long long bw = grid_bar(ls, bk, block_flags(move_flags(L.b.p, nd2, cd2)));
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
        return !kind || bumpy_rebuild(&L, ls, bk, kind, r);
    };
    auto nve_first = [&]() {
        double nd2 = 0.0, cd2 = 0.0;
        bodies_move(&L, r.first, r.last, dt, m.move, [&](int b) { body_kick(&L, b, dt_half); }, nd2, cd2,
                    x.vpos_t, x.vpk_t, x.vq_t);
        return after_move(nd2, cd2);
    };

    if (KIND == 1) ok = nve_first();
    while (ok) {
        if (KIND == 0) {
            double nd2 = 0.0, cd2 = 0.0;
            bodies_fire_move(&L, r.first, r.last, m.move, nd2, cd2);
            ok = after_move(nd2, cd2);
            if (!ok) break;
        }
        for (int b = r.first + wid; b < r.last; b += nw) {
            const double sum = body_forces(&L, b, KIND == 1 && s.walls != 0, fw[wid]);
            if (lane < 4) m.sum[b - r.first][lane] = sum;
        }
        __syncthreads();
        it++;
        const double *q = m.sum[t < np ? t : 0];
        if (KIND == 1) {
            if (t < np) body_nve_second(&L, r.first + t, q[0], q[1], q[2], q[3], dt_half);
            const bool last = it >= iters || s.nve_steps_done + 1 >= s.max_steps;
            __syncthreads();  // every thread has read the state
            if (t == 0 && ++s.nve_steps_done >= s.max_steps) s.flags |= kDone;
            __syncthreads();
            if (last) break;
            ok = nve_first();
        } else {
            double tot[4] = {0.0, 0.0, 0.0, 0.0};
            if (t < np) body_fire_second(&L, r.first + t, q[0], q[1], q[2], q[3], true, tot);
            ok = grid_totals<4>(tot, (np + 31) / 32, L.b.w.partials, ls, bk, red);
            if (!ok) break;
            if (t == 0) bumpy_fire_epilogue(&L, tot, tmax);
            __syncthreads();
            if (s.flags || it >= iters) break;
        }
    }
    if (loop_exit(&L.b, ls, bk, r, red)) *bs = L;
}

}  // namespace
}  // namespace dpg
