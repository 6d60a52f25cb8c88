// The step in two passes: the phase field c of every node first (phase kernels, into the work
// array StepArgs::cw), then the update of every node (update kernels), one thread per node.
//
// The one-pass kernels (step2d_body, step3d_body) compute c on a tile and its halo while they
// march, so a node's g is pulled up to 1.7 times and each plane waits for memory twice and for
// a barrier, one plane after the other.  Here every node is independent: a block asks for all
// it needs at once and the march's chain of planes is gone, for 84 bytes more per node (g
// read a second time, c written and read).  Measured on a B200, FP32 storage: 256x512x256
// bubble 2.92 -> 2.57 ms per step, 128x256x128 428 -> 341 us, 64x96x64 54 -> 41 us (against
// the march at its best planes per block; 488 us at the 64 planes a new solver used to take).
// Cutting the grid into chunks of planes, so that the second read of g comes from L2, did not
// pay: each chunk's two launches drain the GPU (16 planes: 2.72 ms, 64: 2.66, all: 2.66).
#pragma once

#include "kernels.cuh"
#include "tma.cuh"

namespace clipb {

// ---------------------------------------------------------------- any side
// c of this step at (x, y, z), ghost coordinates included.
template <int DIM, class PR, bool kOpen>
__global__ void __launch_bounds__(256) phase_kernel(StepArgs<PR> a, int z_first) {
    using L = Lat<DIM>;
    using TP = typename PR::TP;
    using A = typename PR::A;
    const Geom& g = a.g;
    const Codec<PR> cd(a.pop_scale);
    const int x = 1 + (int)(blockIdx.x * 32 + threadIdx.x), y = (int)(blockIdx.y * 8 + threadIdx.y);
    const int z = DIM == 3 ? z_first + (int)blockIdx.z : 0;
    if (x > g.n[0] || y > g.n[1] + 1) return;
    const unsigned self = nidx32(g, x, y, z);
    typename PR::Ring c;
    if (y >= 1 && y <= g.n[1] && (DIM == 2 || (z >= 1 && z <= g.n[2]))) {
        TP v[L::Q], cs;
        pull_g<DIM, PR, kOpen>(a.gin, a.cin, cd, g, x, y, z, self, cross_mask<DIM>(g, x, y, z), v, cs, a.par);
        c = ring_c<PR>(pulled_sum<PR, L::Q>(v), cs);
    } else {
        c = ring_of<PR>(ghost_c<DIM, A>(a.cin, g, x, y, z));
    }
    a.cw[self] = c;
    if (x == 1) a.cw[self - 1] = ring_of<PR>(ghost_c<DIM, A>(a.cin, g, 0, y, z));
    if (x == g.n[0]) a.cw[self + 1] = ring_of<PR>(ghost_c<DIM, A>(a.cin, g, x + 1, y, z));
}

// Update of every node after phase_kernel.
template <int DIM, class PR, bool kOpen>
__global__ void __launch_bounds__(128, 4) update_kernel(StepArgs<PR> a) {
    using L = Lat<DIM>;
    using TP = typename PR::TP;
    using T = typename PR::T;
    constexpr int Q = L::Q;
    const Geom& g = a.g;
    const Codec<PR> cd(a.pop_scale);
    const int x = 1 + (int)(blockIdx.x * 32 + threadIdx.x), y = 1 + (int)(blockIdx.y * 4 + threadIdx.y);
    const int z = DIM == 3 ? g.zlo + (int)blockIdx.z : 0;
    if (x > g.n[0] || y > g.n[1]) return;
    const unsigned self = nidx32(g, x, y, z), mask = cross_mask<DIM>(g, x, y, z);
    T fpost[Q];
    TP gpost[Q], cold;
    pull_f<DIM, PR, kOpen>(a.fin, cd, g, x, y, z, self, mask, fpost, a.par);
    pull_g<DIM, PR, kOpen>(a.gin, a.cin, cd, g, x, y, z, self, mask, gpost, cold, a.par);
    const typename PR::Ring* cw = a.cw;
    auto Cf = [&](int dx, int dy, int dz) {
        return cw[self + unsigned(dx) + unsigned(dy) * unsigned(g.sy) + (DIM == 3 ? unsigned(dz) * unsigned(g.sz) : 0u)];
    };
    auto Ch = [&](int dx, int dy, int dz) -> TP { return ring_hi<PR>(Cf(dx, dy, dz)); };
    TP mu, dc[3] = {TP(0), TP(0), TP(0)};
    phase_stencil<DIM, PR>(a.pp, Cf, mu, dc);
    const unsigned dmask = cross_mask<DIM, true>(g, x, y, z);
    const TP cown = Ch(0, 0, 0);
    auto cdest = [&](int q) { return dest_shift_q<DIM, PR>(q, dmask, cown, Ch); };
    auto gq = [&](int q) { return gpost[q]; };
    if (kOpen && g.fc[0]) store_open<DIM, PR>(g, a.par, x, y, z, fpost, gq, cold, cown);
    update_node<DIM, PR>(a, cd, a.pt, a.pp, self, fpost, gq, pulled_sum<PR, Q>(gpost), cold, cown, mu, dc, cdest);
    if (kOpen && g.fc[0]) store_open_u<DIM, PR>(g, a.par, x, y, z, a.u, self);
}

// ---------------------------------------------------------------- FP32/FP16, 3D
// Per direction, the source and the destination of a node's populations as functions of its
// element index (nidx32): filled on the host, read from the parameter space, so that the
// address of a load or store is one multiply-add on a constant.
template <class PR>
struct PullPtrs {
    const typename PR::Sf* f[19];
    const typename PR::Sg* g[19];
    typename PR::Sf* fo[19];
    typename PR::Sg* go[19];
};

// Boundary summary of one node away from the z sides: element offsets that wrap a source
// beyond a periodic x side, and whether the node needs the general pull (next to a y side,
// or to an x side that is not periodic).  A quarter of the warps of a 256-wide periodic grid
// hold a node next to an x side; these offsets cost them little, where the general pull
// resolves all 19 directions of every lane.
struct Column {
    unsigned lo, hi;
    bool general;
    __device__ __forceinline__ Column(const Geom& g, int x, int y) {
        const bool per = g.side[0] == kSidePeriodic;
        lo = per && x == 1 ? unsigned(g.n[0]) : 0u;
        hi = per && x == g.n[0] ? unsigned(-g.n[0]) : 0u;
        general = y == 1 || y == g.n[1] || (!per && (x == 1 || x == g.n[0]));
    }
    // element whose fixed lattice offset gives the source of a direction with x component ex
    __device__ __forceinline__ unsigned from(unsigned self, int ex) const {
        return ex == 0 ? self : self + (ex > 0 ? lo : hi);
    }
    __device__ __forceinline__ bool wraps() const { return (lo | hi) != 0u; }
};

// The g that crossed a periodic x side were stored shifted by their own node's c (see Prec):
// wrapped_c requests the c of the five sources, unshift brings the values to this node's c, as
// pull_g does.  Both only for a node whose column wraps.
template <class A>
__device__ __forceinline__ void wrapped_c(const A* __restrict__ C, const Geom& g, const Column& col, unsigned self, float* wc) {
    const unsigned s = self + col.lo + col.hi + (col.lo ? 0u : 2u);
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        constexpr int q[5] = {1, 7, 9, 11, 13};
        wc[i] = C[s + pull_offset<3>(g, q[i]) - unsigned(q[i]) * unsigned(g.ps)];
    }
}
__device__ __forceinline__ void unshift(const Column& col, const float* wc, float cself, float* v) {
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        constexpr int up[5] = {1, 7, 9, 11, 13}, dn[5] = {2, 10, 8, 14, 12};  // e_x = +1 and their mirrors
        const float w = Lat<3>::ws(up[i]), dcs = wc[i] - cself;
        v[up[i]] = col.lo ? fmaf(w, dcs, v[up[i]]) : v[up[i]];
        v[dn[i]] = col.lo ? v[dn[i]] : fmaf(w, dcs, v[dn[i]]);
    }
}

// phase_kernel with the boundary work of most warps reduced to two base offsets, and addresses
// of one multiply-add each (PullPtrs): 230 instead of 382 instructions per node, 70 instead of
// 79 us on the 128x256x128 bubble (88 bytes per node at 5.3 TB/s).
template <class PR>
__global__ void __launch_bounds__(256) phase3_kernel(StepArgs<PR> a, PullPtrs<PR> ptr, int z_first) {
    using L = Lat<3>;
    const Geom& g = a.g;
    const Codec<PR> cd(a.pop_scale);
    const int x = 1 + (int)(blockIdx.x * 32 + threadIdx.x), y = (int)(blockIdx.y * 8 + threadIdx.y);
    const int z = z_first + (int)blockIdx.z;
    // the launch may overlap the end of the kernel before it; the update launched after it may
    // overlap this one only once that kernel has ended
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (x > g.n[0] || y > g.n[1] + 1) return;
    const unsigned self = nidx32(g, x, y, z);
    float2 c;
    if (y >= 1 && y <= g.n[1] && z >= 1 && z <= g.n[2]) {
        const Column col(g, x, y);
        float v[L::Q], cs;
        if (!__any_sync(__activemask(), col.general || z == 1 || z == g.n[2])) {
            float wc[5];
            cs = a.cin[self];
#pragma unroll
            for (int q = 0; q < L::Q; ++q) v[q] = cd.load_dev(ptr.g[q] + col.from(self, L::ex(q)));
            if (col.wraps()) {
                wrapped_c(a.cin, g, col, self, wc);
                unshift(col, wc, cs, v);
            }
        } else {
            pull_g<3, PR>(a.gin, a.cin, cd, g, x, y, z, self, cross_mask<3>(g, x, y, z), v, cs, a.par);
        }
        c = ring_c<PR>(pulled_sum<PR, L::Q>(v), cs);
    } else {
        c = ring_of<PR>(ghost_c<3, float>(a.cin, g, x, y, z));
    }
    a.cw[self] = c;
    if (x == 1) a.cw[self - 1] = ring_of<PR>(ghost_c<3, float>(a.cin, g, 0, y, z));
    if (x == g.n[0]) a.cw[self + 1] = ring_of<PR>(ghost_c<3, float>(a.cin, g, x + 1, y, z));
}

// 8 bytes from global to shared memory without a register between (completion: copy_async_wait
// of the issuing thread, then a barrier).
__device__ __forceinline__ void copy_async8(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Update of one node per thread, blocks of 32 x TY nodes of a plane, after phase3_kernel.
// Bound by memory (340 bytes of DRAM traffic per node at 5.1 TB/s; a bare copy of the same
// populations runs at 5.8).  A block asks for its 38 populations per node, u and the old c
// before it waits for anything; f is reduced to its moments as it arrives, so that 128
// registers hold it all without spills (a spilled load in flight stalls: at 80 registers and
// 24 warps per SM the 128x256x128 update took 370 instead of 277 us).  Small blocks of 4 rows
// keep the loads of some beside the arithmetic of others: 8 rows took 316 us, 2 rows 277.
template <class PR, int TY, bool kMon>
__global__ void __launch_bounds__(32 * TY, 16 / TY) update3_kernel(StepArgs<PR> a, PullPtrs<PR> ptr, int z_first) {
    using L = Lat<3>;
    constexpr int Q = L::Q, CW = 34;  // tile row: the nodes x0 - 1 .. x0 + 32
    __shared__ float2 tile[3][TY + 2][CW];
    const Geom& g = a.g;
    const Codec<PR> cd(a.pop_scale);
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int x0 = 1 + (int)blockIdx.x * 32, x = x0 + tx, y0 = (int)blockIdx.y * TY, y = 1 + y0 + ty;
    // planes in descending order: phase3_kernel left the g of the highest ones in L2
    const int z = z_first + (int)(gridDim.z - 1 - blockIdx.z);
    const bool active = x <= g.n[0] && y <= g.n[1];
    const unsigned self = nidx32(g, x, y, z);
    const Column col(g, x, y);
    const bool fast = !__any_sync(0xffffffffu, active && (col.general || z == 1 || z == g.n[2]));
    float f[Q], d[Q], u[3], cold = 0.f, wc[5];
    if (active) {
        if (fast) {
#pragma unroll
            for (int q = 0; q < Q; ++q) f[q] = cd.load_f(ptr.f[q] + col.from(self, L::ex(q)));
#pragma unroll
            for (int q = 0; q < Q; ++q) d[q] = cd.load_dev(ptr.g[q] + col.from(self, L::ex(q)));
            if (col.wraps()) wrapped_c(a.cin, g, col, self, wc);
        }
        cold = a.cin[self];
#pragma unroll
        for (int k = 0; k < 3; ++k) u[k] = a.uin[self + unsigned(k) * unsigned(g.ps)];
    }
    // c of the tile and the nodes around it: phase3_kernel, which this launch may overlap up to
    // here (the requests above read nothing it writes)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    for (int r = ty; r < 3 * (TY + 2); r += TY) {
        const int dz = r / (TY + 2), dy = r - dz * (TY + 2);
        if (y0 + dy > g.n[1] + 1) continue;
        const float2* src = a.cw + nidx32(g, x - 1, y0 + dy, z - 1 + dz);
        float2* dst = &tile[dz][dy][tx];
        if (x - 1 <= g.n[0] + 1) copy_async8(dst, src);
        if (tx < 2 && x + 31 <= g.n[0] + 1) copy_async8(dst + 32, src + 32);
    }
    Moments m = {};
    float delta = 0.f;
    if (active) {
        const unsigned mask = cross_mask<3>(g, x, y, z);
        if (!fast) pull_f<3, PR>(a.fin, cd, g, x, y, z, self, mask, f, a.par);
        m = lean_moments<3>(f);
        if (!fast) pull_g<3, PR>(a.gin, a.cin, cd, g, x, y, z, self, mask, d, cold, a.par);
        else if (col.wraps()) unshift(col, wc, cold, d);
        delta = pulled_sum<PR, Q>(d);
    }
    copy_async_wait();
    __syncthreads();
    double mon[2] = {0.0, 0.0};
    if (active) {
        auto C = [&](int dx, int dy, int dz) { return tile[1 + dz][1 + ty + dy][1 + tx + dx]; };
        float mu, dc[3];
        stencil_hilo<3>(a.pp, C, mu, dc);
        const float c = C(0, 0, 0).x;
        const unsigned dmask = cross_mask<3, true>(g, x, y, z);
        auto cdest = [&](int q) {
            return dest_shift_q<3, PR>(q, dmask, c, [&](int dx, int dy, int dz) { return C(dx, dy, dz).x; });
        };
        lean_update<3>(a.pt, m, [&](int q) { return d[q]; }, delta, cold, c, mu, dc, u, cdest, [&](int q, float fo, float go) {
            cd.store_dev(ptr.go[q] + self, go);
            cd.store_f(ptr.fo[q] + self, fo);
        });
#pragma unroll
        for (int k = 0; k < 3; ++k) a.u[self + unsigned(k) * unsigned(g.ps)] = u[k];
        a.cout[self] = c;
        if constexpr (kMon) node_monitors<3, PR>(a, c, u, mon);
    }
    if constexpr (kMon) store_monitor_row(a, tx, x0, y, z, mon);
}

}  // namespace clipb
