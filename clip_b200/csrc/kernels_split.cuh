// The step in two passes: the phase field c of every node first (phase_kernel, into the work
// array StepArgs::cw), then the update of every node (update_kernel, update_fp64_kernel), one
// thread per node.
//
// The one-pass kernels (step2d_body, step3d_body) compute c on a tile and its halo while they
// march, so a node's g is pulled up to 1.7 times and each plane waits for memory twice and for
// a barrier, one plane after the other.  Here every node is independent: a block asks for all
// it needs at once and the march's chain of planes is gone, for 92 bytes more per node (FP32;
// g read a second time, c written and read).  Measured on a B200, us per step of one solver with
// nothing else on the GPU, against the march at its best tile and planes per block:
//   FP32 3D: 256x512x256 2575 / 2946 (2730 / 2968 once the 1 kW power cap acts, after some 100
//     steps), 128x256x128 340 / 432, 64x96x64 40 / 54
//   FP64 3D: 128x256x128 868 / 1086, 97x131x83 305 / 396, 64x96x64 92 / 137
//   2D, FP64: 256x1024 25.3 / 32.8, 64x128 6.0 / 8.3; FP32: 201x777 10.0 / 14.0, 64x128 5.7 / 7.0
// Cutting a 3D grid into chunks of planes, so that the second read of g comes from L2, did not
// pay: each chunk's two launches drain the GPU (16 planes: 2.72 ms, 64: 2.66, all: 2.66).
//
// The launches of a step are chained (programmatic dependent launch): the phase field waits for
// the kernel before it and then lets the update start, which asks for its populations, written
// a step ago, before it waits for the phase field.
#pragma once

#include "kernels.cuh"
#include "tma.cuh"

namespace clipb {

// Per direction, the source and the destination of a node's populations as functions of its
// element index (nidx32): filled on the host, read from the parameter space, so that the
// address of a load or store is one multiply-add on a constant.
template <int DIM, class PR>
struct PullPtrs {
    const typename PR::Sf* f[Lat<DIM>::Q];
    const typename PR::Sg* g[Lat<DIM>::Q];
    typename PR::Sf* fo[Lat<DIM>::Q];
    typename PR::Sg* go[Lat<DIM>::Q];
    __device__ __forceinline__ const typename PR::Sf* f_from(int q, unsigned i) const { return f[q] + i; }
    __device__ __forceinline__ const typename PR::Sg* g_from(int q, unsigned i) const { return g[q] + i; }
    __device__ __forceinline__ typename PR::Sf* f_to(int q, unsigned i) const { return fo[q] + i; }
    __device__ __forceinline__ typename PR::Sg* g_to(int q, unsigned i) const { return go[q] + i; }
};
// The same from the buffers' bases, for the cases of a batch, whose arguments are not kernel
// parameters.
template <int DIM, class PR>
struct BasePtrs {
    const StepArgs<PR>& a;
    __device__ __forceinline__ const typename PR::Sf* f_from(int q, unsigned i) const { return a.fin + (i + pull_offset<DIM>(a.g, q)); }
    __device__ __forceinline__ const typename PR::Sg* g_from(int q, unsigned i) const { return a.gin + (i + pull_offset<DIM>(a.g, q)); }
    __device__ __forceinline__ typename PR::Sf* f_to(int q, unsigned i) const { return a.fout + (i + unsigned(q) * unsigned(a.g.ps)); }
    __device__ __forceinline__ typename PR::Sg* g_to(int q, unsigned i) const { return a.gout + (i + unsigned(q) * unsigned(a.g.ps)); }
};

// Boundary summary of one node: element offsets that wrap a source beyond a periodic x side,
// whether the sources beyond its x side lie behind a wall, and whether the node needs the
// general pull (next to a y or z side, or to an x side of another kind).  A quarter of the warps
// of a 256-wide grid hold a node next to an x side; these cost them little, where the general
// pull resolves every direction of every lane.
// kWalls: the instance for cases with a wall in x (FP32/FP16; the others take the general pull
// next to it: the choice of addresses costs a 2D step without such walls 4%, and FP64, bound by
// its arithmetic, gains 2% with them and loses 1% without).  97x131x83 in walls 146 -> 118 us.
template <int DIM, bool kWalls>
struct Column {
    unsigned lo, hi;
    bool wall_lo, wall_hi, general;
    __device__ __forceinline__ Column(const Geom& g, int x, int y, int z) {
        const bool per = g.side[0] == kSidePeriodic;  // then the other x side is as well
        lo = per && x == 1 ? unsigned(g.n[0]) : 0u;
        hi = per && x == g.n[0] ? unsigned(-g.n[0]) : 0u;
        wall_lo = kWalls && x == 1 && g.side[0] == kSideWall;
        wall_hi = kWalls && x == g.n[0] && g.side[1] == kSideWall;
        general = y == 1 || y == g.n[1] || (!per && ((x == 1 && !wall_lo) || (x == g.n[0] && !wall_hi))) ||
                  (DIM == 3 && (z == 1 || z == g.n[2]));
    }
    // element whose fixed lattice offset gives the source of a direction with x component ex
    __device__ __forceinline__ unsigned from(unsigned self, int ex) const {
        return ex == 0 ? self : self + (ex > 0 ? lo : hi);
    }
    __device__ __forceinline__ bool wraps() const { return (lo | hi) != 0u; }
    __device__ __forceinline__ bool walled() const { return wall_lo || wall_hi; }
    // a direction with x component ex bounces back at this node
    __device__ __forceinline__ bool bounces(int ex) const { return ex > 0 ? wall_lo : (ex < 0 ? wall_hi : false); }
};
// The streamed populations of a node that needs no general pull: at(q, i) is the source of
// direction q of element i (PullPtrs).  A warp without a node next to an x wall reads the fixed
// offsets; the others choose each address between the source and the node's own opposite
// population.
template <int DIM, bool kWalls, typename T, class At, class Load>
__device__ __forceinline__ void pull_column(const Geom& g, const Column<DIM, kWalls>& col, unsigned self, T* v, At at, Load load) {
    using L = Lat<DIM>;
    if (kWalls && __any_sync(__activemask(), col.walled())) {
#pragma unroll
        for (int q = 0; q < L::Q; ++q) {
            const int o = opposite<DIM>(q);
            auto* src = at(q, col.from(self, L::ex(q)));
            auto* own = at(o, self - pull_offset<DIM>(g, o) + unsigned(o) * unsigned(g.ps));
            v[q] = load(col.bounces(L::ex(q)) ? own : src);
        }
    } else {
#pragma unroll
        for (int q = 0; q < L::Q; ++q) v[q] = load(at(q, col.from(self, L::ex(q))));
    }
}

// Shifted storage: the g that crossed a periodic x side were stored shifted by their own node's
// c (see Prec).  wrapped_c requests the c of those sources, unshift brings the values to this
// node's c, as pull_g does.  Both only for a node whose column wraps.  Direction i of the A
// with e_x = +1 and its mirror with e_x = -1:
template <int DIM>
__host__ __device__ constexpr int from_low(int i) { return wall_dir<DIM>(0, i); }
template <int DIM>
__host__ __device__ constexpr int from_high(int i) {
    const int q = from_low<DIM>(i);
    for (int m = 0; m < Lat<DIM>::Q; ++m)
        if (Lat<DIM>::ex(m) == -1 && Lat<DIM>::ey(m) == Lat<DIM>::ey(q) && Lat<DIM>::ez(m) == Lat<DIM>::ez(q)) return m;
    return 0;
}
template <int DIM, bool kWalls, class A>
__device__ __forceinline__ void wrapped_c(const A* __restrict__ C, const Geom& g, const Column<DIM, kWalls>& col, unsigned self,
                                          A* wc) {
    const unsigned s = self + col.lo + col.hi + (col.lo ? 0u : 2u);
#pragma unroll
    for (int i = 0; i < Lat<DIM>::A; ++i) {
        const int q = from_low<DIM>(i);
        wc[i] = C[s + pull_offset<DIM>(g, q) - unsigned(q) * unsigned(g.ps)];
    }
}
template <int DIM, bool kWalls>
__device__ __forceinline__ void unshift(const Column<DIM, kWalls>& col, const float* wc, float cself, float* v) {
#pragma unroll
    for (int i = 0; i < Lat<DIM>::A; ++i) {
        const int up = from_low<DIM>(i), dn = from_high<DIM>(i);
        const float w = Lat<DIM>::ws(up), dcs = wc[i] - cself;
        v[up] = col.lo ? fmaf(w, dcs, v[up]) : v[up];
        v[dn] = col.lo ? v[dn] : fmaf(w, dcs, v[dn]);
    }
}


// c of this step at (x, y, z), ghost coordinates included (x an interior node's: its neighbours
// in the x ghost columns with it).
template <int DIM, class PR, bool kOpen, bool kWalls, class Ptr>
__device__ __forceinline__ void phase_node(const StepArgs<PR>& a, const Ptr& ptr, int x, int y, int z) {
    using L = Lat<DIM>;
    using TP = typename PR::TP;
    using A = typename PR::A;
    const Geom& g = a.g;
    const Codec<PR> cd(a.pop_scale);
    const unsigned self = nidx32(g, x, y, z);
    typename PR::Ring c;
    if (y >= 1 && y <= g.n[1] && (DIM == 2 || (z >= 1 && z <= g.n[2]))) {
        const Column<DIM, kWalls> col(g, x, y, z);
        TP v[L::Q], cs = TP(0);
        if (__any_sync(__activemask(), col.general)) {
            pull_g<DIM, PR, kOpen>(a.gin, a.cin, cd, g, x, y, z, self, cross_mask<DIM>(g, x, y, z), v, cs, a.par);
        } else {
            if constexpr (PR::kShift) cs = a.cin[self];
            pull_column(g, col, self, v, [&](int q, unsigned i) { return ptr.g_from(q, i); }, [&](auto* p) { return cd.load_dev(p); });
            if constexpr (PR::kShift)
                if (col.wraps()) {
                    float wc[L::A];
                    wrapped_c(a.cin, g, col, self, wc);
                    unshift(col, wc, cs, v);
                }
        }
        c = ring_c<PR>(pulled_sum<PR, L::Q>(v), cs);
    } else {
        c = ring_of<PR>(ghost_c<DIM, A>(a.cin, g, x, y, z));
    }
    a.cw[self] = c;
    if (x == 1) a.cw[self - 1] = ring_of<PR>(ghost_c<DIM, A>(a.cin, g, 0, y, z));
    if (x == g.n[0]) a.cw[self + 1] = ring_of<PR>(ghost_c<DIM, A>(a.cin, g, x + 1, y, z));
}

// Bound by memory: 70 us on the 128x256x128 bubble in FP32, 88 bytes per node at 5.3 TB/s (79
// us, 382 instead of 230 instructions per node, with the general pull in every warp next to a
// side).
template <int DIM, class PR, bool kOpen, bool kWalls>
__global__ void __launch_bounds__(256) phase_kernel(StepArgs<PR> a, PullPtrs<DIM, PR> ptr, int z_first) {
    const int x = 1 + (int)(blockIdx.x * 32 + threadIdx.x), y = (int)(blockIdx.y * blockDim.y + threadIdx.y);
    // in this order: the update may start once everything before this kernel has ended
    wait_for_predecessor();
    let_successor_start();
    if (x <= a.g.n[0] && y <= a.g.n[1] + 1) phase_node<DIM, PR, kOpen, kWalls>(a, ptr, x, y, DIM == 3 ? z_first + (int)blockIdx.z : 0);
}

// 8 bytes from global to shared memory without a register between (completion: copy_async_wait
// of the issuing thread, then a barrier).
__device__ __forceinline__ void copy_async8(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// FP32/FP16 update of the 32 x TY tile of a plane whose first node is (x0, y0, z), rows up to
// y_last, one node per thread.  PT: a.pt, PP: a.pp (or copies of them in registers).
template <int DIM, class PR, int TY, bool kOpen, bool kWalls, bool kMon, class Ptr>
__device__ __forceinline__ void update_tile(const StepArgs<PR>& a, const Phys<float>& PT, const Phys<float>& PP, const Ptr& ptr,
                                            int x0, int y0, int z, int y_last, float2 (*tile)[TY + 2][34]) {
    using L = Lat<DIM>;
    constexpr int Q = L::Q, PZ = DIM == 3 ? 3 : 1;
    const Geom& g = a.g;
    const Codec<PR> cd(a.pop_scale);
    const int tx = threadIdx.x, ty = threadIdx.y, x = x0 + tx, y = y0 + ty;
    const bool active = x <= g.n[0] && y <= y_last;
    const unsigned self = nidx32(g, x, y, z);
    const Column<DIM, kWalls> col(g, x, y, z);
    const bool fast = !__any_sync(0xffffffffu, active && col.general);
    float f[Q], d[Q], u[3], cold = 0.f, wc[L::A];
    if (active) {
        if (fast) {
            pull_column(g, col, self, f, [&](int q, unsigned i) { return ptr.f_from(q, i); }, [&](auto* p) { return cd.load_f(p); });
            pull_column(g, col, self, d, [&](int q, unsigned i) { return ptr.g_from(q, i); }, [&](auto* p) { return cd.load_dev(p); });
            if (col.wraps()) wrapped_c(a.cin, g, col, self, wc);
        }
        cold = a.cin[self];
#pragma unroll
        for (int k = 0; k < DIM; ++k) u[k] = a.uin[self + unsigned(k) * unsigned(g.ps)];
    }
    // c of the tile and the nodes around it (tile row: x0 - 1 .. x0 + 32), from the phase field,
    // which this launch may overlap up to here (the requests above read nothing it writes)
    wait_for_predecessor();
    let_successor_start();
    for (int r = ty; r < PZ * (TY + 2); r += TY) {
        const int dz = DIM == 3 ? r / (TY + 2) : 0, dy = r - dz * (TY + 2);
        if (y0 + dy > g.n[1] + 2) continue;
        const float2* src = a.cw + nidx32(g, x - 1, y0 - 1 + dy, DIM == 3 ? z - 1 + dz : 0);
        float2* dst = &tile[dz][dy][tx];
        if (x - 1 <= g.n[0] + 1) copy_async8(dst, src);
        if (tx < 2 && x + 31 <= g.n[0] + 1) copy_async8(dst + 32, src + 32);
    }
    Moments m = {};
    float delta = 0.f;
    if (active) {
        const unsigned mask = cross_mask<DIM>(g, x, y, z);
        if (!fast) pull_f<DIM, PR, kOpen>(a.fin, cd, g, x, y, z, self, mask, f, a.par);
        m = lean_moments<DIM>(f);
        if (!fast) {
            pull_g<DIM, PR, kOpen>(a.gin, a.cin, cd, g, x, y, z, self, mask, d, cold, a.par);
            if (kOpen && g.fc[0]) store_open<DIM, PR>(g, a.par, x, y, z, f, [&](int q) { return d[q]; }, cold, a.cw[self].x);
        } else if (col.wraps()) {
            unshift(col, wc, cold, d);
        }
        delta = pulled_sum<PR, Q>(d);
    }
    copy_async_wait();
    __syncthreads();
    double mon[2] = {0.0, 0.0};
    if (active) {
        auto C = [&](int dx, int dy, int dz) { return tile[PZ / 2 + dz][1 + ty + dy][1 + tx + dx]; };
        float mu, dc[3] = {0.f, 0.f, 0.f};
        stencil_hilo<DIM>(PP, C, mu, dc);
        const float c = C(0, 0, 0).x;
        const unsigned dmask = cross_mask<DIM, true>(g, x, y, z);
        auto cdest = [&](int q) {
            return dest_shift_q<DIM, PR>(q, dmask, c, [&](int dx, int dy, int dz) { return C(dx, dy, dz).x; });
        };
        lean_update<DIM>(PT, m, [&](int q) { return d[q]; }, delta, cold, c, mu, dc, u, cdest, [&](int q, float fo, float go) {
            cd.store_dev(ptr.g_to(q, self), go);
            cd.store_f(ptr.f_to(q, self), fo);
        });
#pragma unroll
        for (int k = 0; k < DIM; ++k) a.u[self + unsigned(k) * unsigned(g.ps)] = u[k];
        a.cout[self] = c;
        if (kOpen && g.fc[0]) store_open_u<DIM, PR>(g, a.par, x, y, z, a.u, self);
        if constexpr (kMon) node_monitors<DIM, PR>(a, c, u, mon);
    }
    if constexpr (kMon) store_monitor_row(a, tx, x0, y, z, mon);
}

// In 3D bound by memory (340 bytes of DRAM traffic per node at 5.1 TB/s; a bare copy of the same
// populations runs at 5.8).  A block asks for all populations of its nodes, u and the old c
// before it waits for anything; f is reduced to its moments as it arrives, so that 128
// registers hold it all without spills (a spilled load in flight stalls: at 80 registers and
// 24 warps per SM the 128x256x128 update took 370 instead of 277 us).  Small blocks of 4 rows
// keep the loads of some beside the arithmetic of others: 8 rows took 316 us, 2 rows 277.
template <int DIM, class PR, int TY, bool kOpen, bool kWalls, bool kMon>
__global__ void __launch_bounds__(32 * TY, 16 / TY) update_kernel(StepArgs<PR> a, PullPtrs<DIM, PR> ptr, int z_first) {
    __shared__ float2 tile[DIM == 3 ? 3 : 1][TY + 2][34];
    // planes in descending order: phase_kernel left the g of the highest ones in L2
    update_tile<DIM, PR, TY, kOpen, kWalls, kMon>(a, a.pt, a.pp, ptr, 1 + (int)blockIdx.x * 32, 1 + (int)blockIdx.y * TY,
                                   DIM == 3 ? z_first + (int)(gridDim.z - 1 - blockIdx.z) : 0, a.g.n[1], tile);
}

// The two passes over the cases of a batch (2D, FP32/FP16): a block takes one work item (case,
// tile column bx, rows by * seg + 1 ... of it), its case's step arguments copied from the device
// table into shared memory.  512 seeded-size cases (22.2 M nodes), FP32: 0.97 ms per step at 16
// rows per item (4 rows 1.09, 8 1.00, 64 0.99) against 1.15 ms for the marching batch kernel.
template <class PR>
__device__ __forceinline__ void copy_args(StepArgs<PR>* sa, const StepArgs<PR>* args) {
    static_assert(sizeof(StepArgs<PR>) % 4 == 0, "copied in 4-byte words");
    const unsigned* src = reinterpret_cast<const unsigned*>(args);
    unsigned* dst = reinterpret_cast<unsigned*>(sa);
    for (int w = (int)(threadIdx.y * 32 + threadIdx.x); w < (int)(sizeof(StepArgs<PR>) / 4); w += (int)(32 * blockDim.y)) dst[w] = src[w];
    __syncthreads();
}
template <class PR>
__global__ void __launch_bounds__(128) phase_batch_kernel(const StepArgs<PR>* __restrict__ args, const int* __restrict__ items, int seg) {
    __shared__ StepArgs<PR> a;
    const int* it = items + 3 * blockIdx.x;
    const int x = 1 + it[1] * 32 + (int)threadIdx.x, by = it[2];
    copy_args(&a, args + it[0]);
    wait_for_predecessor();
    let_successor_start();
    const int n1 = a.g.n[1], last = min(by * seg + seg, n1);
    if (x > a.g.n[0]) return;
    const BasePtrs<2, PR> ptr{a};
    for (int y = (by == 0 ? 0 : by * seg + 1) + (int)threadIdx.y; y <= (last == n1 ? n1 + 1 : last); y += 4)
        phase_node<2, PR, false, false>(a, ptr, x, y, 0);
}
template <class PR>
__global__ void __launch_bounds__(128, 8) update_batch_kernel(const StepArgs<PR>* __restrict__ args, const int* __restrict__ items, int seg) {
    __shared__ StepArgs<PR> a;
    __shared__ float2 tile[1][6][34];
    const int* it = items + 3 * blockIdx.x;
    const int bx = it[1], by = it[2];
    copy_args(&a, args + it[0]);
    // the parameters as locals: through a reference to shared memory every use is a load
    const Phys<float> PT = a.pt, PP = a.pp;
    const BasePtrs<2, PR> ptr{a};
    const int y1 = min(by * seg + seg, a.g.n[1]);
    for (int y = by * seg + 1; y <= y1; y += 4) {
        update_tile<2, PR, 4, false, false, false>(a, PT, PP, ptr, 1 + bx * 32, y, 0, y1, tile);
        __syncthreads();  // the tile is reused by the next rows
    }
}

// Rows per block and blocks per SM of update_fp64_kernel.  Bound by the FP64 pipe (64% busy in
// 3D, 2,340 operations per node), the latency of its chains and instruction fetch (3,400
// instructions in a straight line, so that warps of one block, which run close together, share
// fetches).  3D takes 16 warps per SM as two blocks (128x256x128: 876 us per step with
// phase_kernel; four blocks of 4 rows 900, three with 168 registers 913, five 1039; three passes
// of one loop over the transforms 911 to 935); 2D takes 20 warps (512x2048: 117 us, with 16 125).
template <int DIM>
struct ShapeFp64 {
    static constexpr int kRows = DIM == 3 ? 8 : 4, kBlocks = DIM == 3 ? 2 : 5;
};
// The FP64 update, c read through L1.  g is pulled once the new velocity is known, so that its
// 19 values are not live through the force.
template <int DIM, class PR, bool kOpen, bool kMon>
__global__ void __launch_bounds__((32 * ShapeFp64<DIM>::kRows), (ShapeFp64<DIM>::kBlocks))
    update_fp64_kernel(StepArgs<PR> a, PullPtrs<DIM, PR> ptr) {
    using L = Lat<DIM>;
    constexpr int Q = L::Q;
    const Geom& g = a.g;
    const Codec<PR> cd(a.pop_scale);
    const int tx = threadIdx.x, x0 = 1 + (int)blockIdx.x * 32, x = x0 + tx, y = 1 + (int)(blockIdx.y * blockDim.y + threadIdx.y);
    const int z = DIM == 3 ? g.zlo + (int)(gridDim.z - 1 - blockIdx.z) : 0;
    double mon[2] = {0.0, 0.0};
    if (x <= g.n[0] && y <= g.n[1]) {
        const unsigned self = nidx32(g, x, y, z), mask = cross_mask<DIM>(g, x, y, z);
        const Column<DIM, false> col(g, x, y, z);
        const bool fast = !__any_sync(__activemask(), col.general);
        double fpost[Q];
        if (fast) {
            pull_column(g, col, self, fpost, [&](int q, unsigned i) { return ptr.f_from(q, i); }, [&](auto* p) { return cd.load_f(p); });
        } else {
            pull_f<DIM, PR, kOpen>(a.fin, cd, g, x, y, z, self, mask, fpost, a.par);
        }
        wait_for_predecessor();
        let_successor_start();
        const double* cw = a.cw;
        auto C = [&](int dx, int dy, int dz) {
            return cw[self + unsigned(dx) + unsigned(dy) * unsigned(g.sy) + (DIM == 3 ? unsigned(dz) * unsigned(g.sz) : 0u)];
        };
        double mu, dc[3] = {0.0, 0.0, 0.0};
        phase_stencil<DIM, PR>(a.pp, C, mu, dc);
        const double c = C(0, 0, 0);
        double gpost[Q];
        auto pull = [&]() {
            if (fast) {
                pull_column(g, col, self, gpost, [&](int q, unsigned i) { return ptr.g_from(q, i); }, [&](auto* p) { return cd.load_dev(p); });
            } else {
                double cold;
                pull_g<DIM, PR, kOpen>(a.gin, a.cin, cd, g, x, y, z, self, mask, gpost, cold, a.par);
                if (kOpen && g.fc[0]) store_open<DIM, PR>(g, a.par, x, y, z, fpost, [&](int q) { return gpost[q]; }, cold, c);
            }
        };
        update_exact<DIM, PR>(a, cd, self, fpost, pull, gpost, c, mu, dc, kMon ? mon : nullptr);
        if (kOpen && g.fc[0]) store_open_u<DIM, PR>(g, a.par, x, y, z, a.u, self);
    }
    if constexpr (kMon) store_monitor_row(a, tx, x0, y, z, mon);
}

}  // namespace clipb
