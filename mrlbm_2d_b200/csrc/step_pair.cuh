// step_pair.cuh -- two time steps for one read and one write of the populations.
//
// A single step moves 18 populations per node through HBM and computes for a third to a half of
// that time, so a large lattice is bound by memory traffic alone.  Here a warp carries the nodes of
// a strip of columns through two steps: it marches up the rows, computes level n + 1 of a row
// from level n in registers, hands the populations that cross columns to the neighbouring lanes by
// shuffles, keeps those that cross rows for one or two rows, and computes level n + 2 of the row
// below.  Level n + 1 never leaves the registers.  The strip's outer columns and the rows above and
// below its chunk are computed at level n + 1 only (again by the neighbouring warps).
//
// Nodes whose two steps are not plain (domain edges, the curved wall and what touches them) go
// through memory: an auxiliary launch computes level n + 1 of a band of nodes along the edges and
// around the cylinder into a buffer of its own, a second one steps the edge nodes, the wall nodes and
// the nodes next to them from that band.  Both run the single-step code (aux_item, finish), so every
// node's arithmetic is that of two single steps.
//
// Two launches per pair, ordered by programmatic dependent launch as in step_common.cuh:
//   * pair_first (level n + 1 of the band): waits for its predecessor in the stream, then allows the
//     second launch;
//   * pair_second: its wall and edge blocks, first in the grid, wait for pair_first to complete and
//     step to level n + 2; so do the blocks of the band's inner nodes, last in the grid, by when
//     pair_first is long done; the blocks between them are the two-step tiles, which read level n
//     only and do not wait (pair_first's predecessor had completed before this launch could start).
#pragma once
#include "step_pair.h"
#include "step_tma.cuh"

namespace mrlbm {

// The band of an auxiliary launch: rings of `w` nodes inside the edge rows and columns, and the
// rectangle x0.., y0.. of rw x rh nodes (clear of the rings).
struct PairBand { int w, x0, y0, rw, rh; };

__host__ __device__ inline int band_nodes(const PairBand& b, int nx, int ny) {
    return 2 * b.w * (nx - 2) + 2 * b.w * (ny - 2 - 2 * b.w) + b.rw * b.rh;
}

// `core`: at the first level, the nodes of the band that the second launch steps on (the innermost ring and
// the core); the field sums of the others are the two-step tiles'.
template <class Phys, bool FIRST>
__device__ __forceinline__ void band_node(const typename Phys::P& p, const PairBand& b, const PairRect& core, int q) {
    const int nx = p.L.nx, ny = p.L.ny, w = b.w;
    const int nrow = w * (nx - 2), ncol = w * (ny - 2 - 2 * w);
    int i, j;
    if (q < 2 * nrow) {
        const int side = q >= nrow, r = q - side * nrow, row = r / (nx - 2);
        i = 2 + (r - row * (nx - 2));
        j = side ? ny - 1 - row : 2 + row;
    } else if (q < 2 * (nrow + ncol)) {
        const int s = q - 2 * nrow, side = s >= ncol, r = s - side * ncol, row = r / w, c = r - row * w;
        i = side ? nx - 1 - c : 2 + c;
        j = 2 + w + row;
    } else {
        const int r = q - 2 * (nrow + ncol);
        if (r >= b.rw * b.rh) return;
        const int row = r / b.rw;
        i = b.x0 + (r - row * b.rw);
        j = b.y0 + row;
    }
    int cls = node_class(p, i, j);
    if (cls >= 0) return;                                        // curved-wall node: boundary blocks
    if (cls == CLS_SOLID && p.call && p.plot_every > 0 && (__ldg(p.call) + p.bstep + 1) % p.plot_every == 0)
        cls = CLS_SOLID_ZERO;
    typename Phys::T f[Q];
    gather_written(p, i, j, f);                                  // at the second level the other launch wrote it
    if (FIRST && p.fstat && i > 2 && i < nx - 1 && j > 2 && j < ny - 1 &&
        !(i >= core.x0 && i <= core.x1 && j >= core.y0 && j <= core.y1)) {
        typename Phys::P nosum = p;
        nosum.fstat = nullptr;
        Phys::finish(nosum, i, j, cls, f);
    } else {
        Phys::finish(p, i, j, cls, f);
    }
}

// Level n + 1 of the band: wall blocks, edge blocks, then the band's nodes, one thread each.
template <class Phys>
__global__ void __launch_bounds__(AUX_THREADS) pair_first(const __grid_constant__ typename Phys::P p,
                                                          const __grid_constant__ PairBand band, const PairRect core) {
    __shared__ __align__(16) unsigned char smem[aux_smem_bytes<typename Phys::T>()];
    const int b = (int)blockIdx.x, na = p.nbblk + p.neblk;
    if (b < na) {
        aux_item<Phys, true, true>(p, smem, b);
        return;
    }
    wait_prior_grid();
    band_node<Phys, true>(p, band, core, (b - na) * AUX_THREADS + (int)threadIdx.x);
}

// Shared-memory ring of a block of the two-step tiles: a slot holds one row of all nine planes, as
// wide as the block's strips and one column more on either side (a multiple of 16 bytes).  A row is
// one tensor copy (3-D map: columns, rows, planes; box COLS x 1 x 9): nine separate row copies cost
// the issuing warp about 800 ns a row, more than the arithmetic.
template <class T, int STRIPS, int STAGES>
struct PairRing {
    static constexpr int COLS = pair_box_cols(STRIPS);
    static constexpr int BYTES = Q * COLS * (int)sizeof(T);
    static constexpr int PITCH = (BYTES + 127) / 128 * 128 / (int)sizeof(T);   // elements between slots
    static_assert(COLS <= 256 && (COLS * (int)sizeof(T)) % 16 == 0 && (PAIR_COLS * STRIPS * (int)sizeof(T)) % 16 == 0,
                  "tensor copies");
    alignas(128) T row[STAGES][PITCH];
    alignas(8) uint64_t full[STAGES], empty[STAGES];
};

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
            smem_u32(dst)),
        "l"((unsigned long long)map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
        : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// One block's two-step tiles: WARPS * NS strips of columns, NS per warp (lane l of a warp has column l of
// each of its strips), over one chunk of rows of level n + 2.
template <class Phys, int WARPS, int NS, int STAGES, bool FULL>
__device__ __forceinline__ void pair_tile(const typename Phys::P& p, unsigned char* smem, const PairRect& core, int t, int strips,
                                          int chunks, int flip) {
    using T = typename Phys::T;
    using R = PairRing<T, WARPS * NS, STAGES>;
    using M = typename Phys::M;
    R& ring = *reinterpret_cast<R*>(smem);
    const int nx = p.L.nx, ny = p.L.ny, pitch = p.L.pitch, plane = (int)p.L.plane;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int bx = (strips + WARPS * NS - 1) / (WARPS * NS);
    int cy = t / bx;
    const int b0 = (t - cy * bx) * WARPS * NS, strip = b0 + warp * NS;
    if (flip) cy = chunks - 1 - cy;
    const int c0 = 1 + PAIR_COLS * b0;                     // first column of the ring's rows
    const int i = 2 + PAIR_COLS * strip + lane;            // this lane's column in the warp's first strip
    const int r0 = 3 + (int)((long long)(ny - 4) * cy / chunks), r1 = 2 + (int)((long long)(ny - 4) * (cy + 1) / chunks);
    const int nr = r1 - r0 + 3;                            // rows r0 - 1 .. r1 + 1 at level n + 1
    const bool core_rows = r0 >= core.y0 && r1 <= core.y1;
    // nothing of the block, or of this warp's strips, to store: all of it inside the cylinder's core
    if (core_rows && c0 + 2 >= core.x0 && c0 + 1 + PAIR_COLS * WARPS * NS <= core.x1) return;
    const int s0 = 3 + PAIR_COLS * strip, s1 = s0 + PAIR_COLS * NS - 1;
    const bool skip = strip >= strips || (core_rows && s0 >= core.x0 && s1 <= core.x1);
    // ring row t holds lattice row r0 - 2 + t of level n, t < nr + 2, in slot t % STAGES; row q of level
    // n + 1 pulls from ring rows q, q + 1 and q + 2
    auto issue = [&](int t) {
        uint64_t* bar = &ring.full[t % STAGES];
        mbar_expect_tx(bar, R::BYTES);
        tma_load_3d(&ring.row[t % STAGES][0], &p.tmap, bar, c0 + p.L.off, r0 - 2 + t, 0);
    };
    int sent = min(STAGES, nr + 2);
    if (threadIdx.x == 0) {
        for (int t = 0; t < STAGES; ++t) {
            mbar_init(&ring.full[t], 1);
            mbar_init(&ring.empty[t], WARPS);
        }
        fence_proxy_async();
        for (int t = 0; t < sent; ++t) issue(t);
    }
    __syncthreads();
    // the strips reach into the core's rows and columns (uniform across the warp)
    const bool meets = s1 >= core.x0 && s0 <= core.x1 && r1 >= core.y0 && r0 <= core.y1;
    bool own[NS], core_col[NS];
#pragma unroll
    for (int n = 0; n < NS; ++n) {
        const int c = i + n * PAIR_COLS;
        own[n] = lane > 0 && lane < 31 && c <= nx - 2;      // this lane stores its column of strip n
        core_col[n] = meets && c >= core.x0 && c <= core.x1;
    }
    T* d = p.dst + ((int64_t)(r0 - 2) * pitch + i + p.L.off);             // row r - 1 of the loop below
    const int at = 1 + PAIR_COLS * NS * warp + lane;                       // this lane's column in a ring row
    T h0[NS], h1[NS], h3[NS], h2[NS], h5[NS], h6[NS];                      // level n + 1 of row r - 1, moved along x
    T q2[NS], q5[NS], q6[NS];                                             // of row r - 2
    double hr[NS], hu[NS], hv[NS];                                        // FULL: rho, u, v of row r - 1 at level n + 1
#pragma unroll
    for (int n = 0; n < NS; ++n) h0[n] = h1[n] = h3[n] = h2[n] = h5[n] = h6[n] = q2[n] = q5[n] = q6[n] = T(0);
    bool low = false;
    bool dead = !mbar_wait(&ring.full[0], 0u) || !mbar_wait(&ring.full[1], 0u);
#pragma unroll 2
    for (int q = 0; q < nr; ++q) {
        const int r = r0 - 1 + q;
        if (warp == 0 && q >= 1 && sent < nr + 2) {        // ring row q - 1 is read: its slot takes row `sent`
            const int t = q - 1;
            if (!dead && !mbar_wait(&ring.empty[t % STAGES], (unsigned)(t / STAGES) & 1u)) dead = true;
            if (!dead) {
                if (lane == 0) {
                    fence_proxy_async();
                    issue(sent);
                }
                ++sent;
            }
        }
        if (!dead && !mbar_wait(&ring.full[(q + 2) % STAGES], (unsigned)((q + 2) / STAGES) & 1u)) dead = true;
        if (dead) break;
        T f[Q][NS];
#pragma unroll
        for (int k = 0; k < Q; ++k)
#pragma unroll
            for (int n = 0; n < NS; ++n)
                f[k][n] = ring.row[(q + 1 - ey(k)) % STAGES][k * R::COLS + at + n * PAIR_COLS - ex(k)];
        // Ring row q is not read again.  Its release must follow the arrival of the values, not just the issue
        // of the loads: a copy into the slot does overtake loads still under way (seen as a node wrong in
        // some hundreds of pairs).  The lane that releases it comes from a vote on the densities, which
        // need every lane's nine values; a warp that uses none of them may release at once.
        if (skip) {
            if (lane == 0) mbar_arrive(&ring.empty[q % STAGES]);
            continue;
        }
        T g[Q][NS];
        M m[NS];
        Phys::template plain<NS>(p, f, g, m);
        unsigned vote = 0;
#pragma unroll
        for (int n = 0; n < NS; ++n) vote ^= __ballot_sync(0xffffffffu, m[n].rho > T(0));
        if (lane == (int)(vote & 1u)) mbar_arrive(&ring.empty[q % STAGES]);
        T c1[NS], c3[NS], c5[NS], c6[NS], c7[NS], c8[NS];
#pragma unroll
        for (int n = 0; n < NS; ++n) {
            if (FULL && p.body && i + n * PAIR_COLS <= nx) {
                T fo[Q];
#pragma unroll
                for (int k = 0; k < Q; ++k) fo[k] = g[k][n];
                add_body_force(p, i + n * PAIR_COLS, r, fo);
#pragma unroll
                for (int k = 0; k < Q; ++k) g[k][n] = fo[k];
            }
            // the density of the rows beside the chunk and of the core is other blocks' to check
            low = low || (own[n] && !(m[n].rho > T(0)) && r >= r0 && r <= r1 && !(core_col[n] && r >= core.y0 && r <= core.y1));
        }
        const unsigned w = 0xffffffffu;
#pragma unroll
        for (int n = 0; n < NS; ++n) {
            c1[n] = __shfl_up_sync(w, g[1][n], 1);
            c3[n] = __shfl_down_sync(w, g[3][n], 1);
            c5[n] = __shfl_up_sync(w, g[5][n], 1);
            c6[n] = __shfl_down_sync(w, g[6][n], 1);
            c7[n] = __shfl_down_sync(w, g[7][n], 1);
            c8[n] = __shfl_up_sync(w, g[8][n], 1);
        }
        const int j = r - 1;                               // the row whose level n + 2 is now known
        if (q >= 2) {
            T fi[Q][NS], fo[Q][NS];
            M m2[NS];
#pragma unroll
            for (int n = 0; n < NS; ++n) {
                fi[0][n] = h0[n]; fi[1][n] = h1[n]; fi[2][n] = q2[n]; fi[3][n] = h3[n]; fi[4][n] = g[4][n];
                fi[5][n] = q5[n]; fi[6][n] = q6[n]; fi[7][n] = c7[n]; fi[8][n] = c8[n];
            }
            Phys::template plain<NS>(p, fi, fo, m2);
#pragma unroll
            for (int n = 0; n < NS; ++n) {
                if (own[n] && !(core_col[n] && j >= core.y0 && j <= core.y1)) {
                    low = low || !(m2[n].rho > T(0));
                    T out[Q];
#pragma unroll
                    for (int k = 0; k < Q; ++k) out[k] = fo[k][n];
                    if (FULL) {
                        const int c = i + n * PAIR_COLS;
                        if (p.body) add_body_force(p, c, j, out);
                        if (p.fstat) {                     // both steps' values on one read and write of the sums
                            FieldPre a;
                            fields_load(p, c, j, a);
                            fields_add(a, hr[n], hu[n], hv[n]);
                            fields_store(p, c, j, a, Phys::rho_of(m2[n]), (double)m2[n].ux, (double)m2[n].uy);
                        }
                    }
#pragma unroll
                    for (int k = 0; k < Q; ++k) d[k * plane + n * PAIR_COLS] = out[k];
                }
            }
        }
        d += pitch;
#pragma unroll
        for (int n = 0; n < NS; ++n) {
            q2[n] = h2[n]; q5[n] = h5[n]; q6[n] = h6[n];
            h0[n] = g[0][n]; h1[n] = c1[n]; h3[n] = c3[n]; h2[n] = g[2][n]; h5[n] = c5[n]; h6[n] = c6[n];
            if (FULL) { hr[n] = Phys::rho_of(m[n]); hu[n] = m[n].ux; hv[n] = m[n].uy; }
        }
    }
    if (low) flag_bad_density(p);
    if (dead) {
        // a wait gave up: report it, and let the copies in flight land before the block's shared memory
        // goes away (again bounded)
        if (lane == 0) atomicOr(p.errflag, ERR_TMA_TIMEOUT);
        if (warp == 0)
            for (int t = max(0, sent - STAGES); t < sent; ++t) (void)mbar_wait(&ring.full[t % STAGES], (unsigned)(t / STAGES) & 1u);
    }
}

// Level n + 2: p describes the second step (src: the band's buffer, tmap: level n).
template <class Phys, int WARPS, int NS, int STAGES, int MINB, bool FULL>
__global__ void __launch_bounds__(WARPS * 32, MINB) pair_second(const __grid_constant__ typename Phys::P p,
                                                                const __grid_constant__ PairBand band, const PairRect core,
                                                                const int strips, const int chunks, const int flip) {
    extern __shared__ __align__(128) unsigned char pair_smem[];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int na = p.nbblk + p.neblk, nt = (strips + WARPS * NS - 1) / (WARPS * NS) * chunks;
    const int b = (int)blockIdx.x;
    if (b >= na && b < na + nt) {
        pair_tile<Phys, WARPS, NS, STAGES, FULL>(p, pair_smem, core, b - na, strips, chunks, flip);
        return;
    }
    if (b < na) {
        aux_item<Phys, wide_wall<Phys>(WARPS * 32, MINB), true>(p, pair_smem, b);
        return;
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    band_node<Phys, false>(p, band, core, (b - na - nt) * WARPS * 32 + (int)threadIdx.x);
}

// Band of an auxiliary launch: rings of width w and the rectangle clipped clear of them.
inline PairBand pair_band(int w, const PairRect& r, int nx, int ny) {
    PairBand b{w, std::max(r.x0, 2 + w), std::max(r.y0, 2 + w), 0, 0};
    const int x1 = std::min(r.x1, nx - 1 - w), y1 = std::min(r.y1, ny - 1 - w);
    b.rw = std::max(0, x1 - b.x0 + 1);
    b.rh = std::max(0, y1 - b.y0 + 1);
    if (b.rw == 0 || b.rh == 0) b.rw = b.rh = 0;
    return b;
}

// FULL instantiations carry the field sums and the body force.
template <class Phys, bool FULL, int WARPS, int NS, int STAGES, int MINB>
int launch_pair(typename Phys::P p1, typename Phys::P p2, const PairPlan& plan, bool flip, cudaStream_t s) {
    using T = typename Phys::T;
    using R = PairRing<T, WARPS * NS, STAGES>;
    static_assert(WARPS * NS == (sizeof(T) == 8 ? PAIR_STRIPS64 : PAIR_STRIPS32), "the handle's tensor maps");
    static_assert((int)sizeof(R) >= aux_smem_bytes<T>(), "the auxiliary blocks' tables fit the ring");
    const int nx = p1.L.nx, ny = p1.L.ny;
    if (nx < PAIR_MIN_NX || ny < PAIR_MIN_NY || plan.chunks < 1 || plan.chunks > ny - 4) return -1;
    auto k = pair_second<Phys, WARPS, NS, STAGES, MINB, FULL>;
    static unsigned long long attr_set = 0;                // one bit per device
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 64 || !((attr_set >> dev) & 1ull)) {
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(R)) != cudaSuccess) return -1;
        if (dev < 64) attr_set |= 1ull << dev;
    }
    p1.nbblk = wall_blocks(p1.nb, AUX_THREADS, sizeof(T) == 8);
    p1.neblk = edge_blocks(p1, AUX_THREADS);
    const PairBand b1 = pair_band(2, plan.halo, nx, ny), b2 = pair_band(1, plan.core, nx, ny);
    const int n1 = p1.nbblk + p1.neblk + (band_nodes(b1, nx, ny) + AUX_THREADS - 1) / AUX_THREADS;
    if (launch_after_prior(pair_first<Phys>, (unsigned)n1, AUX_THREADS, 0, s, p1, b1, plan.core) != cudaSuccess) return -1;
    const int strips = (nx - 4 + PAIR_COLS - 1) / PAIR_COLS;
    p2.nbblk = wall_blocks(p2.nb, WARPS * 32, sizeof(T) == 8);
    p2.neblk = edge_blocks(p2, WARPS * 32);
    p2.tmap = p1.tmap;                                     // of level n
    const int n2 = p2.nbblk + p2.neblk + (strips + WARPS * NS - 1) / (WARPS * NS) * plan.chunks +
                   (band_nodes(b2, nx, ny) + WARPS * 32 - 1) / (WARPS * 32);
    return launch_after_prior(k, (unsigned)n2, WARPS * 32, sizeof(R), s, p2, b2, plan.core, strips, plan.chunks,
                              flip ? 1 : 0) == cudaSuccess
               ? 0
               : -1;
}

}  // namespace mrlbm
