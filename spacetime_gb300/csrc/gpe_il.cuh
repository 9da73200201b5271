// gpe_il.cuh -- the cell-interleaved layout of FP32 states and its leapfrog step.
//
// Why this layout.  In the handle's own layout a node's record (C complex FP32
// values) follows the previous node's, so a warp of 32 consecutive nodes reads
// 32 records 8C bytes apart: each neighbour gather becomes two requests (16 + 8
// bytes for spin-1) whose lanes straddle several 128-byte lines, and the spin-1
// BCC step is bound by the L1 data stage (85 % busy) with DRAM at 57 %.  Here a
// warp takes one node l of 32 consecutive cells along x.  The lattice's stencil
// is the same in every cell, so node l's k-th neighbour in those cells is node l'
// of 32 consecutive cells shifted by (dx, dy, dz): with the layout of ILGrid
// (gpe_internal.h) every load and store of the step -- own record, old next
// record, the neighbours, the update -- is one contiguous 256-byte run per
// component, a single line pair per request.
//
// The handle's slots stay in the handle's layout; a multi-step call converts the
// two psi slots in (il_convert_kernel), steps in this layout and converts both
// back.  The arithmetic and its order are those of parabolic_node_t + node_finish,
// so the state after the steps is the one the gather kernels give.
#pragma once

namespace gpe {

__host__ __device__ inline size_t il_row(const ILGrid& G, uint32_t y, uint32_t z) {
    return ((size_t)(z + 1) * (G.Y + 2) + (y + 1)) * G.row;
}

// Handle layout <-> interleaved layout of the interior cells, one tile of KG
// consecutive groups' cells (TC = KG cells of a row, contiguous in the handle's
// layout) x JT complex values (j = l C + s) per pass, staged in shared memory (TC x
// (JT + 1) float2, the padding against bank conflicts) so that both sides are read
// and written in contiguous 16-byte runs.  The tile keeps a thread's share within
// kIlConvLoads 16-byte loads (for J = 36, spin-1 BCC, three groups of 32 cells: one
// group per pass left 2 loads per thread and ran at half the copy rate).  aos: the slot's interior pointer.  J = V C and JT are even (every
// lattice with 4 entries per node has an even node count), so a cell's values and
// the tiles start on 16-byte boundaries.  Each thread issues all its loads of a
// tile before it stores any of them.  The interleaved halo rows and padding cells
// are not touched.
constexpr uint32_t kIlConvThreads = 256;
constexpr uint32_t kIlConvLoads = 8;  // 16-byte loads per thread and tile: TC x JT <= 4096 values
template <bool TO_IL>
__global__ void __launch_bounds__(kIlConvThreads, 4) il_convert_kernel(char* aos, Grid g, char* il, ILGrid G, uint32_t JT,
                                                                    uint32_t KG, uint32_t GXT, uint32_t jtiles,
                                                                    uint32_t tiles, FastDiv djt, FastDiv dgx,
                                                                    FastDiv dy) {
    extern __shared__ float2 il_tile[];  // TC x (JT + 1)
    let_next_kernel_in();
    const uint32_t J = G.V * G.C;
    const uint32_t cells = G.cells;
    const uint32_t TC = KG * cells, htc = TC / 2;
    const uint32_t ld = JT + 1;
    for (uint32_t w = blockIdx.x; w < tiles; w += gridDim.x) {
        const uint32_t r1 = fdiv(w, djt);
        const uint32_t jt = w - r1 * jtiles;
        const uint32_t r2 = fdiv(r1, dgx);
        const uint32_t gxt = r1 - r2 * GXT;
        const uint32_t z = fdiv(r2, dy);
        const uint32_t y = r2 - z * G.Y;
        const uint32_t j0 = jt * JT;
        const uint32_t nj = min(JT, J - j0);   // even
        const uint32_t x0 = gxt * TC;
        const uint32_t nc = min(TC, G.X - x0);
        const uint32_t half = nj / 2;          // 16-byte runs per cell of the tile
        char* arow = aos + (size_t)z * g.slice + (size_t)y * g.pitch + (size_t)x0 * g.cell_bytes + (size_t)j0 * 8;
        // cell c of the tile: group gxt KG + c / cells, cell c % cells of it
        char* irow = il + il_row(G, y, z) + (size_t)gxt * KG * G.gb + (size_t)j0 * cells * 8;
        float4 buf[kIlConvLoads];
        if (TO_IL) {
            // cell-major 16-byte runs of the handle's layout
            const uint32_t n4 = nc * half;
#pragma unroll
            for (uint32_t k = 0; k < kIlConvLoads; ++k) {
                const uint32_t i = threadIdx.x + k * kIlConvThreads;
                if (i < n4) {
                    const uint32_t c = i / half, q = i - c * half;
                    buf[k] = __ldg(reinterpret_cast<const float4*>(arow + (size_t)c * g.cell_bytes + (size_t)q * 16));
                }
            }
#pragma unroll
            for (uint32_t k = 0; k < kIlConvLoads; ++k) {
                const uint32_t i = threadIdx.x + k * kIlConvThreads;
                if (i < n4) {
                    const uint32_t c = i / half, q = i - c * half;
                    il_tile[c * ld + 2 * q] = make_float2(buf[k].x, buf[k].y);
                    il_tile[c * ld + 2 * q + 1] = make_float2(buf[k].z, buf[k].w);
                }
            }
            __syncthreads();
            // value-major pairs of cells of the interleaved layout
#pragma unroll
            for (uint32_t k = 0; k < kIlConvLoads; ++k) {
                const uint32_t i = threadIdx.x + k * kIlConvThreads;
                const uint32_t jj = i / htc, c = 2 * (i % htc);
                if (jj < nj && c < nc) {
                    const uint32_t gl = c / cells, cl = c - gl * cells;
                    const float2 a = il_tile[c * ld + jj];
                    char* dst = irow + (size_t)gl * G.gb + ((size_t)jj * cells + cl) * 8;
                    if (c + 1 < nc) {
                        const float2 b = il_tile[(c + 1) * ld + jj];
                        *reinterpret_cast<float4*>(dst) = make_float4(a.x, a.y, b.x, b.y);
                    } else {
                        *reinterpret_cast<float2*>(dst) = a;
                    }
                }
            }
        } else {
#pragma unroll
            for (uint32_t k = 0; k < kIlConvLoads; ++k) {
                const uint32_t i = threadIdx.x + k * kIlConvThreads;
                const uint32_t jj = i / htc, c = 2 * (i % htc);
                if (jj < nj && c < nc) {
                    const uint32_t gl = c / cells, cl = c - gl * cells;
                    buf[k] = __ldg(reinterpret_cast<const float4*>(irow + (size_t)gl * G.gb + ((size_t)jj * cells + cl) * 8));
                }
            }
#pragma unroll
            for (uint32_t k = 0; k < kIlConvLoads; ++k) {
                const uint32_t i = threadIdx.x + k * kIlConvThreads;
                const uint32_t jj = i / htc, c = 2 * (i % htc);
                if (jj < nj && c < nc) {
                    il_tile[c * ld + jj] = make_float2(buf[k].x, buf[k].y);
                    if (c + 1 < nc) il_tile[(c + 1) * ld + jj] = make_float2(buf[k].z, buf[k].w);
                }
            }
            __syncthreads();
            const uint32_t n4 = nc * half;
#pragma unroll
            for (uint32_t k = 0; k < kIlConvLoads; ++k) {
                const uint32_t i = threadIdx.x + k * kIlConvThreads;
                if (i < n4) {
                    const uint32_t c = i / half, q = i - c * half;
                    const float2 a = il_tile[c * ld + 2 * q], b = il_tile[c * ld + 2 * q + 1];
                    *reinterpret_cast<float4*>(arow + (size_t)c * g.cell_bytes + (size_t)q * 16) = make_float4(a.x, a.y, b.x, b.y);
                }
            }
        }
        __syncthreads();
    }
    // a launch beside the one before it ends after that one, so that what follows may
    // count on both
    after_previous_kernel<false>();
}

// A neighbour in the interleaved layout, for cell `sub` of a group (the lane's cell in
// its group): node (or edge) `item` of the cells shifted by (dx, dy, dz), at a fixed
// byte offset from the group's base: the rows (dz, dy), the item's run, and sub + dx
// within the group or (first / last cell) the last / first cell of the group before /
// after it.
template <int CELLS>
__device__ __forceinline__ int32_t il_lane_off(const ILGrid& G, int dx, int dy, int dz, uint32_t item, uint32_t sub) {
    const int xl = (int)sub + dx;   // -1 .. CELLS
    const int64_t gshift = xl < 0 ? -1 : (xl >= CELLS ? 1 : 0);
    const int64_t cell = xl - gshift * (int64_t)CELLS;
    return (int32_t)(((int64_t)dz * (G.Y + 2) + dy) * (int64_t)G.row + (int64_t)item * (G.C * CELLS * 8) +
                     gshift * (int64_t)G.gb + cell * 8);
}

// Which of a lane's neighbours lie outside [0, X): only the cell x = 0 has some to the
// left and only x = X - 1 to the right, so one bit per neighbour for each side, fixed
// for the launch, that count in the first and the last group of a row.
struct ILEdge {
    uint32_t left, right;
    __device__ __forceinline__ ILEdge() : left(0), right(0) {}
    __device__ __forceinline__ void add(int k, int dx, bool first, bool last) {
        left |= (uint32_t)(dx < 0 && first) << k;
        right |= (uint32_t)(dx > 0 && last) << k;
    }
    __device__ __forceinline__ uint32_t outside(uint32_t gx, uint32_t GX) const {
        return (gx == 0 ? left : 0u) | (gx == GX - 1 ? right : 0u);
    }
};

// The group a lane works on: the q-th group of the rows row0 .. (counted row after
// row), as (gx, y, z), stepped through the rows without divisions: a warp's next task
// is a fixed number of groups further on.
template <int CELLS>
struct ILWalk {
    uint32_t q, gx, y, z;   // this task's group
    uint32_t dq, dgx, dy, dz;
    // warp task u (32 / CELLS groups) of `step` tasks apart
    __device__ __forceinline__ ILWalk(const ILGrid& G, uint32_t u, uint32_t step, uint32_t row0, FastDiv dGX, FastDiv dY) {
        constexpr uint32_t kWG = 32 / CELLS;
        q = kWG * u + (threadIdx.x & 31) / CELLS;
        const uint32_t r = fdiv(q, dGX), row = row0 + r;
        gx = q - r * G.GX;
        z = fdiv(row, dY);
        y = row - z * G.Y;
        dq = kWG * step;
        const uint32_t dr = fdiv(dq, dGX);
        dgx = dq - dr * G.GX;
        dz = fdiv(dr, dY);
        dy = dr - dz * G.Y;
    }
    __device__ __forceinline__ void next(const ILGrid& G) {
        q += dq;
        gx += dgx;
        y += dy;
        z += dz;
        if (gx >= G.GX) {
            gx -= G.GX;
            ++y;
        }
        if (y >= G.Y) {
            y -= G.Y;
            ++z;
        }
    }
    // byte offset of the group in its buffer (a plane of rows is below 2^31 bytes)
    __device__ __forceinline__ size_t base(const ILGrid& G) const {
        const uint32_t r = (z + 1) * (G.Y + 2) + (y + 1);
        return (size_t)r * (uint32_t)G.row + (size_t)gx * (uint32_t)G.gb;
    }
    // from the group's base to the first value of the plane's zero row y = -1
    __device__ __forceinline__ int32_t zero(const ILGrid& G) const {
        return -(int32_t)((y + 1) * (uint32_t)G.row + gx * (uint32_t)G.gb);
    }
};

// One lane's node of an interleaved leapfrog step, cell (x, y, z): next <- next + 2 dt
// (-i H prev), with the arithmetic and its order of parabolic_node_t + node_finish.
// prev, next: the group's base in the two buffers (old: in the buffer of the old next
// values, next itself unless the step goes out of place); own: the node's offset from it; off:
// its neighbours', those with their bit set in `outside` read the zero row at `zero`
// instead.  F: where the step's fields come from (P if null); oa: where the observables
// of prev go.  With a NormAcc for oa: an imaginary-time iteration (kModeItpNorm), next =
// prev - dt H prev with prev read times inv.
//
// What bounds the plain step is the latency of the loads and the instructions between
// them (spin-1 BCC 96^3: warps issue on 51 % of the cycles, on 63 % before the local terms
// were multiply-adds, DRAM at 75 %), so nothing is computed here that is the same for the
// whole launch or row.
template <int C, int D, int CELLS, class OA>
__device__ __forceinline__ void il_task(const PhysR<float>& P, const PhysR<float>* F, const char* prev, char* next,
                                        const char* old, uint32_t own, const int32_t* off, uint32_t outside, int32_t zero, const float* w,
                                        int nd, const float* pos, uint32_t x, uint32_t y, uint32_t z, OA* oa,
                                        float inv = 1.f) {
    constexpr bool kItp = std::is_same<OA, NormAcc<float>>::value;
    constexpr uint32_t kComp = CELLS * 8;   // bytes between a record's components
    Cx<float> prv[C], nv[C], H[C];
    const char* pp = prev + own;
    char* np = next + own;
#pragma unroll
    for (int s = 0; s < C; ++s) {
        prv[s] = ldc<float>(pp + s * kComp);
        if constexpr (!kItp) nv[s] = ldc<float>(old + own + s * kComp);
    }
    if constexpr (kItp) scale_record(prv, C, inv);
#pragma unroll
    for (int s = 0; s < C; ++s) H[s] = cx<float>(0.f, 0.f);
    // DEC Laplacian, sum_f w_f (psi_nb - psi) in entry order (Spin1GpeBCC.cu:835-865),
    // the loads of a group of 4 entries issued together
#pragma unroll
    for (int k0 = 0; k0 < D; k0 += 4) {
        if (k0 >= nd) break;
        Cx<float> v[4][C];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const char* p = prev + ((outside >> (k0 + k)) & 1 ? zero : off[k0 + k]);
#pragma unroll
            for (int s = 0; s < C; ++s) v[k][s] = ldc<float>(p + s * kComp);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if constexpr (kItp) scale_record(v[k], C, inv);
#pragma unroll
            for (int s = 0; s < C; ++s) add_scaled(H[s], w[k0 + k], v[k][s] - prv[s]);
        }
    }
    // local terms and the leapfrog update, as node_finish
    float rr[3];
    node_pos(P, x, y, z, pos, rr);
    const float pot = trap<float>(P, rr, F);
    if constexpr (kItp) {
        local_terms<float, C>(P, rr, pot, GPE_MODE_ITP, false, prv, H, F);
#pragma unroll
        for (int s = 0; s < C; ++s) {
            nv[s] = prv[s];
            add_scaled(nv[s], -P.dt, H[s]);
            stc<float>(np + s * kComp, nv[s]);
        }
        oa->template add<C>(nv);
    } else {
        local_terms<float, C>(P, rr, pot, GPE_MODE_LEAPFROG, false, prv, H, F);
        if constexpr (!std::is_same<OA, NoObs>::value) oa->template node<float, C>(P, rr, prv, H);
#pragma unroll
        for (int s = 0; s < C; ++s) {
            add_scaled(nv[s], 2.f * P.dt, cx<float>(H[s].y, -H[s].x));
            stc<float>(np + s * kComp, nv[s]);
        }
    }
}

// Warp tasks per node of an interleaved step (the grid's groups counted row after
// row, 32 / cells per warp task).
__host__ __device__ inline uint32_t il_warp_tasks(const ILGrid& G) {
    const uint32_t wg = 32 / G.cells;
    return (G.Y * G.Z * G.GX + wg - 1) / wg;
}

constexpr unsigned kIlPlainThreads = 128;
constexpr unsigned kIlObsThreads = 256;

// One FP32 leapfrog step in the interleaved layout: next <- next + 2 dt (-i H prev).
// D = 4: every node has 4 stencil entries (BCC, A15, C15, Z); D = 8: rows of 4 or 8
// entries (FCC's tetrahedra and octahedra).  Warp task t = u V + l: node l of the
// u-th group (or groups, ILWalk).  The grid's warp count is a multiple
// of V, so a warp keeps its node, and with it its entries and position, in
// registers; the row length is the same in every lane of a warp, so the second
// group of 4 entries is a uniform branch.  OBS: the observables of prev are summed
// on the way (ObsAcc, as the gather kernels' observed step).  MODE kModeItpNorm: an
// imaginary-time iteration instead; kModeLeapfrogFrom: the old next values are read
// from a.hpsi and stay as they were.
template <int C, int D, int CELLS, bool OBS, int MODE = GPE_MODE_LEAPFROG>
__device__ __forceinline__ void il_step_body(const StepArgs& a, const ILGrid& G, FastDiv dGX) {
    static_assert(D == 4 || D == 8, "rows of 4, or of 4 and 8 entries");
    const PhysR<float>& P = make_phys<float>(a);
    using OA = typename AccOf<MODE, OBS, float>::type;
    __shared__ double obs_sums[OBS ? kObsSums * 256 : 1];
    OA oa = AccOf<MODE, OBS, float>::make(obs_sums);
    const uint32_t sub = threadIdx.x & (CELLS - 1);
    const uint32_t warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
    const uint32_t u0 = fdiv(warp, a.divV), l = warp - u0 * G.V;
    const uint32_t nq = G.Y * G.Z * G.GX;
    // the warp's node's table, read once from global memory (no shared tables: the
    // block then needs no shared memory, which left the plain kernel at 7 blocks per
    // SM); weights h / bs^2 of the step's block scale, as load_tables scales them
    const int f0 = a.tab.row_ptr[l];
    const int nd = D == 4 ? 4 : a.tab.row_ptr[l + 1] - f0;   // 4 or 8, the same in the whole warp
    int32_t off[D];
    float w[D];
    ILEdge edge;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        off[k] = 0;
        w[k] = 0.f;
        if (k < nd) {
            const int4 e = a.tab.ent4[f0 + k];
            off[k] = il_lane_off<CELLS>(G, e.x, e.y, e.z, (uint32_t)e.w, sub);
            w[k] = a.tab.w32[f0 + k] * P.ks;
            edge.add(k, e.x, sub == 0, sub == (G.X - 1) % CELLS);
        }
    }
    const float pos[3] = {a.tab.pos32[3 * l], a.tab.pos32[3 * l + 1], a.tab.pos32[3 * l + 2]};
    const uint32_t own = l * (C * CELLS * 8) + sub * 8;
    after_previous_kernel<false>();
    const float inv = MODE == kModeItpNorm && a.scale_in ? a.scale_in->inv : 1.f;
    // the grid's warp count is a multiple of V
    for (ILWalk<CELLS> g(G, u0, fdiv(nwarps, a.divV), 0, dGX, a.divY); g.q < nq; g.next(G)) {
        const uint32_t x = g.gx * CELLS + sub;
        if (x >= G.X) continue;
        const size_t base = g.base(G);
        const char* old = MODE == kModeLeapfrogFrom ? a.hpsi + base : a.next + base;
        il_task<C, D, CELLS, OA>(P, nullptr, a.prev + base, a.next + base, old, own, off, edge.outside(g.gx, G.GX), g.zero(G), w,
                                 nd, pos, x, g.y, g.z, &oa, inv);
    }
    if constexpr (OBS) {
        __shared__ double red[8][OBS_COUNT];
        oa.block_reduce(red, a.partials);
    }
    if constexpr (MODE == kModeItpNorm) {
        __shared__ double nred[kIlPlainThreads / 32];
        oa.finish(nred, a.partials, a.dv, a.scale_out);
    }
}

// Launch shapes: the plain step in blocks of kIlPlainThreads with at least
// IlBounds<C>::kMin of them per SM (the register cap that keeps the most warps in
// flight without spills), the observed step in blocks of 256 (its FP64 sums take
// shared memory per thread).
template <int C, int D>
struct IlBounds {
    // D = 4: spin-1 BCC 96^3 at 7 blocks (72 registers) 0.125 ms per step, at 8 (64)
    // 0.132; spin-2 BCC 64^3 at 5 blocks (96) 0.065 ms, at 6 (80) 0.067.  D = 8 keeps
    // 12 more registers for the second group of entries: spin-1 FCC 64^3 at 6 blocks
    // (80) 0.0563 ms, at 5 (96) 0.0595; spin-2 at 4 blocks (128).
    static constexpr int kMin = D == 8 ? (C == 5 ? 4 : (C == 3 ? 6 : 8)) : (C == 5 ? 5 : (C == 3 ? 7 : 8));
    static constexpr int kMinObs = (C == 5 || (C == 3 && D == 8)) ? 2 : 3;
};

template <int C, int D, int CELLS>
__global__ void __launch_bounds__(kIlPlainThreads, IlBounds<C, D>::kMin) il_step_kernel(StepArgs a, ILGrid G,
                                                                                    FastDiv dGX) {
    il_step_body<C, D, CELLS, false>(a, G, dGX);
}
template <int C, int D, int CELLS>
__global__ void __launch_bounds__(kIlObsThreads, IlBounds<C, D>::kMinObs) il_step_obs_kernel(StepArgs a, ILGrid G,
                                                                                        FastDiv dGX) {
    il_step_body<C, D, CELLS, true>(a, G, dGX);
}

// One imaginary-time iteration of gpe_itp before its last: next = prev - dt H prev
// with prev read times the factor of the normalisation before (a.scale_in), the sum
// |next|^2 and the next factor left in a.scale_out.  Reads prev and writes next, 16 C
// bytes per site, where the separate step, norm and scale passes of the handle's
// layout move 48 C.
template <int C, int D, int CELLS>
__global__ void __launch_bounds__(kIlPlainThreads, IlBounds<C, D>::kMin) il_itp_kernel(StepArgs a, ILGrid G,
                                                                                   FastDiv dGX) {
    il_step_body<C, D, CELLS, false, kModeItpNorm>(a, G, dGX);
}

// The leapfrog step out of place (the adjoint's checkpoints and recomputed states).
template <int C, int D, int CELLS>
__global__ void __launch_bounds__(kIlPlainThreads, IlBounds<C, D>::kMin) il_step_from_kernel(StepArgs a, ILGrid G,
                                                                                         FastDiv dGX) {
    il_step_body<C, D, CELLS, false, kModeLeapfrogFrom>(a, G, dGX);
}

// Blocks of one interleaved step (rows of D entries at most): one wave at the
// kernel's occupancy or one warp per task if that is fewer, as a multiple of m =
// V / gcd(V, warps per block) (the grid's warp count a multiple of V), and at most
// `max_blocks` (the handle's partial-sum rows); 0 if no such grid.
inline unsigned il_wave(const ILGrid& G, unsigned threads, int occ, size_t max_blocks) {
    const unsigned wpb = threads / 32;
    uint32_t gv = G.V, gb = wpb;
    while (gb) {
        const uint32_t r = gv % gb;
        gv = gb;
        gb = r;
    }
    const uint64_t m = G.V / gv;
    const uint64_t tasks = (uint64_t)il_warp_tasks(G) * G.V;
    uint64_t nb = std::min<uint64_t>((uint64_t)occ * (unsigned)device_sm_count(), (tasks + wpb - 1) / wpb);
    // rounded down (a block past the wave would start only when another ends);
    // grids of fewer tasks than m blocks' warps take m blocks, some warps idle
    nb = nb >= m ? nb / m * m : m;
    if (nb > max_blocks) nb = max_blocks / m * m;
    return (unsigned)nb;
}

template <int C, int D, int CELLS>
unsigned il_blocks_d(const ILGrid& G, bool obs, size_t max_blocks) {
    static int occ[2] = {0, 0};
    const unsigned threads = obs ? kIlObsThreads : kIlPlainThreads;
    int& o = occ[obs ? 1 : 0];
    if (o == 0) {
        auto k = obs ? il_step_obs_kernel<C, D, CELLS> : il_step_kernel<C, D, CELLS>;
        cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, obs ? 50 : 0);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k, (int)threads, 0);
        if (o < 1) o = 1;
    }
    return il_wave(G, threads, o, max_blocks);
}

// f(<cells of a group>, <entries of a row>) as compile-time constants; bad where the
// kernels have no such form.
template <class T, class F>
T il_form(const ILGrid& G, int deg, T bad, F f) {
    auto with = [&](auto cells) {
        if (deg == 4) return f(cells, std::integral_constant<int, 4>());
        if (deg == 8) return f(cells, std::integral_constant<int, 8>());
        return bad;
    };
    if (G.cells == 32) return with(std::integral_constant<int, 32>());
    if (G.cells == 16) return with(std::integral_constant<int, 16>());
    if (G.cells == 8) return with(std::integral_constant<int, 8>());
    return bad;
}

template <int C>
unsigned il_blocks(const ILGrid& G, int deg, bool obs, size_t max_blocks) {
    return il_form(G, deg, 0u, [&](auto cells, auto d) { return il_blocks_d<C, d(), cells()>(G, obs, max_blocks); });
}

// One interleaved leapfrog step (a.prev / a.next: interleaved buffers) on rows of
// at most deg (4 or 8) entries; obs: sum the observables of a.prev into a.partials
// and finalize them into out.
template <int C, int D, int CELLS>
cudaError_t launch_il_step_d(const StepArgs& a, const ILGrid& G, size_t max_blocks, bool obs, double* out, cudaStream_t s) {
    const unsigned nb = il_blocks_d<C, D, CELLS>(G, obs, max_blocks);
    if (nb == 0) return cudaErrorInvalidConfiguration;
    const FastDiv dGX = make_fastdiv(G.GX);
    if (obs) {
        il_step_obs_kernel<C, D, CELLS><<<nb, kIlObsThreads, 0, s>>>(a, G, dGX);
        finalize_observables(a.partials, nb, out, s);
    } else {
        return launch_overlapped(il_step_kernel<C, D, CELLS>, nb, kIlPlainThreads, 0, s, a, G, dGX);
    }
    return cudaGetLastError();
}

template <int C>
cudaError_t launch_il_step(const StepArgs& a, const ILGrid& G, int deg, size_t max_blocks, bool obs, double* out,
                           cudaStream_t s) {
    return il_form(G, deg, cudaErrorInvalidValue, [&](auto cells, auto d) {
        return launch_il_step_d<C, d(), cells()>(a, G, max_blocks, obs, out, s);
    });
}

template <int C, int D, int CELLS>
cudaError_t launch_il_step_from_d(const StepArgs& a, const ILGrid& G, size_t max_blocks, cudaStream_t s) {
    static int occ = 0;
    if (occ == 0) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, il_step_from_kernel<C, D, CELLS>, (int)kIlPlainThreads, 0);
        if (occ < 1) occ = 1;
    }
    const unsigned nb = il_wave(G, kIlPlainThreads, occ, max_blocks);
    if (nb == 0) return cudaErrorInvalidConfiguration;
    return launch_overlapped(il_step_from_kernel<C, D, CELLS>, nb, kIlPlainThreads, 0, s, a, G, make_fastdiv(G.GX));
}

// One leapfrog step next <- hpsi + F(prev) (interleaved buffers).
template <int C>
cudaError_t launch_il_step_from(const StepArgs& a, const ILGrid& G, int deg, size_t max_blocks, cudaStream_t s) {
    return il_form(G, deg, cudaErrorInvalidValue,
                   [&](auto cells, auto d) { return launch_il_step_from_d<C, d(), cells()>(a, G, max_blocks, s); });
}

template <int C, int D, int CELLS>
cudaError_t launch_il_itp_d(const StepArgs& a, const ILGrid& G, size_t max_blocks, cudaStream_t s) {
    static int occ = 0;
    if (occ == 0) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, il_itp_kernel<C, D, CELLS>, (int)kIlPlainThreads, 0);
        if (occ < 1) occ = 1;
    }
    const unsigned nb = il_wave(G, kIlPlainThreads, occ, max_blocks);
    if (nb == 0) return cudaErrorInvalidConfiguration;
    return launch_overlapped(il_itp_kernel<C, D, CELLS>, nb, kIlPlainThreads, 0, s, a, G, make_fastdiv(G.GX));
}

// One imaginary-time iteration (a.prev / a.next: interleaved buffers).
template <int C>
cudaError_t launch_il_itp(const StepArgs& a, const ILGrid& G, int deg, size_t max_blocks, cudaStream_t s) {
    return il_form(G, deg, cudaErrorInvalidValue,
                   [&](auto cells, auto d) { return launch_il_itp_d<C, d(), cells()>(a, G, max_blocks, s); });
}

#define GPE_INSTANTIATE_IL(C)                                                                                           \
    template cudaError_t launch_il_step<C>(const StepArgs&, const ILGrid&, int, size_t, bool, double*, cudaStream_t); \
    template cudaError_t launch_il_itp<C>(const StepArgs&, const ILGrid&, int, size_t, cudaStream_t);                 \
    template cudaError_t launch_il_step_from<C>(const StepArgs&, const ILGrid&, int, size_t, cudaStream_t);           \
    template unsigned il_blocks<C>(const ILGrid&, int, bool, size_t);                                                 \
    template cudaError_t launch_il_hyper<C>(const StepArgs&, const ILGrid&, const ILGrid&, const int32_t*, cudaStream_t);

// ---------------------------------------------- hyperbolic (psi + q) leapfrog

// The fused hyperbolic leapfrog step (update_psi + update_q of
// RelativisticSpin2Gpe.cu:1873-1874, both reading the previous (psi, q)) in the
// interleaved layout: psi in G (V nodes per cell), q in Gq (the E = 2V edges of a
// cell in place of the nodes).  A warp keeps node j and edges 2j, 2j + 1 for the
// whole launch (the grid's warp count is a multiple of V): warp task t = u V + j
// updates node j of the u-th group from its 4 incident edges (d1 q,
// RelativisticSpin2Gpe.cu:1051-1066), then its two edges from their nodes (d0 psi,
// :986-1019).  Every warp does the same work, so the warps that read a group's psi
// and q lines stay together (a warp per node or edge let the edge warps run ahead
// of the node warps, and spin-2 then read 48 % more from DRAM than the algorithmic
// bytes).  tab: the handle's interleaved offset tables (il_hyper_tables: V*4
// incidences relative to the q group base, E to-nodes relative to the psi group
// base, both with dx + 1 in the two low bits, and E from-nodes).  The arithmetic
// and its order are hyper_step_kernel's (fused leapfrog), so the states are its
// states bit for bit.  EDGES edges are loaded before the first of them is stored
// (IlHyperEdges).
template <int C, int CELLS, int EDGES>
__device__ __forceinline__ void il_hyper_body(const StepArgs& a, const ILGrid& G, const ILGrid& Gq, const int32_t* tab,
                                              FastDiv dGX) {
    const uint32_t V = G.V, E = Gq.V;
    const uint32_t sub = threadIdx.x & (CELLS - 1);
    const uint32_t warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
    const uint32_t u0 = fdiv(warp, a.divV), j = warp - u0 * V;
    const PhysR<float>& P = make_phys<float>(a);
    constexpr uint32_t kComp = CELLS * 8;
    const uint32_t nq = G.Y * G.Z * G.GX;
    // this lane's offsets (cell sub + dx, stepping into the next / previous group
    // where it leaves this one): the node's 4 incidences in q, its edges' to-nodes
    // in psi; the edges' from-nodes; the node's weights and position
    auto lane_off = [&](int32_t b, int32_t wrap) {
        const int xl = (int)sub + (b & 3) - 1;
        const int32_t gs = xl < 0 ? -1 : (xl >= CELLS ? 1 : 0);
        return (b & ~3) + (int32_t)sub * 8 + gs * wrap;
    };
    int32_t off[4], eto[2], efrom[2];
    float w[4];
    ILEdge edge;   // bits 0..3 the incidences, 4 and 5 the to-nodes
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int32_t b = tab[4 * j + k];
        off[k] = lane_off(b, (int32_t)Gq.gb - (int32_t)kComp);
        edge.add(k, (b & 3) - 1, sub == 0, sub == (G.X - 1) % CELLS);
        w[k] = a.tab.inc_w32[4 * j + k];
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int32_t b = tab[4 * V + 2 * j + r];
        eto[r] = lane_off(b, (int32_t)G.gb - (int32_t)kComp);
        edge.add(4 + r, (b & 3) - 1, sub == 0, sub == (G.X - 1) % CELLS);
        efrom[r] = tab[4 * V + E + 2 * j + r] + (int32_t)sub * 8;
    }
    const float pos[3] = {a.tab.pos32[3 * j], a.tab.pos32[3 * j + 1], a.tab.pos32[3 * j + 2]};
    const float dts = P.dts;
    for (ILWalk<CELLS> g(G, u0, fdiv(nwarps, a.divV), 0, dGX, a.divY); g.q < nq; g.next(G)) {
        const uint32_t x = g.gx * CELLS + sub, y = g.y, z = g.z;
        if (x >= G.X) continue;
        const size_t gbase = g.base(G), qbase = g.base(Gq);
        const uint32_t outside = edge.outside(g.gx, G.GX);
        {
            // node j
            const size_t own = gbase + (size_t)j * (C * kComp) + (size_t)sub * 8;
            Cx<float> prv[C], H[C], nv[C];
#pragma unroll
            for (int s = 0; s < C; ++s) {
                prv[s] = ldc_nc<float>(a.prev + own + s * kComp);
                nv[s] = ldc<float>(a.next + own + s * kComp);   // in flight with the q loads
            }
#pragma unroll
            for (int s = 0; s < C; ++s) H[s] = cx<float>(0.f, 0.f);
            Cx<float> qv[4][C];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const bool in = !((outside >> k) & 1);
                const char* p = a.q + qbase + off[k];
#pragma unroll
                for (int s = 0; s < C; ++s) qv[k][s] = in ? ldc_nc<float>(p + s * kComp) : cx<float>(0.f, 0.f);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
#pragma unroll
                for (int s = 0; s < C; ++s) add_scaled(H[s], w[k], qv[k][s]);
            }
            float r[3];
            node_pos(P, x, y, z, pos, r);
            const float pot = trap<float>(P, r);
            if constexpr (C == 1) {
                local_scalar<float>(P, pot, false, true, prv, H);
            } else if constexpr (C == 3) {
                local_spin1<float>(P, r, pot, true, false, true, prv, H);
            } else {
                local_spin2<float>(P, r, pot, true, false, true, prv, H);
            }
            // the leapfrog update, as write_update
#pragma unroll
            for (int s = 0; s < C; ++s) {
                add_scaled(nv[s], 2.f * P.dt, cx<float>(H[s].y, -H[s].x));
                stc<float>(a.next + own + s * kComp, nv[s]);
            }
        }
        // edges 2j and 2j + 1: q_update, hyperbolic leapfrog: next_q += i 2 (dt/sigma)(prev_q + d0 psi)
#pragma unroll 1
        for (int e0 = 0; e0 < 2; e0 += EDGES) {
            Cx<float> to[EDGES][C], fr[EDGES][C], pq[EDGES][C], v[EDGES][C];
#pragma unroll
            for (int i = 0; i < EDGES; ++i) {
                const int e = e0 + i;
                const size_t own = qbase + (size_t)(2 * j + e) * (C * kComp) + (size_t)sub * 8;
                const bool in = !((outside >> (4 + e)) & 1);
                const char* pt = a.prev + gbase + eto[e];
#pragma unroll
                for (int s = 0; s < C; ++s) {
                    to[i][s] = in ? ldc_nc<float>(pt + s * kComp) : cx<float>(0.f, 0.f);
                    fr[i][s] = ldc_nc<float>(a.prev + gbase + efrom[e] + s * kComp);
                    pq[i][s] = ldc_nc<float>(a.q + own + s * kComp);
                    v[i][s] = ldc<float>(a.qnext + own + s * kComp);
                }
            }
#pragma unroll
            for (int i = 0; i < EDGES; ++i) {
                const size_t own = qbase + (size_t)(2 * j + e0 + i) * (C * kComp) + (size_t)sub * 8;
#pragma unroll
                for (int s = 0; s < C; ++s) {
                    const Cx<float> d0psi = to[i][s] - fr[i][s];
                    const Cx<float> qq = pq[i][s] + d0psi;
                    add_scaled(v[i][s], 2.f * dts, cx<float>(-qq.y, qq.x));
                    stc<float>(a.qnext + own + s * kComp, v[i][s]);
                }
            }
        }
    }
}

// Register caps: spin-2 at 5 blocks of 128 threads (96 registers, no spills),
// spin-1 at 6 (80 registers).  At 6 blocks (80 registers) spin-2 is within 1 % on
// C15 40^3 and 48^3 and BCC 64^3 (0.545 / 0.544, 0.818 / 0.819, 0.172 / 0.170 ms), but on
// C15 128^3 (285 M sites) it fell from 0.87 to 0.73 of peak; spin-1 BCC 64^3 at 7
// blocks 0.109 ms, at 6 0.107.
template <int C>
struct IlHyperBounds {
    static constexpr int kMin = C == 5 ? 5 : (C == 3 ? 6 : 8);
};

// The edges of a node that are in flight together.  On small grids a step is one wave: the
// node's loads, then each edge's behind the store before it, and both edges at once take a
// round trip off that (spin-1 BCC 8^3 4.8 -> 4.3 us a step, 6^3 6.3 -> 4.3, scalar C15 5^3 6.4 -> 4.3;
// such steps follow each other in quanta of 2 us).  On large ones it is more bytes in flight:
// scalar BCC 64^3 57.7 -> 50.1 us, C15 40^3 144 -> 131, spin-1 BCC 64^3 120 -> 116, C15 32^3 156 -> 152.
// Not where spin-1 groups are of 8 cells and the state is beyond il_cost8's line, whose short
// runs C15 then reads 0.4 to 1.4 % slower (40^3 338 -> 340 us; 22-cell rows of 13 MB 9 %), and not
// for spin-2, whose records would not fit the registers.
template <int C>
struct IlHyperEdges {
    static constexpr int kMost = C <= 3 ? 2 : 1;
};

template <int C, int CELLS, int EDGES>
__global__ void __launch_bounds__(kIlPlainThreads, IlHyperBounds<C>::kMin)
    il_hyper_kernel(StepArgs a, ILGrid G, ILGrid Gq, const int32_t* tab, FastDiv dGX) {
    il_hyper_body<C, CELLS, EDGES>(a, G, Gq, tab, dGX);
}

template <int C, int CELLS, int EDGES>
unsigned il_hyper_blocks_c(const ILGrid& G, const ILGrid& Gq) {
    static int occ = 0;
    const unsigned wpb = kIlPlainThreads / 32;
    if (occ == 0) {
        cudaFuncSetAttribute(il_hyper_kernel<C, CELLS, EDGES>, cudaFuncAttributePreferredSharedMemoryCarveout, 25);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, il_hyper_kernel<C, CELLS, EDGES>, (int)kIlPlainThreads, 0);
        if (occ < 1) occ = 1;
    }
    const uint32_t items = G.V;
    uint32_t gv = items, gb = wpb;
    while (gb) {
        const uint32_t r = gv % gb;
        gv = gb;
        gb = r;
    }
    const uint64_t m = items / gv;
    const uint64_t tasks = (uint64_t)il_warp_tasks(G) * items;
    uint64_t nb = std::min<uint64_t>((uint64_t)occ * (unsigned)device_sm_count(), (tasks + wpb - 1) / wpb);
    nb = nb >= m ? nb / m * m : m;
    return (unsigned)nb;
}

// One fused hyperbolic leapfrog step in the interleaved layout (a.prev / a.next /
// a.q / a.qnext: interleaved buffers).
template <int C>
cudaError_t launch_il_hyper(const StepArgs& a, const ILGrid& G, const ILGrid& Gq, const int32_t* tab, cudaStream_t s) {
    const uint64_t tasks64 = (uint64_t)il_warp_tasks(G) * G.V;
    if (tasks64 > 0xffffffffu || G.cells != Gq.cells || G.GX != Gq.GX || Gq.V != 2 * G.V) return cudaErrorInvalidValue;
    const FastDiv dGX = make_fastdiv(G.GX);
    constexpr int kEdges = IlHyperEdges<C>::kMost;
    auto launch = [&](auto kernel, unsigned blocks) { kernel<<<blocks, kIlPlainThreads, 0, s>>>(a, G, Gq, tab, dGX); };
    switch (G.cells) {
        case 32: launch(il_hyper_kernel<C, 32, kEdges>, il_hyper_blocks_c<C, 32, kEdges>(G, Gq)); break;
        case 16: launch(il_hyper_kernel<C, 16, kEdges>, il_hyper_blocks_c<C, 16, kEdges>(G, Gq)); break;
        case 8:
            if (C == 3 && !hyper_state_in_l2((uint64_t)G.X * G.Y * G.Z * G.V * C * 8)) {
                launch(il_hyper_kernel<C, 8, C == 3 ? 1 : kEdges>, il_hyper_blocks_c<C, 8, C == 3 ? 1 : kEdges>(G, Gq));
            } else {
                launch(il_hyper_kernel<C, 8, kEdges>, il_hyper_blocks_c<C, 8, kEdges>(G, Gq));
            }
            break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

// The tile of a layout change: KG groups x JT values with as few idle slots of the
// threads' loads as can be (kIlConvLoads each, and 1024 cells): whole rows of cells
// where they fit, runs of at least 32 values (256 bytes of the handle's layout).  Taking
// as many groups as fit first left a row of five groups in tiles of four and one.
struct IlTile {
    uint32_t KG, JT;
};
inline IlTile il_convert_tile(const ILGrid& G) {
    const uint32_t J = G.V * G.C, most = 2 * kIlConvLoads * kIlConvThreads;
    IlTile best = {1, 2};
    uint64_t slots = ~0ull;
    for (uint32_t KG = 1; KG <= G.GX && KG * G.cells <= 1024; ++KG) {
        uint32_t JT = std::min(J, most / (KG * G.cells) & ~1u);
        if (JT < std::min(J, 32u)) break;
        const uint32_t jt = (J + JT - 1) / JT, gt = (G.GX + KG - 1) / KG;
        if (jt > 1) JT = ((J + jt - 1) / jt + 1) & ~1u;
        const uint32_t k = (G.GX + gt - 1) / gt;
        const uint64_t n = (uint64_t)jt * gt;
        if (n <= slots) {
            slots = n;
            best = {k, JT};
        }
    }
    return best;
}

// Both directions of the layout change for one state buffer (interior pointer aos).
// beside: the launch may run beside the layout change launched before it, of other
// buffers (a change of a small state is as long as its launch's ramp and tail).
// Defined once (GPE_DEFINE_IL_CONVERT in one translation unit).
cudaError_t launch_il_convert(char* aos, const Grid& g, char* il, const ILGrid& G, bool to_il, bool beside, cudaStream_t s);

#define GPE_DEFINE_IL_CONVERT                                                                                        \
    cudaError_t launch_il_convert(char* aos, const Grid& g, char* il, const ILGrid& G, bool to_il, bool beside,      \
                                  cudaStream_t s) {                                                                  \
        const uint32_t J = G.V * G.C;                                                                                \
        if (J % 2 || g.cell_bytes != J * 8) return cudaErrorInvalidValue;                                            \
        const IlTile t = il_convert_tile(G);                                                                         \
        const uint32_t JT = t.JT, KG = t.KG;                                                                         \
        const uint32_t jtiles = (J + JT - 1) / JT;                                                                   \
        const uint32_t GXT = (G.GX + KG - 1) / KG;                                                                   \
        const uint64_t tiles = (uint64_t)G.Y * G.Z * GXT * jtiles;                                                   \
        if (tiles == 0) return cudaSuccess;                                                                          \
        if (tiles > 0xffffffffu) return cudaErrorInvalidValue;                                                       \
        const size_t smem = (size_t)KG * G.cells * (JT + 1) * sizeof(float2);                                        \
        const unsigned nb = (unsigned)std::min<uint64_t>(tiles, (uint64_t)device_sm_count() * 8);                    \
        const FastDiv djt = make_fastdiv(jtiles), dgx = make_fastdiv(GXT), dy = make_fastdiv(G.Y);                   \
        auto k = to_il ? il_convert_kernel<true> : il_convert_kernel<false>;                                         \
        if (beside)                                                                                                  \
            return launch_overlapped(k, nb, kIlConvThreads, smem, s, aos, g, il, G, JT, KG, GXT, jtiles,             \
                                     (uint32_t)tiles, djt, dgx, dy);                                                 \
        k<<<nb, kIlConvThreads, smem, s>>>(aos, g, il, G, JT, KG, GXT, jtiles, (uint32_t)tiles, djt, dgx, dy);       \
        return cudaGetLastError();                                                                                   \
    }

}  // namespace gpe
