// gpe_split.cuh -- the FP32 split-scheme step (RelativisticGpeC15/GPUGrossPitaevskii_C15.cu:
// 90-155) on four interleaved planes.
//
// A half-step reads one half of every complex value (R and q_R, or I and q_I) and
// updates the other.  In the handle's layout the halves sit next to each other, so
// both travel whole over DRAM in both half-steps (96 bytes per node and step for the
// 72 that are read or written), the neighbours' records are scattered, and a node
// costs 131 instructions a warp (warps issue on 63 % of the cycles; C15 36^3 97 us per
// half-step, 0.35 of the copy peak).  Here R, I, q_R and q_I are planes of their own in
// the layout of ILGrid, 4 bytes per value: node (edge) l of a group's 32, 16 or 8
// cells is one run, a warp keeps one node and its two edges for the whole launch, and
// every load is full.  A call of 16 or more steps changes psi and q in and out.
#pragma once

namespace gpe {

// The planes of one half-step: the half that is read and the half that is updated.
struct SplitPlanes {
    const char* psi_rd;
    char* psi_wr;
    const char* q_rd;
    char* q_wr;
};

// Geometry of one plane of V values per cell (ILGrid with 4-byte values).
inline ILGrid make_plane_grid(const Grid& g, uint32_t V) {
    ILGrid G;
    G.X = g.X;
    G.Y = g.Y;
    G.Z = g.Z;
    G.V = V;
    G.C = 1;
    // narrow groups cost what they cost spin-1 (C15 32^3, 32 / 16 / 8 cells: 64.5 / 67.3 / 74.5 us)
    G.cells = il_group_cells(g.X, 3);
    G.GX = (g.X + G.cells - 1) / G.cells;
    G.gb = (size_t)V * G.cells * 4;
    G.row = G.GX * G.gb;
    G.bytes = (size_t)(g.Y + 2) * (g.Z + 2) * G.row;
    return G;
}

// One half-step, PART as in split_step_kernel and its arithmetic: PART 0 reads R, q_R and
// updates I, q_I; PART 1 the other way round.  tab: V*4 incidences (byte offsets from a
// q group's base, for the group's first cell, dx + 1 in the two low bits), E to-nodes
// (likewise from a psi group's base) and E from-nodes, E = 2V.
//
// Groups of 32 cells: bound by latency (C15 32^3 64.5 us a step, 0.73 of the copy peak);
// of 8: by L1, whose every request then touches four lines (C15 36^3 118 us, L1 88 %, where
// 16 cells take 123 and 32 cells 154).  Two of a warp's groups in flight at a time gave
// 64.0 and 116; blocks per SM 6 / 7 / 8 / 10: 126 / 128 / 118 / 138.
template <int PART, int CELLS>
__global__ void __launch_bounds__(kIlPlainThreads, 8) il_split_kernel(StepArgs a, SplitPlanes p, ILGrid G, ILGrid Gq,
                                                                      const int32_t* tab, FastDiv dGX) {
    const uint32_t V = G.V, E = Gq.V;
    const PhysR<float>& P = a.pf;
    const uint32_t sub = threadIdx.x & (CELLS - 1);
    const uint32_t warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
    const uint32_t u0 = fdiv(warp, a.divV), l = warp - u0 * V;
    const uint32_t nq = G.Y * G.Z * G.GX;
    constexpr int32_t kRun = CELLS * 4;   // bytes of one node's run
    auto lane_off = [&](int32_t b, const ILGrid& g) {
        const int xl = (int)sub + (b & 3) - 1;
        const int32_t gs = xl < 0 ? -1 : (xl >= CELLS ? 1 : 0);
        return (b & ~3) + (int32_t)sub * 4 + gs * ((int32_t)g.gb - kRun);
    };
    int32_t off[4], eto[2], efrom[2];
    float w[4];
    ILEdge edge;   // bits 0..3 the incidences, 4 and 5 the to-nodes
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int32_t b = tab[4 * l + k];
        off[k] = lane_off(b, Gq);
        edge.add(k, (b & 3) - 1, sub == 0, sub == (G.X - 1) % CELLS);
        w[k] = a.tab.inc_w32[4 * l + k];
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int32_t b = tab[4 * V + 2 * l + r];
        eto[r] = lane_off(b, G);
        edge.add(4 + r, (b & 3) - 1, sub == 0, sub == (G.X - 1) % CELLS);
        efrom[r] = tab[4 * V + E + 2 * l + r] + (int32_t)sub * 4;
    }
    const float pos[3] = {a.tab.pos32[3 * l], a.tab.pos32[3 * l + 1], a.tab.pos32[3 * l + 2]};
    const int32_t own = (int32_t)l * kRun + (int32_t)sub * 4;
    const int32_t qown = 2 * (int32_t)l * kRun + (int32_t)sub * 4;   // edge 2l; edge 2l + 1 a run further
    auto ld = [](const char* q) { return *reinterpret_cast<const float*>(q); };
    after_previous_kernel<false>();
    for (ILWalk<CELLS> g(G, u0, fdiv(nwarps, a.divV), 0, dGX, a.divY); g.q < nq; g.next(G)) {
        const uint32_t x = g.gx * CELLS + sub;
        if (x >= G.X) continue;
        const size_t base = g.base(G), qbase = g.base(Gq);
        const uint32_t outside = edge.outside(g.gx, G.GX);
        const int32_t zero = g.zero(G), qzero = g.zero(Gq);
        const char *pr = p.psi_rd + base, *qr = p.q_rd + qbase;
        char *pw = p.psi_wr + base + own, *qw = p.q_wr + qbase + qown;
        // every load of the node and its two edges is in flight before the first use
        const float vr = ld(pr + own), vw = ld(pw);
        float qv[4], to[2], fr[2], qo[2], qn[2];
#pragma unroll
        for (int k = 0; k < 4; ++k) qv[k] = ld(qr + ((outside >> k) & 1 ? qzero : off[k]));
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            to[r] = ld(pr + ((outside >> (4 + r)) & 1 ? zero : eto[r]));
            fr[r] = ld(pr + efrom[r]);
            qo[r] = ld(qr + qown + r * kRun);
            qn[r] = ld(qw + r * kRun);
        }
        float d1q = 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) d1q = fm(w[k], qv[k], d1q);
        float r3[3];
        node_pos(P, x, g.y, g.z, pos, r3);
        const Cx<float> v = PART == 0 ? cx<float>(vr, vw) : cx<float>(vw, vr);
        const float tp = fm(P.c0, norm_sq(v), trap<float>(P, r3));
        *reinterpret_cast<float*>(pw) = fm(PART == 0 ? -P.dt : P.dt, fm(tp, vr, -d1q), vw);
#pragma unroll
        for (int r = 0; r < 2; ++r)
            *reinterpret_cast<float*>(qw + r * kRun) = fm(PART == 0 ? P.dts : -P.dts, qo[r] + (to[r] - fr[r]), qn[r]);
    }
}

template <int PART, int CELLS>
cudaError_t launch_il_split_p(const StepArgs& a, const SplitPlanes& p, const ILGrid& G, const ILGrid& Gq, const int32_t* tab,
                              cudaStream_t s) {
    static int occ = 0;
    if (occ == 0) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, il_split_kernel<PART, CELLS>, (int)kIlPlainThreads, 0);
        if (occ < 1) occ = 1;
    }
    const unsigned nb = il_wave(G, kIlPlainThreads, occ, UINT32_MAX);
    return launch_overlapped(il_split_kernel<PART, CELLS>, nb, kIlPlainThreads, 0, s, a, p, G, Gq, tab, make_fastdiv(G.GX));
}

// One half-step (part 0 or 1) on the planes.
inline cudaError_t launch_il_split(const StepArgs& a, int part, const SplitPlanes& p, const ILGrid& G, const ILGrid& Gq,
                                   const int32_t* tab, cudaStream_t s) {
    if (G.cells != Gq.cells || Gq.V != 2 * G.V) return cudaErrorInvalidValue;
    switch (G.cells) {
        case 32: return part ? launch_il_split_p<1, 32>(a, p, G, Gq, tab, s) : launch_il_split_p<0, 32>(a, p, G, Gq, tab, s);
        case 16: return part ? launch_il_split_p<1, 16>(a, p, G, Gq, tab, s) : launch_il_split_p<0, 16>(a, p, G, Gq, tab, s);
        case 8: return part ? launch_il_split_p<1, 8>(a, p, G, Gq, tab, s) : launch_il_split_p<0, 8>(a, p, G, Gq, tab, s);
        default: return cudaErrorInvalidValue;
    }
}

// The handle's layout <-> planes, a tile of one group's cells x kSplitTile values of a cell
// per pass through shared memory: contiguous complex values on the one side, runs of
// one half on the other.  aos: the slot's interior pointer; re, im: the planes.
constexpr uint32_t kSplitTile = 64;
template <bool TO_PLANES>
__global__ void __launch_bounds__(256) split_convert_kernel(char* aos, size_t pitch, size_t slice, uint32_t cell_bytes, char* re,
                                                            char* im, ILGrid G, uint32_t jtiles, uint32_t tiles, FastDiv djt,
                                                            FastDiv dgx, FastDiv dy) {
    __shared__ float2 tile[32 * (kSplitTile + 1)];
    let_next_kernel_in();
    const uint32_t cells = G.cells;
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const uint32_t r1 = fdiv(t, djt), j0 = (t - r1 * jtiles) * kSplitTile;
        const uint32_t r2 = fdiv(r1, dgx), gx = r1 - r2 * G.GX;
        const uint32_t z = fdiv(r2, dy), y = r2 - z * G.Y;
        const uint32_t nj = min(kSplitTile, G.V - j0), nc = min(cells, G.X - gx * cells);
        char* arow = aos + (size_t)z * slice + (size_t)y * pitch + (size_t)gx * cells * cell_bytes + (size_t)j0 * 8;
        const size_t base = il_row(G, y, z) + (size_t)gx * G.gb + (size_t)j0 * cells * 4;
        if (TO_PLANES) {
            for (uint32_t i = threadIdx.x; i < nc * nj; i += 256) {
                const uint32_t c = i / nj, j = i - c * nj;
                tile[c * (kSplitTile + 1) + j] = *reinterpret_cast<const float2*>(arow + (size_t)c * cell_bytes + j * 8);
            }
            __syncthreads();
        }
        for (uint32_t i = threadIdx.x; i < nj * cells; i += 256) {
            const uint32_t j = i / cells, c = i - j * cells;
            if (c >= nc) continue;
            float2& v = tile[c * (kSplitTile + 1) + j];
            float* pr = reinterpret_cast<float*>(re + base) + i;
            float* pi = reinterpret_cast<float*>(im + base) + i;
            if (TO_PLANES) {
                *pr = v.x;
                *pi = v.y;
            } else {
                v = make_float2(*pr, *pi);
            }
        }
        __syncthreads();
        if (!TO_PLANES) {
            for (uint32_t i = threadIdx.x; i < nc * nj; i += 256) {
                const uint32_t c = i / nj, j = i - c * nj;
                *reinterpret_cast<float2*>(arow + (size_t)c * cell_bytes + j * 8) = tile[c * (kSplitTile + 1) + j];
            }
            __syncthreads();
        }
    }
    after_previous_kernel<false>();   // see il_convert_kernel
}

// beside: as launch_il_convert.
inline cudaError_t launch_split_convert(char* aos, size_t pitch, size_t slice, uint32_t cell_bytes, char* re, char* im,
                                        const ILGrid& G, bool to_planes, bool beside, cudaStream_t s) {
    const uint32_t jtiles = (G.V + kSplitTile - 1) / kSplitTile;
    const uint64_t tiles = (uint64_t)G.Y * G.Z * G.GX * jtiles;
    if (tiles == 0) return cudaSuccess;
    if (tiles > 0xffffffffu) return cudaErrorInvalidValue;
    const unsigned nb = (unsigned)std::min<uint64_t>(tiles, (uint64_t)device_sm_count() * 8);
    const FastDiv djt = make_fastdiv(jtiles), dgx = make_fastdiv(G.GX), dy = make_fastdiv(G.Y);
    auto k = to_planes ? split_convert_kernel<true> : split_convert_kernel<false>;
    if (beside)
        return launch_overlapped(k, nb, 256, 0, s, aos, pitch, slice, cell_bytes, re, im, G, jtiles, (uint32_t)tiles, djt, dgx, dy);
    k<<<nb, 256, 0, s>>>(aos, pitch, slice, cell_bytes, re, im, G, jtiles, (uint32_t)tiles, djt, dgx, dy);
    return cudaGetLastError();
}

}  // namespace gpe
