// gpe_split.cuh -- the FP32 split-scheme step (RelativisticGpeC15/GPUGrossPitaevskii_C15.cu:
// 90-155) on four planes of cells in a line.
//
// A half-step reads one half of every complex value (R and q_R, or I and q_I) and
// updates the other.  In the handle's layout the halves sit next to each other, so
// both travel whole over DRAM in both half-steps (96 bytes per node and step for the
// 72 that are read or written), the neighbours' records are scattered, and a node
// costs 131 instructions a warp (warps issue on 63 % of the cycles; C15 36^3 97 us per
// half-step, 0.35 of the copy peak).  Here R, I, q_R and q_I are planes of their own,
// 4 bytes per value.  The cells of the grid are numbered in one line, row after row and
// plane after plane, with one cell that stays zero between rows and one row of them
// between planes; the line is cut into groups of 32 cells, and node (edge) l of a
// group's cells is one run of 128 bytes.  A neighbour is a fixed number of cells along
// the line, a neighbour outside the grid reads a zero cell, and only the lanes on zero
// cells idle (5 % at 36^3).  A warp keeps one node and its two edges for the whole
// launch.  A call of 16 or more steps changes psi and q in and out.
#pragma once

namespace gpe {

// The planes of one half-step: the half that is read and the half that is updated.
struct SplitPlanes {
    const char* psi_rd;
    char* psi_wr;
    const char* q_rd;
    char* q_wr;
};

// Geometry of a plane of V values per cell.  Cell (x, y, z), each from -1, sits at
// ((z + 1) Yp + y + 1) Xp + x + 1 of the line: x = X of a row is x = -1 of the next.
struct LineGrid {
    uint32_t X, Y, Z, V;
    uint32_t Xp, Yp;      // cells from row to row, rows from plane to plane
    uint32_t g0, groups;  // the groups that hold interior cells
    size_t gb, bytes;     // bytes of a group and of the plane
};
inline LineGrid make_line_grid(const Grid& g, uint32_t V) {
    LineGrid G;
    G.X = g.X;
    G.Y = g.Y;
    G.Z = g.Z;
    G.V = V;
    G.Xp = g.X + 1;
    G.Yp = g.Y + 1;
    auto at = [&](uint64_t x, uint64_t y, uint64_t z) { return ((z + 1) * G.Yp + y + 1) * G.Xp + x + 1; };
    G.g0 = (uint32_t)(at(0, 0, 0) / 32);
    G.groups = (uint32_t)(at(G.X - 1, G.Y - 1, G.Z - 1) / 32) - G.g0 + 1;
    G.gb = (size_t)V * 128;
    G.bytes = (size_t)(at(G.X, G.Y, G.Z) / 32 + 1) * G.gb;
    return G;
}
// The cells of a line and the offsets from a cell to its neighbours' fit 32 bits.
inline bool line_fits(const LineGrid& G) {
    return (uint64_t)(G.Z + 2) * G.Yp * G.Xp + G.Xp + 64 <= (uint64_t)INT32_MAX &&
           ((uint64_t)(G.Yp + 1) * G.Xp / 32 + 3) * G.gb <= (uint64_t)INT32_MAX &&
           (uint64_t)G.groups * G.V <= (uint64_t)INT32_MAX;
}

// A lane's cell, stepped along the line without divisions; zero cells have x = X, y = Y
// or z outside 0 .. Z - 1.
struct LineWalk {
    uint32_t x, y, z, dx, dy, dz;
    // cell c of the line, `step` cells from one to the next
    __device__ __forceinline__ LineWalk(const LineGrid& G, uint32_t c, uint32_t step, FastDiv dXp, FastDiv dYp) {
        // c - 1 is ((z + 1) Yp + y + 1) Xp + x; from two planes further on, so that nothing is
        // negative (Yp >= 2)
        split(G, c + (G.Yp - 1) * G.Xp - 1, dXp, dYp, x, y, z);
        z -= 2;
        split(G, step, dXp, dYp, dx, dy, dz);
    }
    __device__ static __forceinline__ void split(const LineGrid& G, uint32_t c, FastDiv dXp, FastDiv dYp, uint32_t& x, uint32_t& y,
                                                 uint32_t& z) {
        const uint32_t r = fdiv(c, dXp);
        x = c - r * G.Xp;
        z = fdiv(r, dYp);
        y = r - z * G.Yp;
    }
    __device__ __forceinline__ void next(const LineGrid& G) {
        x += dx;
        y += dy;
        z += dz;
        if (x >= G.Xp) {
            x -= G.Xp;
            ++y;
        }
        if (y >= G.Yp) {
            y -= G.Yp;
            ++z;
        }
    }
    __device__ __forceinline__ bool inside(const LineGrid& G) const { return x < G.X && y < G.Y && z < G.Z; }
};

// One half-step, PART as in split_step_kernel and its arithmetic: PART 0 reads R, q_R and
// updates I, q_I; PART 1 the other way round.  tab: V*4 incidences (cells along the line,
// edge), E to-nodes (cells, node); from: E from-nodes; E = 2V.
//
// Bound by the loads' latency: C15 64^3 0.77 of the copy peak.  Against groups cut row by
// row (of 32, 16 or 8 cells, by the lanes left idle; 8-cell runs put four lines into a
// request, L1 88 %), a step in us: C15 20^3 23.6 -> 14.1, 32^3 64.2 / 64.2, 36^3 117 -> 94, 40^3
// 144 -> 127, 64^3 497 -> 492; BCC 30^3 8.5 -> 7.3, 64^3 41 -> 31, 96^3 149 -> 146.
template <int PART>
__global__ void __launch_bounds__(kIlPlainThreads, 8) line_split_kernel(StepArgs a, SplitPlanes p, LineGrid G, LineGrid Gq,
                                                                        const int2* tab, const int32_t* from, FastDiv dXp,
                                                                        FastDiv dYp) {
    const uint32_t V = G.V;
    const PhysR<float>& P = a.pf;
    const uint32_t sub = threadIdx.x & 31;
    const uint32_t warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
    const uint32_t u0 = fdiv(warp, a.divV), l = warp - u0 * V, du = fdiv(nwarps, a.divV);
    // value t.y of the cell t.x along the line from this lane's, from the group's first byte
    auto lane_off = [&](int2 t, const LineGrid& g) {
        const int c = (int)sub + t.x;
        return (c >> 5) * (int32_t)g.gb + t.y * 128 + (c & 31) * 4;
    };
    int32_t off[4], eto[2], efrom[2];
    float w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        off[k] = lane_off(tab[4 * l + k], Gq);
        w[k] = a.tab.inc_w32[4 * l + k];
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        eto[r] = lane_off(tab[4 * V + 2 * l + r], G);
        efrom[r] = from[2 * l + r] * 128 + (int32_t)sub * 4;
    }
    const float pos[3] = {a.tab.pos32[3 * l], a.tab.pos32[3 * l + 1], a.tab.pos32[3 * l + 2]};
    const int32_t own = (int32_t)l * 128 + (int32_t)sub * 4;
    const int32_t qown = (int32_t)l * 256 + (int32_t)sub * 4;   // edge 2l; edge 2l + 1 a run further
    auto ld = [](const char* q) { return *reinterpret_cast<const float*>(q); };
    LineWalk at(G, (G.g0 + u0) * 32 + sub, du * 32, dXp, dYp);
    size_t base = (size_t)(G.g0 + u0) * G.gb;
    after_previous_kernel<false>();
    for (uint32_t u = u0; u < G.groups; u += du, at.next(G), base += (size_t)du * G.gb) {
        if (!at.inside(G)) continue;
        const char *pr = p.psi_rd + base, *qr = p.q_rd + 2 * base;
        char *pw = p.psi_wr + base + own, *qw = p.q_wr + 2 * base + qown;
        // every load of the node and its two edges is in flight before the first use
        const float vr = ld(pr + own), vw = ld(pw);
        float qv[4], to[2], fr[2], qo[2], qn[2];
#pragma unroll
        for (int k = 0; k < 4; ++k) qv[k] = ld(qr + off[k]);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            to[r] = ld(pr + eto[r]);
            fr[r] = ld(pr + efrom[r]);
            qo[r] = ld(qr + qown + r * 128);
            qn[r] = ld(qw + r * 128);
        }
        float d1q = 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) d1q = fm(w[k], qv[k], d1q);
        float r3[3];
        node_pos(P, at.x, at.y, at.z, pos, r3);
        const Cx<float> v = PART == 0 ? cx<float>(vr, vw) : cx<float>(vw, vr);
        const float tp = fm(P.c0, norm_sq(v), trap<float>(P, r3));
        *reinterpret_cast<float*>(pw) = fm(PART == 0 ? -P.dt : P.dt, fm(tp, vr, -d1q), vw);
#pragma unroll
        for (int r = 0; r < 2; ++r)
            *reinterpret_cast<float*>(qw + r * 128) = fm(PART == 0 ? P.dts : -P.dts, qo[r] + (to[r] - fr[r]), qn[r]);
    }
}

template <int PART>
cudaError_t launch_line_split_p(const StepArgs& a, const SplitPlanes& p, const LineGrid& G, const LineGrid& Gq, const int32_t* tab,
                                cudaStream_t s) {
    static int occ = 0;
    if (occ == 0) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, line_split_kernel<PART>, (int)kIlPlainThreads, 0);
        if (occ < 1) occ = 1;
    }
    ILGrid W{};   // the line's groups as one row
    W.V = G.V;
    W.Y = W.Z = 1;
    W.GX = G.groups;
    W.cells = 32;
    const unsigned nb = il_wave(W, kIlPlainThreads, occ, UINT32_MAX);
    const uint32_t entries = 4 * G.V + Gq.V;
    return launch_overlapped(line_split_kernel<PART>, nb, kIlPlainThreads, 0, s, a, p, G, Gq, reinterpret_cast<const int2*>(tab),
                             tab + 2 * entries, make_fastdiv(G.Xp), make_fastdiv(G.Yp));
}

// One half-step (part 0 or 1) on the planes.
inline cudaError_t launch_line_split(const StepArgs& a, int part, const SplitPlanes& p, const LineGrid& G, const LineGrid& Gq,
                                     const int32_t* tab, cudaStream_t s) {
    if (Gq.V != 2 * G.V) return cudaErrorInvalidValue;
    return part ? launch_line_split_p<1>(a, p, G, Gq, tab, s) : launch_line_split_p<0>(a, p, G, Gq, tab, s);
}

// The handle's layout <-> planes, a tile of one group's 32 cells x kSplitTile values of a
// cell per pass through shared memory: contiguous complex values on the one side, runs of
// one half on the other.  aos: the slot's interior pointer; re, im: the planes.
constexpr uint32_t kSplitTile = 64;
template <bool TO_PLANES>
__global__ void __launch_bounds__(256) split_convert_kernel(char* aos, size_t pitch, size_t slice, uint32_t cell_bytes, char* re,
                                                            char* im, LineGrid G, uint32_t jtiles, uint32_t tiles, FastDiv djt,
                                                            FastDiv dXp, FastDiv dYp) {
    __shared__ float2 tile[32 * (kSplitTile + 1)];
    __shared__ char* cell[32];   // the cells' records, null for zero cells
    let_next_kernel_in();
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const uint32_t u = fdiv(t, djt), j0 = (t - u * jtiles) * kSplitTile;
        const uint32_t nj = min(kSplitTile, G.V - j0);
        if (threadIdx.x < 32) {
            const LineWalk at(G, (G.g0 + u) * 32 + threadIdx.x, 0, dXp, dYp);
            cell[threadIdx.x] = at.inside(G) ? aos + (size_t)at.z * slice + (size_t)at.y * pitch + (size_t)at.x * cell_bytes +
                                                   (size_t)j0 * 8
                                             : nullptr;
        }
        __syncthreads();
        const size_t base = (size_t)(G.g0 + u) * G.gb + (size_t)j0 * 128;
        if (TO_PLANES) {
            for (uint32_t i = threadIdx.x; i < 32 * nj; i += 256) {
                const uint32_t c = i / nj, j = i - c * nj;
                if (cell[c]) tile[c * (kSplitTile + 1) + j] = *reinterpret_cast<const float2*>(cell[c] + j * 8);
            }
            __syncthreads();
        }
        for (uint32_t i = threadIdx.x; i < nj * 32; i += 256) {
            const uint32_t j = i / 32, c = i & 31;
            if (!cell[c]) continue;
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
            for (uint32_t i = threadIdx.x; i < 32 * nj; i += 256) {
                const uint32_t c = i / nj, j = i - c * nj;
                if (cell[c]) *reinterpret_cast<float2*>(cell[c] + j * 8) = tile[c * (kSplitTile + 1) + j];
            }
            __syncthreads();
        }
    }
    after_previous_kernel<false>();   // see il_convert_kernel
}

// beside: as launch_il_convert.
inline cudaError_t launch_split_convert(char* aos, size_t pitch, size_t slice, uint32_t cell_bytes, char* re, char* im,
                                        const LineGrid& G, bool to_planes, bool beside, cudaStream_t s) {
    const uint32_t jtiles = (G.V + kSplitTile - 1) / kSplitTile;
    const uint64_t tiles = (uint64_t)G.groups * jtiles;
    if (tiles > 0xffffffffu) return cudaErrorInvalidValue;
    const unsigned nb = (unsigned)std::min<uint64_t>(tiles, (uint64_t)device_sm_count() * 8);
    const FastDiv djt = make_fastdiv(jtiles), dXp = make_fastdiv(G.Xp), dYp = make_fastdiv(G.Yp);
    auto k = to_planes ? split_convert_kernel<true> : split_convert_kernel<false>;
    if (beside)
        return launch_overlapped(k, nb, 256, 0, s, aos, pitch, slice, cell_bytes, re, im, G, jtiles, (uint32_t)tiles, djt, dXp, dYp);
    k<<<nb, 256, 0, s>>>(aos, pitch, slice, cell_bytes, re, im, G, jtiles, (uint32_t)tiles, djt, dXp, dYp);
    return cudaGetLastError();
}

}  // namespace gpe
