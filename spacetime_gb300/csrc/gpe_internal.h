// gpe_internal.h -- shared host/device definitions of libgpe (not part of the ABI).
#pragma once

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <climits>
#include <cstdint>
#include <string>
#include <cuda_runtime.h>

#include "../../include/gpe.h"

namespace gpe {

// Largest tables the kernels stage in shared memory.  C15 (V=136, 544 stencil
// entries, E=272) is the largest lattice of the reference.
// Internal step mode beside GPE_MODE_LEAPFROG / EULER / ITP: a leapfrog step that
// reads the old value from StepArgs::hpsi and writes next, leaving the old buffer
// as it was (the adjoint's recomputation keeps every state of a segment).
constexpr int kModeLeapfrogFrom = 3;
// An imaginary-time step that also sums |next|^2 (ItpScale): the iterations of
// gpe_itp before its last.  FP32: prev is read times ItpScale::inv, so that the
// normalisation of the iteration before needs no pass of its own.
constexpr int kModeItpNorm = 4;

// The normalisation of one imaginary-time iterate: sum |psi|^2 over the nodes, the
// factor sqrt(sum dv) the state is divided by and (FP32 storage) its reciprocal
// rounded once; written by the last block of a NormAcc kernel (`count` blocks
// arrived so far, zero between launches).
struct ItpScale {
    double sum;
    double sq;
    float inv;
    uint32_t count;
};

constexpr int kMaxNodes = 160;
constexpr int kMaxEntries = 640;
constexpr int kMaxEdges = 320;
constexpr int kMaxFaces = 8;

// The items first, first + stride, ... below total, one thread's share of a grid.  A grid
// may have up to 2^32 - 1 sites, so a plain 32-bit index could step past 2^32 and start over
// in a loop that never ends; this one stops at total.
struct Strided {
    uint32_t i, stride, total;
    __host__ __device__ Strided(uint32_t first, uint32_t stride, uint32_t total) : i(first), stride(stride), total(total) {}
    __host__ __device__ bool more() const { return i < total; }
    __host__ __device__ void next() { i = stride < total - i ? i + stride : total; }
};

constexpr uint32_t kMostCells = 64;   // per column

// For a kernel of 256 threads a block (occ blocks per SM) whose threads walk up columns of up to
// kMostCells cells, and of which one block saturates an SM (the FP64 pipe's), so that an SM's
// blocks cost their sum: the cells per column that leave the busiest SM the least work, with what
// is done once per column counted as a quarter of a node.  A pass that only some of the blocks
// make (a last one, or the whole columns in it) costs an SM one block more than those blocks'
// share of the SMs from three quarters of an SM's on: the hardware does not deal blocks out in
// turn.  Measured, every choice is the fastest of all column lengths, or within 4 % of it.  A step
// in us, by the busiest thread's work and by the busiest SM's: spin-1 BCC 16^3 21.1 / 19.0, 20^3 36.2 /
// 26.6, 22^3 36.2 / 34.2, 24^3 51.5 / 41.8, 32^3 96.9 / 87.4; scalar 20^3 10.2 / 9.0; spin-2 20^3 65.7 /
// 49.4; C15 spin-1 9^3 36.7 / 27.2; cube 60^3 61.2 / 59.3; larger grids equal.
inline uint32_t cells_by_sm(uint64_t columns, uint32_t Z, uint64_t occ, uint64_t sms) {
    uint32_t zc = 1;
    uint64_t best = ~0ull;
    for (uint32_t c = (Z + kMostCells - 1) / kMostCells;;) {
        const uint32_t z = (Z + c - 1) / c, chunks = (Z + z - 1) / z, last = Z - (chunks - 1) * z;
        const uint64_t total = columns * chunks, whole = columns * (chunks - 1);   // items, those of z cells
        const uint64_t blocks = std::min((total + 255) / 256, occ * sms), pass = blocks * 256;
        const uint64_t per = (blocks + sms - 1) / sms, full = 4ull * z + 1, part = 4ull * last + 1;
        auto share = [&](uint64_t n) { return n == 0 ? 0 : std::min(per, (n + sms / 4) / sms + 1); };
        uint64_t cost = 0, at = 0;
        if (total > 8 * pass) {   // many passes: shorter columns in the last ones do not matter
            at = total / pass * pass;
            cost = total / pass * per * full;
        }
        for (; at < total; at += pass) {
            const uint64_t n = std::min(blocks, (total - at + 255) / 256);
            uint64_t busy = per, whole_busy = 0;
            if (n < blocks) {
                busy = share(n);
                whole_busy = at < whole ? share(std::min(n, (whole - at + 255) / 256)) : 0;
            } else {
                while (whole_busy < per && at + whole_busy * sms * 256 < whole) ++whole_busy;
            }
            cost += whole_busy * full + (busy - whole_busy) * part;
        }
        if (cost < best) {
            best = cost;
            zc = z;
        }
        if (z == 1) return zc;
        c = (Z + z - 2) / (z - 1);   // the next shorter columns
    }
}

// Unsigned division by a run-time constant: q = umulhi(n, mul) >> shift
// (Granlund & Montgomery, "Division by invariant integers using multiplication", 1994).
struct FastDiv {
    uint32_t d, mul, shift;
};

inline FastDiv make_fastdiv(uint32_t d) {
    FastDiv f;
    f.d = d;
    if (d == 1) {
        f.mul = 0;
        f.shift = 0;
        return f;
    }
    uint32_t l = 0;
    while ((1ull << l) < d) ++l;
    // mul = floor(2^32 * (2^l - d) / d) + 1, shift = l - 1 for the "add" variant; we use
    // the 64-bit form q = (umulhi(n, m) + n) >> l which is exact for all 32-bit n.
    uint64_t m = ((1ull << 32) * ((1ull << l) - d)) / d + 1;
    f.mul = (uint32_t)m;
    f.shift = l;
    return f;
}

#ifdef __CUDACC__
__device__ __forceinline__ uint32_t fdiv(uint32_t n, const FastDiv& f) {
    if (f.d == 1) return n;
    uint32_t t = __umulhi(n, f.mul);
    return (uint32_t)(((uint64_t)t + n) >> f.shift);
}
#endif

// Observables accumulated per block (FP64), in this order.
enum ObsIndex {
    OBS_NORM = 0,
    OBS_HEXP,
    OBS_EINT,
    OBS_MAGX,
    OBS_MAGY,
    OBS_MAGZ,
    OBS_SPIN,
    OBS_COMX,
    OBS_COMY,
    OBS_COMZ,
    OBS_MAXABS,
    OBS_NONFINITE,
    OBS_COUNT
};

// Geometry of one state buffer (bytes).
struct Grid {
    uint32_t X, Y, Z;
    uint32_t V, C, E;
    size_t pitch, slice;         // psi buffers
    size_t qpitch, qslice;       // q buffers
    uint32_t cell_bytes, qcell_bytes;
};

// Geometry of an FP32 state in the cell-interleaved layout.  Rows (y, z) run from
// -1 to Y and -1 to Z (the halo rows and planes are zero); a row holds GX groups of
// `cells` (32, 16 or 8) consecutive cells along x; a group holds [node l][component
// s][cell of the group][re, im], so that node l's component s of a group's cells
// is one contiguous run of 8 cells bytes.  Cells x >= X of the last group, and the
// cells x = -1 and x = X, read as zero.  A warp takes node l of 32 / cells groups,
// the grid's groups counted row after row.
struct ILGrid {
    uint32_t X, Y, Z, V, C, GX;
    uint32_t cells; // cells per group: 32, 16 or 8
    size_t gb;      // bytes per group: V * C * cells * 8
    size_t row;     // bytes per row: GX * gb
    size_t bytes;   // the buffer: (Y + 2) (Z + 2) rows
};

// The group width, per grid: narrow groups leave fewer lanes idle in a row's last
// group, but a warp's loads then fall into 2 (16 cells) or 4 (8 cells) shorter runs.
// What that costs where no lane is idle (FP32, one launch, 32 / 16 / 8 cells): spin-1
// BCC 96^3 124.7 / 129.2 / 141.6 us, A15 64^3 142.1 / 147.6 / 164.0; spin-2 BCC 64^3
// 64.9 / 67.2 / 68.9, C15 32^3 90.3 / 94.2 / 99.4; hyperbolic spin-2 BCC 64^3 171.9 /
// 174.1 / 180.5 -- taken as 3 % and 15 % (6 % for the spin-2's longer records) on the
// lanes' count.  Where lanes are idle: spin-1 C15 40^3 141.6 / 124.3 / 120.9, Z 40^3
// 85.9 / 75.9 / 71.6, BCC 72^3 67.3 / 62.6 / 63.6; hyperbolic spin-2 C15 40^3 620.5 /
// 545.4 / 501.3, 48^3 923.7 / 818.3 / 863.9.
// The hyperbolic step of spinors whose psi and q stay in L2 is bound by L1 requests, where the
// four lines of an 8-cell run count in full: below 9 MB a psi slot they are taken as 35 %, and
// only rows of less than half a group of 16 are cut in them.  A step in us, 8 cells / wider: spin-2 BCC
// 24^3 (6.6 MB) 12.3 / 10.3, 36 x 16 x 16 (4.4 MB) 10.2 / 9.0, C15 24 x 8 x 8 (8.4 MB) 14.3 / 12.3, spin-1 BCC 40 x 24 x 24
// (6.6 MB) 12.3 / 10.2; above, spin-2 BCC 20 x 32 x 32 (9.8 MB) 16.4 / 18.5, 23 x 32 x 32 (11.3 MB) 16.5 / 20.1,
// C15 36 x 8 x 8 (12.5 MB) 20.5 / 24.1, spin-1 BCC 20 x 48 x 48 (13.3 MB) 23.0 / 31.0; rows of 5 and 8 cells
// gain at any size (8.8 MB 14.3 / 24.6).  Scalars and the parabolic step (its launches overlap): no such
// loss.
inline bool hyper_state_in_l2(uint64_t slot_bytes) { return slot_bytes < 9000000; }
inline uint32_t il_cost8(uint32_t C, bool hyperbolic, uint64_t slot_bytes) {
    return hyperbolic && C > 1 && hyper_state_in_l2(slot_bytes) ? 135 : (C == 3 ? 115 : 106);
}
inline uint32_t il_group_cells(uint32_t X, uint32_t cost8) {
    auto cost = [X](uint32_t cells, uint32_t percent) { return (uint64_t)((X + cells - 1) / cells) * cells * percent; };
    uint32_t best = 32;
    if (cost(16, 103) < cost(32, 100)) best = 16;
    if (cost(8, cost8) < (best == 32 ? cost(32, 100) : cost(16, 103))) best = 8;
    return best;
}

// The interleaved kernels keep a neighbour's offset from its group's base in 32
// bits: a plane of rows and two groups more must stay below 2^31 bytes.
inline bool il_offsets_fit(const ILGrid& G) {
    return (uint64_t)(G.Y + 3) * G.row + 2 * (uint64_t)G.gb < (uint64_t)INT32_MAX;
}

inline ILGrid make_il_grid(const Grid& g, uint32_t cost8) {
    ILGrid G;
    G.X = g.X;
    G.Y = g.Y;
    G.Z = g.Z;
    G.V = g.V;
    G.C = g.C;
    G.cells = il_group_cells(g.X, cost8);
    G.GX = (g.X + G.cells - 1) / G.cells;
    G.gb = (size_t)g.V * g.C * G.cells * 8;
    G.row = G.GX * G.gb;
    G.bytes = (size_t)(g.Y + 2) * (g.Z + 2) * G.row;
    return G;
}

// Physics constants of a step (double; converted per kernel).
struct Phys {
    double p0[3];
    double bs;
    double bw[3];
    double dt;
    double lambda[3];
    double trap_offset;
    double trap_off_time;
    double c0, c2, c4, alpha, sigma;
    double quad_center[3];
    double ks;       // kinetic scale (bs0 / bs)^2 of the step's block scale bs (1 without expansion)
    int flags;
};

// Physics constants of a step in the arithmetic type of a kernel, prepared on the
// host so that kernels do no precision conversion (FP64 is slow on GB300).
template <typename R>
struct PhysR {
    R p0[3], bs, bw[3], lambda[3], trap_offset, c0, c2, c4, alpha, sigma, qc[3];
    R bq, bb[3], bqq, bbq[3];
    R dt, dts;       // dt and dt/sigma
    R ks;            // kinetic scale (bs0 / bs)^2; bs above is the step's block scale
    int trap_on;     // trap() is zero after trap_off_time (Spin1GpeBCC.cu:114)
    int flags;
};

// Per-handle device tables.  Byte offsets are relative to the base of the
// thread's own cell in the buffer being read.
struct DevTables {
    int32_t* row_ptr;     // V+1
    int32_t* nb_off;      // entries: byte offset of the neighbour value in prev
    int32_t* nb_soff;     // entries: offset inside a contiguous row of cells, INT32_MIN if the neighbour is off-row
    double* w64;          // entries: (-0.5*h)/bs^2
    float* w32;
    double* pos64;        // V*3
    float* pos32;
    int32_t* inc_off;     // V*F: byte offset of the incident edge value in q (relative to own q cell)
    double* inc_w64;      // V*F
    float* inc_w32;
    int32_t* e_from_off;  // E: byte offset of from-node in own psi cell
    int32_t* e_to_off;    // E: byte offset of to-node relative to own psi cell base
    int32_t* e_to_soff;   // E: the same inside a contiguous row of cells, INT32_MIN if off-row
    int32_t* inc_soff;    // V*F: incident edge inside a contiguous row of q cells, INT32_MIN if off-row
    int4* ent4;           // entries: (dx, dy, dz, node)
    int32_t* ent_row;     // entries: index of the (dy, dz) row in the multi-row tile
    int entries;
    int faces;
    int uniform_deg;      // > 0 when every node has the same number of entries
    int quad_rows;        // 1 when rows differ in length and every row is a positive multiple of 4 long
    int max_deg;          // the longest row
};

struct StepArgs {
    const char* prev;
    char* next;
    char* hpsi;
    const char* q;        // hyperbolic: q_prev
    char* qnext;          // hyperbolic: q_next
    Grid g;
    DevTables tab;
    Phys ph;
    gpe_fields B;
    double t;
    PhysR<float> pf;
    PhysR<double> pd;
    FastDiv divV, divRow, divY;   // nodes: within-row node index, X*V per row, rows
    FastDiv divE, divRowE;        // edges: within-row edge index, X*E per row
    uint32_t row_items;   // X*V
    uint32_t row_items_e; // X*E
    uint64_t total;       // total threads of work
    double* partials;     // observables
    double dv;            // bs0^3 VOLUME
    const ItpScale* scale_in;  // kModeItpNorm, FP32: the scale of prev (null: 1)
    ItpScale* scale_out;       // NormAcc kernels: the scale of what was summed
    int* err;             // device error flag (bounded waits that ran out)
};

#ifdef __CUDACC__
#define GPE_HD __host__ __device__
#else
#define GPE_HD
#endif

// getSignal + scaling (Spin1GpeBCC/AliceRingRamps.h:74-141): each channel walks its
// consecutive segment durations; inside segment k the value goes from the previous
// target (0 before the first) to target k by the segment's type; past the end the
// last target holds.  The same code runs on the host (gpe_ramp_eval) and on the
// device (batched stepping).  Segment counts must be in [0, GPE_RAMP_MAX_SEGMENTS].
GPE_HD inline void ramp_channel(int nseg, const double* tgt, int stride, const double* dur, const int32_t* type,
                                double tau, double* val, int dims) {
    for (int a = 0; a < dims; ++a) val[a] = 0;
    if (nseg <= 0) return;
    int k = 0;
    double t = tau;
    while (k < nseg && t - dur[k] >= 0) {
        t -= dur[k];
        ++k;
    }
    if (k == nseg) {
        k = nseg - 1;
        t = dur[k];
    }
    for (int a = 0; a < dims; ++a) {
        const double target = tgt[k * stride + a];
        const double prev = k > 0 ? tgt[(k - 1) * stride + a] : 0.0;
        if (type[k] == GPE_RAMP_CONSTANT) val[a] = target;
        else if (type[k] == GPE_RAMP_LINEAR) val[a] = prev + t * (target - prev) / dur[k];
        else val[a] = prev + (target - prev) * sqrt(t / dur[k]);
    }
}

GPE_HD inline void ramp_eval(const gpe_ramp& r, double tau, gpe_fields& out) {
    double bq = 0, bb[3];
    ramp_channel(r.bq_segments, r.bq_target, 1, r.bq_duration, r.bq_type, tau, &bq, 1);
    ramp_channel(r.bb_segments, &r.bb_target[0][0], 3, r.bb_duration, r.bb_type, tau, bb, 3);
    out.bq = r.bq_scale * bq;
    out.bq_quad = r.bq_quad_scale * bq;
    for (int a = 0; a < 3; ++a) {
        out.bb[a] = r.bb_scale * bb[a];
        out.bb_quad[a] = r.bb_quad_scale * bb[a];
    }
}

// Sets the text returned by gpe_last_error() for this thread (gpe_capi.cu).
void set_last_error(const std::string& msg);

}  // namespace gpe
