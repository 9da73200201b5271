// gpe_observe.cuh -- the observables of a psi buffer and the integrated node fields
// with FP64-quality sums that spend next to no FP64 operation per node.
//
// GB300 runs one FP64 operation for every 64 FP32 ones, and a conversion from FP32
// costs as much as an FP64 operation: with per-node terms in FP64, observe_kernel
// spent 290 FP64 operations on a spin-1 node and ran at 87 % of the FP64 pipe with
// DRAM at 1 % (1463 us on spin-1 BCC 64^3, whose state is read in 11 us; this form
// takes 146 us, bound by the FP32 instructions of the exact sums).  Here
//  - everything that is the same for a column of cells -- the stencil weights, the
//    trap, the fields, the coupling constants, the position -- is left out of the
//    per-node terms and multiplied in once per column, in FP64;
//  - the per-node terms, products of stored values alone, are exact pairs of FP32
//    values for FP32 storage (two-products and two-sums: Dekker 1971, Knuth; the
//    sums are PairSum's and, for terms of one sign and for the products of a spin,
//    which cancel within a node of an unpolarised state, TripleSum's), plain FP64 for
//    FP64 storage.
// A pair keeps 47 bits or more of each node's term, and the errors of different nodes
// are independent, so that the sums carry the error of their FP64 additions.  (Densities
// in FP64 node by node instead of three FP32 words: observables, density and spin sums of
// that state together 487 us against 335; the spins' third words are 25 us more.)  Measured
// against sums in more than 64 bits on Thomas-Fermi clouds and noise (BCC 12^3 .. 24^3,
// C15 9^3; root mean square, relative): norm 1e-16 to 2.5e-16, centre of mass 1e-16 to
// 3e-16, energy 1e-16 to 3e-16, M_z 1e-16 to 2e-16, |F| 1e-16 -- observe_kernel's are 1e-16
// to 2.5e-16, 1e-16 to 2.5e-16, 1e-16 to 3e-16, 1e-16 to 6e-16 and 1e-16 (spin-1, whose sqrt2
// it takes from the reference's constant, 1e-15 to 3e-15).
#pragma once

namespace gpe {

__device__ __forceinline__ Pair operator+(Pair a, Pair b) {
    const Pair s = two_sum(a.h, b.h);
    return pair_norm(s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l)));
}
__device__ __forceinline__ Pair operator-(Pair a, Pair b) {
    b.h = -b.h;
    b.l = -b.l;
    return a + b;
}
__device__ __forceinline__ Pair operator*(Pair a, Pair b) {
    const Pair p = two_prod(a.h, b.h);
    return pair_norm(p.h, __fadd_rn(p.l, __fmaf_rn(a.h, b.l, __fmul_rn(a.l, b.h))));
}
__device__ __forceinline__ Pair twice(Pair a) {
    a.h = __fadd_rn(a.h, a.h);
    a.l = __fadd_rn(a.l, a.l);
    return a;
}
// a^2 with the term l^2, which a product of two pairs may leave out (its sign is random
// there) but which has the same sign in every square: 6e-16 of the sum of squares.  Half
// of it goes into h l, which is doubled exactly; added later it would fall to the rounding.
__device__ __forceinline__ Pair square(Pair a) {
    const Pair p = two_prod(a.h, a.h);
    const float hl = __fmaf_rn(a.l, a.h, __fmul_rn(__fmul_rn(0.5f, a.l), a.l));
    return pair_norm(p.h, __fmaf_rn(2.f, hl, p.l));
}
// sqrt(a) = s + d + d^2 / (2 sqrt(a)) + ..., s the correctly rounded root of the high word and
// d = (a - s^2) / (2 sqrt(a)).  With i = 1 / (2 sqrt(a.h)) for the reciprocal the terms of
// second order are i d (d - 2 i a.l): 5e-16 on average and always of one sign, so they are
// added before the rounding of d.
__device__ __forceinline__ Pair square_root(Pair a) {
    if (!(a.h > 0.f)) return Pair{a.h, 0.f};
    const float s = __fsqrt_rn(a.h), i = __fmul_rn(0.5f, rsqrtf(a.h));
    const float r = __fadd_rn(__fmaf_rn(-s, s, a.h), a.l);
    const float d = __fmul_rn(i, r);
    return pair_norm(s, __fmaf_rn(i, r, __fmul_rn(__fmul_rn(i, d), __fmaf_rn(-2.f * i, a.l, d))));
}
// sqrt(6) a: the constant in three parts, since two leave an error of 1e-15 that is the
// same for every node
__device__ __forceinline__ TripleSum times_sqrt6(const TripleSum& a) {
    constexpr double c = 2.449489742783178098;
    constexpr float c1 = (float)c, c2 = (float)(c - (double)c1), c3 = (float)(c - (double)c1 - (double)c2);
    TripleSum r(c1, a.h);
    const Pair p = two_prod(c1, a.l), q = two_prod(c2, a.h);
    r.add_low(p.h);
    r.add_low(q.h);
    r.m = __fadd_rn(r.m, __fadd_rn(__fadd_rn(p.l, q.l), __fmaf_rn(c3, a.h, __fmaf_rn(c2, a.l, __fmul_rn(c1, a.m)))));
    return r;
}
__device__ __forceinline__ double times_sqrt6(double a) { return 2.449489742783178098 * a; }
__device__ __forceinline__ TripleSum twice(TripleSum a) {
    a.h = __fadd_rn(a.h, a.h);
    a.l = __fadd_rn(a.l, a.l);
    a.m = __fadd_rn(a.m, a.m);
    return a;
}
__device__ __forceinline__ double twice(double a) { return 2.0 * a; }
__device__ __forceinline__ double square(double a) { return a * a; }
__device__ __forceinline__ double square_root(double a) { return sqrt(a); }

// The per-node arithmetic by storage type: T a node's term, S a running sum of terms, E one
// of terms of one sign.
template <typename R>
struct ObsArith;
template <>
struct ObsArith<float> {
    using T = Pair;
    using S = PairSum;
    using E = TripleSum;
    // a b + c d and a b - c d
    __device__ static __forceinline__ T dot2(float a, float b, float c, float d) { return two_prod(a, b) + two_prod(c, d); }
    __device__ static __forceinline__ T cross2(float a, float b, float c, float d) { return two_prod(a, b) - two_prod(c, d); }
    __device__ static __forceinline__ void add(S& s, T v) {
        s.add(v.h);
        s.l = __fadd_rn(s.l, v.l);
    }
    // s += k v for a small integer k
    __device__ static __forceinline__ void add_times(S& s, float k, T v) {
        s.add_prod(k, v.h);
        s.l = __fmaf_rn(k, v.l, s.l);
    }
    // s += p (v - u)
    __device__ static __forceinline__ void add_diff(S& s, float p, float v, float u) {
        const T d = two_sum(v, -u);
        s.add_prod(p, d.h);
        s.l = __fmaf_rn(p, d.l, s.l);
    }
    __device__ static __forceinline__ void add_prod(E& s, float a, float b) { s.add_prod(a, b); }
    // a0 b0 + a1 b1 + a2 b2 + a3 b3 and the same with the second and fourth product subtracted
    __device__ static __forceinline__ E dot4(float a0, float b0, float a1, float b1, float a2, float b2, float a3, float b3) {
        const Pair p0 = two_prod(a0, b0), p1 = two_prod(a1, b1), p2 = two_prod(a2, b2), p3 = two_prod(a3, b3);
        const Pair s0 = two_sum(p0.h, p1.h), s1 = two_sum(p2.h, p3.h), t = two_sum(s0.h, s1.h);
        E s;
        s.h = t.h;
        s.l = p0.l;
        s.add_low(p1.l);
        s.add_low(p2.l);
        s.add_low(p3.l);
        s.add_low(s0.l);
        s.add_low(s1.l);
        s.add_low(t.l);
        return s;
    }
    __device__ static __forceinline__ E cross4(float a0, float b0, float a1, float b1, float a2, float b2, float a3, float b3) {
        return dot4(a0, b0, -a1, b1, a2, b2, -a3, b3);
    }
    // a a + b b; k (a - b) for k a power of two; a sum in E as a term
    __device__ static __forceinline__ E norm2(float a, float b) {
        E s(a, a);
        s.add_prod(b, b);
        return s;
    }
    __device__ static __forceinline__ E difference(float k, E a, E b) {
        b.h = -b.h;
        b.l = -b.l;
        b.m = -b.m;
        a.add(b);
        a.h *= k;
        a.l *= k;
        a.m *= k;
        return a;
    }
    __device__ static __forceinline__ E product(const E& a, const E& b) {
        E r(a.h, b.h);
        const Pair p = two_prod(a.h, b.l), q = two_prod(a.l, b.h);
        r.add_low(p.h);
        r.add_low(q.h);
        r.m = __fadd_rn(r.m, __fadd_rn(__fadd_rn(p.l, q.l), __fmaf_rn(a.l, b.l, __fmaf_rn(a.h, b.m, __fmul_rn(a.m, b.h)))));
        return r;
    }
    __device__ static __forceinline__ T term(const E& s) { return s.pair(); }
    // as a term where the words may cancel: h + l exactly first
    __device__ static __forceinline__ T rest(const E& s) {
        const Pair p = two_sum(s.h, s.l);
        return pair_norm(p.h, __fadd_rn(p.l, s.m));
    }
    // s^2 (rounding s to a pair first would leave 4e-16 of the interaction energy)
    __device__ static __forceinline__ T square_of(const E& s) {
        const Pair n = pair_norm(s.h, s.l), p = two_prod(n.h, n.h);
        const float hl = __fmaf_rn(n.l, n.h, __fmaf_rn(s.m, n.h, __fmul_rn(__fmul_rn(0.5f, n.l), n.l)));
        return pair_norm(p.h, __fmaf_rn(2.f, hl, p.l));
    }
    template <class V>
    __device__ static __forceinline__ void add(E& s, const V& v) {
        s.add(v);
    }
    __device__ static __forceinline__ void add_times(E& s, float k, const E& v) { s.add_times(k, v); }
    __device__ static __forceinline__ double value(const S& s) { return s.value(); }
    __device__ static __forceinline__ double value(const E& s) { return s.value(); }
    __device__ static __forceinline__ bool less(T a, T b) { return a.h < b.h || (a.h == b.h && a.l < b.l); }
    __device__ static __forceinline__ T zero() { return Pair{0.f, 0.f}; }
    // the power of two that takes rho near 1 (1 where it is zero or subnormal), and v
    // times a power of two
    __device__ static __forceinline__ float unit(T rho) {
        const uint32_t e = __float_as_uint(rho.h) >> 23;   // rho >= 0
        return e > 0 && e < 254 ? __uint_as_float((254u - e) << 23) : 1.f;
    }
    __device__ static __forceinline__ T times(T v, float p) { return Pair{__fmul_rn(v.h, p), __fmul_rn(v.l, p)}; }
};
template <>
struct ObsArith<double> {
    using T = double;
    using S = double;
    using E = double;
    __device__ static __forceinline__ void add_prod(E& s, double a, double b) { s = fm(a, b, s); }
    __device__ static __forceinline__ E norm2(double a, double b) { return fm(a, a, b * b); }
    __device__ static __forceinline__ E difference(double k, E a, E b) { return k * (a - b); }
    __device__ static __forceinline__ E product(E a, E b) { return a * b; }
    __device__ static __forceinline__ T term(E s) { return s; }
    __device__ static __forceinline__ T rest(E s) { return s; }
    __device__ static __forceinline__ E dot4(double a0, double b0, double a1, double b1, double a2, double b2, double a3, double b3) {
        return fm(a0, b0, a1 * b1) + fm(a2, b2, a3 * b3);
    }
    __device__ static __forceinline__ E cross4(double a0, double b0, double a1, double b1, double a2, double b2, double a3,
                                               double b3) {
        return fm(a0, b0, -(a1 * b1)) + fm(a2, b2, -(a3 * b3));
    }
    __device__ static __forceinline__ T square_of(E s) { return s * s; }
    __device__ static __forceinline__ T dot2(double a, double b, double c, double d) { return fm(a, b, c * d); }
    __device__ static __forceinline__ T cross2(double a, double b, double c, double d) { return fm(a, b, -(c * d)); }
    __device__ static __forceinline__ void add(S& s, T v) { s += v; }
    __device__ static __forceinline__ void add_times(S& s, double k, T v) { s = fm(k, v, s); }
    __device__ static __forceinline__ void add_diff(S& s, double p, double v, double u) { s = fm(p, v - u, s); }
    __device__ static __forceinline__ double value(const S& s) { return s; }
    // both >= 0: the order of the bits, without the FP64 pipe (a NaN is never larger)
    __device__ static __forceinline__ bool less(T a, T b) {
        const long long x = __double_as_longlong(a), y = __double_as_longlong(b);
        return x < y && y <= 0x7ff0000000000000ll;
    }
    __device__ static __forceinline__ T zero() { return 0.0; }
    __device__ static __forceinline__ double unit(T) { return 1.0; }
    __device__ static __forceinline__ T times(T v, double p) { return v * p; }
};

// Bilinears of one node's spinor: densities n[s], their sum rho, and (spinors) F_z and
// the transverse spin as the reference's spin-1 sum m = conj(a) b + conj(b) c of three
// neighbouring components; spin-2 adds the sum of its outer pairs.
template <typename R, int C>
struct NodeTerms {
    using A = ObsArith<R>;
    using T = typename A::T;
    using E = typename A::E;
    E n[C], density;
    T rho;   // the density rounded to a term
    __device__ __forceinline__ explicit NodeTerms(const Cx<R>* p) {
#pragma unroll
        for (int s = 0; s < C; ++s) n[s] = A::norm2(p[s].x, p[s].y);
        density = n[0];
#pragma unroll
        for (int s = 1; s < C; ++s) A::add(density, n[s]);
        rho = A::term(density);
    }
    // F_z of components b .. (spin-2: of all five)
    template <int b>
    __device__ __forceinline__ E fz() const {
        if constexpr (b == 0 && C == 5) {
            E f = A::difference((R)2, n[0], n[4]);
            A::add(f, A::difference((R)1, n[1], n[3]));
            return f;
        } else {
            return A::difference((R)1, n[b], n[b + 2]);
        }
    }
    // Re and Im of conj(a) b + conj(c) d
    __device__ static __forceinline__ void pairs(Cx<R> a, Cx<R> b, Cx<R> c, Cx<R> d, E& re, E& im) {
        re = A::dot4(a.x, b.x, a.y, b.y, c.x, d.x, c.y, d.y);
        im = A::cross4(a.x, b.y, a.y, b.x, c.x, d.y, c.y, d.x);
    }
    // the transverse spin of three neighbouring components over sqrt2, conj(a) b + conj(b) c.  In
    // three words until its products are summed: in nematic and cyclic states they cancel, and
    // what pairs left of |F| there was 30 to 60 times as far off as FP64 terms (a polar cloud turned
    // by its texture, 1e-3 noise, relative: 4.5e-15 for 1e-16; with 1e-6 noise 4e-12 for 6e-14).
    __device__ static __forceinline__ void chain(Cx<R> a, Cx<R> b, Cx<R> c, T& re, T& im) {
        E er, ei;
        pairs(a, b, b, c, er, ei);
        re = A::rest(er);
        im = A::rest(ei);
    }
    // spin-2: <F_+> = 2 (conj(psi_2) psi_1 + conj(psi_-1) psi_-2) + sqrt6 (conj(psi_1) psi_0 +
    // conj(psi_0) psi_-1), likewise
    __device__ static __forceinline__ void transverse(const Cx<R>* p, T& fx, T& fy) {
        E re2, im2, re6, im6;
        pairs(p[0], p[1], p[3], p[4], re2, im2);
        pairs(p[1], p[2], p[2], p[3], re6, im6);
        re6 = times_sqrt6(re6);
        im6 = times_sqrt6(im6);
        A::add(re6, twice(re2));
        A::add(im6, twice(im2));
        fx = A::rest(re6);
        fy = A::rest(im6);
    }
    // the record whose |psi_s| is the largest so far, kept by its value (its modulus is
    // taken once per thread, in FP64)
    __device__ __forceinline__ void track_max(const Cx<R>* p, T& top, Cx<R>& at) const {
#pragma unroll
        for (int s = 0; s < C; ++s) {
            const T m = A::term(n[s]);
            if (A::less(top, m)) {
                top = m;
                at = p[s];
            }
        }
    }
};

// The largest |re|, |im| of the records so far (a NaN is none).
template <typename R, int C>
__device__ __forceinline__ R largest(R top, const Cx<R>* p) {
#pragma unroll
    for (int s = 0; s < C; ++s) top = fmax(top, fmax(fabs(p[s].x), fabs(p[s].y)));
    return top;
}

template <typename R, int C>
__device__ __forceinline__ uint32_t count_nonfinite(const Cx<R>* p) {
    uint32_t n = 0;
#pragma unroll
    for (int s = 0; s < C; ++s) n += (!isfinite(p[s].x) || !isfinite(p[s].y)) ? 1u : 0u;
    return n;
}

// Observables of a.prev (the quantities of observe_kernel, without the quadratic
// Zeeman term): a thread takes node l of the cells (x, y, z0 .. z0 + zc - 1) in turn,
// consecutive threads consecutive nodes along x, so that the rows are read as in the
// step kernels and the neighbours in z come from the thread's own recent reads.  D: the
// longest row (4, 6 or 8 entries).  The sums of a column's nodes are combined in FP64
// once per column of zc cells.  FP32 has two blocks per SM (128 registers): spin-1 without
// spills, spin-2 with 84 to 184 bytes of them.  gpe_observe as a whole, before (FP64 terms) and
// now: spin-1 BCC 64^3 1527 -> 191 us, spin-2 BCC 64^3 3512 -> 310, C15 32^3 4964 -> 434.
template <typename R, int C, int D>
__global__ void __launch_bounds__(256, sizeof(R) == 4 ? 2 : 1) observe_columns_kernel(StepArgs a, uint32_t zc, uint32_t columns,
                                                                                    uint32_t total, FastDiv dcol) {
    using A = ObsArith<R>;
    using T = typename A::T;
    using S = typename A::S;
    __shared__ SmemTables<double> st;
    __shared__ double red[8][OBS_COUNT];
    {
        const int V = a.g.V, n = a.tab.entries;
        for (int i = threadIdx.x; i <= V; i += blockDim.x) st.row_ptr[i] = a.tab.row_ptr[i];
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            st.nb_off[i] = a.tab.nb_off[i];
            st.w[i] = a.tab.w64[i] * a.pd.ks;  // condensate expansion: weights h / bs^2 of the step's bs
        }
        for (int i = threadIdx.x; i < 3 * V; i += blockDim.x) st.pos[i] = a.tab.pos64[i];
    }
    __syncthreads();
    const PhysR<double>& P = a.pd;
    double acc[OBS_COUNT];
#pragma unroll
    for (int k = 0; k < OBS_COUNT; ++k) acc[k] = 0.0;
    T top = A::zero();
    Cx<R> at = cx<R>((R)0, (R)0);
    R big = (R)0;
    uint32_t nbad = 0;
    const uint32_t node_bytes = C * 2 * sizeof(R);
    for (Strided it(blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x, total); it.more(); it.next()) {
        const uint32_t i = it.i;
        const uint32_t chunk = fdiv(i, dcol);
        const uint32_t col = i - chunk * columns;   // (y X + x) V + l
        const uint32_t y = fdiv(col, a.divRow);
        const uint32_t within = col - y * a.row_items;
        const uint32_t x = fdiv(within, a.divV);
        const uint32_t l = within - x * a.g.V;
        // moments in z are taken about the column's middle
        const uint32_t z0 = chunk * zc, nz = min(zc, a.g.Z - z0), mid = nz / 2;
        const char* base = a.prev + (size_t)z0 * a.g.slice + (size_t)y * a.g.pitch + (size_t)x * a.g.cell_bytes;
        const int f0 = st.row_ptr[l], nd = st.row_ptr[l + 1] - f0;
        int32_t off[D];
#pragma unroll
        for (int k = 0; k < D; ++k) off[k] = k < nd ? st.nb_off[f0 + k] : (int32_t)(l * node_bytes);
        S kin[D], mx{}, my{};
        typename A::E s0{}, s1{}, s2{}, srr{}, sff{}, sth{}, sabs{}, fz{}, fz1{};
#pragma unroll
        for (int k = 0; k < D; ++k) kin[k] = S{};
#pragma unroll 1
        for (uint32_t j = 0; j < nz; ++j, base += a.g.slice) {
            Cx<R> p[C];
            ld_node<R, C, true>(base + l * node_bytes, p);
            constexpr int G = C == 5 ? 2 : 4;
#pragma unroll
            for (int k0 = 0; k0 < D; k0 += G) {
                Cx<R> v[G][C];
#pragma unroll
                for (int k = 0; k < G; ++k)
                    if (k0 + k < D) ld_node<R, C, true>(base + off[k0 + k], v[k]);
#pragma unroll
                for (int k = 0; k < G; ++k) {
                    if (k0 + k < D) {
#pragma unroll
                        for (int s = 0; s < C; ++s) {
                            A::add_diff(kin[k0 + k], p[s].x, v[k][s].x, p[s].x);
                            A::add_diff(kin[k0 + k], p[s].y, v[k][s].y, p[s].y);
                        }
                    }
                }
            }
            nbad += count_nonfinite<R, C>(p);
            if constexpr (sizeof(R) == 4) big = largest<R, C>(big, p);
            const NodeTerms<R, C> t(p);
            t.track_max(p, top, at);
            const R zj = (R)((int32_t)j - (int32_t)mid);
            A::add(s0, t.density);
            A::add_times(s1, zj, t.density);
            A::add_times(s2, zj * zj, t.density);
            A::add(srr, A::square_of(t.density));
            if constexpr (C == 3) {
                T re, im;
                t.chain(p[0], p[1], p[2], re, im);
                const typename A::E fe = t.template fz<0>();
                const T f = A::rest(fe);
                const T ff = twice(square(re) + square(im)) + square(f);
                A::add(mx, re);
                A::add(my, im);
                A::add(fz, fe);
                A::add_times(fz1, zj, fe);
                A::add(sff, ff);
                A::add(sabs, square_root(ff));
            } else if constexpr (C == 5) {
                T fx, fy;
                t.transverse(p, fx, fy);
                const typename A::E fe = t.template fz<0>();
                const T f = A::rest(fe);
                const T ff = square(fx) + square(fy) + square(f);
                A::add(mx, fx);
                A::add(my, fy);
                A::add(fz, fe);
                A::add_times(fz1, zj, fe);
                A::add(sff, ff);
                A::add(sabs, square_root(ff));
                // |theta|^2 of the singlet sum theta = psi_0^2 - 2 psi_1 psi_-1 + 2 psi_2 psi_-2
                const T tx = A::cross2(p[2].x, p[2].x, p[2].y, p[2].y) +
                             twice(A::cross2(p[0].x, p[4].x, p[0].y, p[4].y) - A::cross2(p[1].x, p[3].x, p[1].y, p[3].y));
                const T ty = twice(A::dot2(p[2].x, p[2].y, (R)0, (R)0) + A::dot2(p[0].x, p[4].y, p[0].y, p[4].x) -
                                   A::dot2(p[1].x, p[3].y, p[1].y, p[3].x));
                A::add(sth, square(tx) + square(ty));
            }
        }
        // the column's sums with what is the same for all its nodes
        const double S0 = A::value(s0), S1 = A::value(s1), S2 = A::value(s2);
        const double rx = P.p0[0] + P.bs * ((double)x * P.bw[0] + st.pos[3 * l + 0]);
        const double ry = P.p0[1] + P.bs * ((double)y * P.bw[1] + st.pos[3 * l + 1]);
        // the middle's height and the step, whose roundings are the same for all the column's
        // nodes, with what they leave out (heights rounded as a whole put up to 1e-15 of the
        // centre of mass)
        const double zm = (double)(z0 + mid), hm = zm * P.bw[2], hl = fm(zm, P.bw[2], -hm);
        const double rz = fm(P.bs, st.pos[3 * l + 2] + hl, fm(P.bs, hm, P.p0[2]));
        const double gz = P.bs * P.bw[2], gl = fm(P.bs, P.bw[2], -gz);
        double hexp = 0.0, eint = P.c0 * A::value(srr);
#pragma unroll
        for (int k = 0; k < D; ++k)
            if (k < nd) hexp += st.w[f0 + k] * A::value(kin[k]);
        if (P.trap_on) {
            const double tx = rx * P.lambda[0], ty = ry * P.lambda[1], hz = 0.5 * P.lambda[2] * P.lambda[2];
            hexp += (0.5 * (tx * tx + ty * ty) + P.trap_offset) * S0 + 
                    hz * (rz * rz * S0 + (gz * (2.0 * rz * S1 + gz * S2) + 2.0 * gl * (rz * S1 + gz * S2)));
        }
        if constexpr (C > 1) {
            const double q = C == 3 ? GPE_REF_SQRT_2 : 1.0, Mx = q * A::value(mx), My = q * A::value(my);
            const double Mz = A::value(fz), Mz1 = A::value(fz1);
            const bool qo = P.flags & GPE_FLAG_QUADRUPOLE_OFFSET;
            const double bx = P.bq * (rx - (qo ? P.qc[0] : 0.0)) + P.bb[0], by = P.bq * (ry - (qo ? P.qc[1] : 0.0)) + P.bb[1];
            const double bz = -2.0 * P.bq * (rz - (qo ? P.qc[2] : 0.0)) + P.bb[2];
            const double zee = bx * Mx + by * My + bz * Mz - 2.0 * P.bq * gz * Mz1;
            hexp += C == 3 ? zee : -zee;
            eint += P.c2 * A::value(sff);
            if constexpr (C == 5) eint += 0.2 * P.c4 * A::value(sth);
            acc[OBS_MAGX] += Mx;
            acc[OBS_MAGY] += My;
            acc[OBS_MAGZ] += Mz;
            acc[OBS_SPIN] += A::value(sabs);
        }
        acc[OBS_NORM] += S0;
        acc[OBS_HEXP] += hexp + eint;
        acc[OBS_EINT] += eint;
        acc[OBS_COMX] += rx * S0;
        acc[OBS_COMY] += ry * S0;
        acc[OBS_COMZ] += rz * S0 + (gz * S1 + gl * S1);
    }
    // FP32: densities that overflow, or all vanish, leave no record to track; the largest
    // |re|, |im| (never above the modulus) then takes the state out of the pairs' range
    acc[OBS_MAXABS] = fmax(sqrt((double)at.x * at.x + (double)at.y * at.y), (double)big);
    acc[OBS_NONFINITE] = (double)nbad;
    block_observables(acc, red, a.partials);
}

// ------------------------------------------------------------- integrated node fields

constexpr int kFieldSums = 6;  // the five sums and the largest |re|, |im|

// Block partials of the integrated DENSITY (one sum) or SPIN fields (integrateSpin-
// AndDensity, Spin1GpeBCC.cu:992-1020, of localAvgSpinAndDensity, :235-271) of a.prev,
// straight from the state: rho |s|, rho s_x, rho s_y, rho s_z, rho with the x, y spin
// of the normalised and the z spin of the unnormalised spinor, as the reference has
// them, so that rho s_x = sqrt2 Re m needs no division.  A node without density has
// no direction: its x, y spin is 0 / 0 in the reference and here, and so are the sums
// over it.  (Writing five FP64 values a node and summing them in a second pass, with
// two FP64 square roots and six divisions a node, took 310 + 51 us on spin-1 BCC
// 64^3.)  A: the arithmetic's type, the storage's or double.
template <typename R, typename A, int C, bool SPIN>
__global__ void __launch_bounds__(256) field_sums_kernel(StepArgs a) {
    using O = ObsArith<A>;
    using T = typename O::T;
    __shared__ double red[8][kFieldSums];
    typename O::S sx{}, sy{};
    typename O::E spin{}, density{}, sz{};
    A top = (A)0;
    bool empty = false;
    for (uint64_t gid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; gid < a.total;
         gid += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t i = (uint32_t)gid;
        const uint32_t row = fdiv(i, a.divRow);
        const uint32_t within = i - row * a.row_items;
        const uint32_t x = fdiv(within, a.divV);
        const uint32_t l = within - x * a.g.V;
        const uint32_t z = fdiv(row, a.divY);
        const uint32_t y = row - z * a.g.Y;
        Cx<R> v[C];
        ld_node<R, C, true>(a.prev + (size_t)z * a.g.slice + (size_t)y * a.g.pitch + (size_t)x * a.g.cell_bytes +
                                l * (C * 2 * sizeof(R)), v);
        Cx<A> p[C];
#pragma unroll
        for (int c = 0; c < C; ++c) p[c] = cx<A>((A)v[c].x, (A)v[c].y);
        if constexpr (sizeof(A) == 4) top = largest<A, C>(top, p);
        const NodeTerms<A, C> t(p);
        O::add(density, t.density);
        if constexpr (SPIN && C > 1) {
            constexpr int b = C == 5 ? 1 : 0;  // s1, s0, s_1
            T re, im;
            t.chain(p[b], p[b + 1], p[b + 2], re, im);
            const typename O::E fe = t.template fz<b>();
            const T f = O::rest(fe);
            O::add(sx, re);
            O::add(sy, im);
            O::add(sz, O::product(t.density, fe));
            // rho |s| with m and rho taken near 1, so that no square leaves the range
            const A u = O::unit(t.rho);
            const T rx = O::times(re, u), ry = O::times(im, u), rz = O::times(t.rho, u) * f;
            O::add(spin, O::times(square_root(twice(square(rx) + square(ry)) + square(rz)), (A)1 / u));
            bool none = true;
#pragma unroll
            for (int c = 0; c < C; ++c) none = none && p[c].x == (A)0 && p[c].y == (A)0;
            empty = empty || none;
        }
    }
    double v[kFieldSums] = {O::value(SPIN && C > 1 ? spin : density), 0.0, 0.0, 0.0, 0.0, (double)top};
    if constexpr (SPIN) {
        v[1] = GPE_REF_SQRT_2 * O::value(sx);
        v[2] = GPE_REF_SQRT_2 * O::value(sy);
        v[3] = O::value(sz);
        v[4] = O::value(density);
        if (empty) v[0] = v[1] = v[2] = nan("");
    }
#pragma unroll
    for (int k = 0; k < kFieldSums; ++k)
        for (int o = 16; o > 0; o >>= 1) {
            const double u = __shfl_down_sync(0xffffffffu, v[k], o);
            v[k] = k == 5 ? fmax(v[k], u) : v[k] + u;
        }
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int k = 0; k < kFieldSums; ++k) red[threadIdx.x >> 5][k] = v[k];
    }
    __syncthreads();
    if (threadIdx.x < kFieldSums) {
        double u = red[0][threadIdx.x];
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
            u = threadIdx.x == 5 ? fmax(u, red[w][threadIdx.x]) : u + red[w][threadIdx.x];
        a.partials[(size_t)blockIdx.x * kFieldSums + threadIdx.x] = u;
    }
}

// ------------------------------------------------------------------------- launchers

template <typename R, int C, int D>
cudaError_t launch_observe_columns_d(const StepArgs& a, double* out, cudaStream_t s) {
    static int occ = 0;
    auto k = observe_columns_kernel<R, C, D>;
    if (occ == 0) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, 256, 0);
        occ = std::max(occ, 1);
    }
    // a column's FP64 part, about 100 operations, costs what 9 nodes cost
    const ColumnGrid g = column_grid(a, (unsigned)occ, cells_by_thread(a, (unsigned)occ, 9));
    k<<<g.blocks, 256, 0, s>>>(a, g.zc, g.columns, g.total, make_fastdiv(g.columns));
    finalize_observables(a.partials, g.blocks, out, s);
    return cudaGetLastError();
}

template <typename R, int C>
cudaError_t launch_observe_columns(const StepArgs& a, double* out, cudaStream_t s) {
    if (a.tab.max_deg <= 4) return launch_observe_columns_d<R, C, 4>(a, out, s);
    if (a.tab.max_deg == 6) return launch_observe_columns_d<R, C, 6>(a, out, s);
    if (a.tab.max_deg == 8) return launch_observe_columns_d<R, C, 8>(a, out, s);
    return cudaErrorInvalidValue;
}

// The sums of field_sums_kernel into out[kFieldSums], in pairs of FP32 values (FP32
// storage) unless fp64.
template <typename R, int C>
cudaError_t launch_field_sums(const StepArgs& a, bool spin, bool fp64, double* out, cudaStream_t s) {
    const unsigned nb = std::min<unsigned>(nblocks(a.total, 256), 4u * (unsigned)device_sm_count());
    auto go = [&](auto k) { k<<<nb, 256, 0, s>>>(a); };
    if (fp64 || sizeof(R) == 8) spin ? go(field_sums_kernel<R, double, C, true>) : go(field_sums_kernel<R, double, C, false>);
    else spin ? go(field_sums_kernel<R, R, C, true>) : go(field_sums_kernel<R, R, C, false>);
    sum_partials_kernel<kFieldSums, 5><<<1, 32 * kFieldSums, 0, s>>>(a.partials, nb, out);
    return cudaGetLastError();
}

#define GPE_INSTANTIATE_OBSERVE(R, C)                                                            \
    template cudaError_t launch_observe_columns<R, C>(const StepArgs&, double*, cudaStream_t);   \
    template cudaError_t launch_field_sums<R, C>(const StepArgs&, bool, bool, double*, cudaStream_t);

}  // namespace gpe
