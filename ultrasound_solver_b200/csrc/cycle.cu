// The Arnoldi steps of a whole restart cycle in one cooperative launch, for
// solves whose passes over the Krylov basis are short.
//
// gmres.cu runs two launches per Arnoldi step and reduces in the last CTA of
// each. On small grids those launches do little but wait. Here the CTAs of a
// right-hand side own a fixed range of its nodes for the whole cycle and meet
// once per step:
//
//   w = s K u_j and the dots of the own nodes; the per-CTA sums (and that of
//   ||u_j||^2) are published, one CTA per entry adds them and publishes the
//   total -> u_{j+1} = w - sum_t h_t sigma_t u_t
//
// The norm of u_j travels with the dots of step j: w is scaled by the last
// known scale (sigma_{j-1}, so the stored values keep their range) and the
// ratio sigma_j / sigma_{j-1} enters the coefficients. Between steps a CTA only
// waits for the CTAs whose nodes its stencil reads.
//
// What is published carries the step's number in the same 16 bytes, so a
// reader polls the values themselves: no barrier counter and, for the sums, no
// memory fence. Measured per meeting at 48^3 (148 CTAs, SM cycles): all CTAs
// polling all partial sums 10500 (the polls crowd the few lines they wait for),
// an arrival counter with the totals formed in every CTA 6000-6400, this tree
// 6000-6400 without the fence of a counter. The slices of the basis stay in
// shared memory as far as they fit, first vectors first (each is read twice
// per later step), and the row coefficients when everything fits. The Givens
// rotations of all columns are applied once, in the least-squares kernel.
//
// The launch is cooperative: all CTAs are resident, and CTAs only wait for
// CTAs of the same right-hand side. Every wait is bounded; one that runs out
// ends the right-hand side with ST_DEVICE_TIMEOUT.
#include "cycle.cuh"

#include <type_traits>

namespace usv {

namespace {

constexpr int kCycWarps = kCycThreads / 32;
static_assert((USV_MAX_RESTART + 1 + kDotVecs) / kDotVecs <= 32, "group counts of the segment table");

// UN 16-byte loads per thread and vector slice; NL nodes per load.
template <typename S, int UN> struct Geo {
    static constexpr int NL = 16 / int(sizeof(S));
    static constexpr int NODES = NL * UN;               // nodes per thread
    static constexpr int MAX = kCycThreads * NODES;     // nodes per CTA
    static constexpr size_t COEF = 6 * sizeof(S);       // row coefficients per node
    static constexpr int LOADS = UN >= 4 ? 1 : 4 / UN;  // vectors in flight per thread (update)
};

// Shared memory: dot sums per task, reduced values, update coefficients, scales,
// w; then, as far as it goes, slices of the basis and row coefficients.
template <typename S> struct CycFixed {
    size_t dots, hs, hm, sig, segs, w, total;
    __host__ __device__ CycFixed(int m, int max_nodes) {
        auto up = [](size_t b) { return (b + 127) / 128 * 128; };
        dots = 0;
        // (a step has at most m dots)
        hs = up(sizeof(double) * 2 * kDotVecs * cycle_task_room((m + kDotVecs - 1) / kDotVecs, max_nodes));
        hm = hs + up(sizeof(double2) * (m + 2));
        sig = hm + up(sizeof(double2) * (m + 2));
        segs = sig + up(sizeof(double) * (m + 2));
        w = segs + 128;
        total = w + up(sizeof(typename DotW<S>::T) * max_nodes);
    }
};

// A published value: 16 bytes, written and read as one.
__device__ __forceinline__ void publish(ulonglong2* p, double v, unsigned long long epoch) {
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}"
                 ::"l"(p), "l"(__double_as_longlong(v)), "l"(epoch)
                 : "memory");
}
__device__ __forceinline__ double peek(const ulonglong2* p, unsigned long long& epoch) {
    long long v;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(v), "=l"(epoch)
                 : "l"(p)
                 : "memory");
    return __longlong_as_double(v);
}
// One warp: the sum of the ncta values at p (fixed order), waiting for values of
// this epoch. False when the wait ran out (about a second).
__device__ __noinline__ bool warp_gather(const ulonglong2* p, int ncta, unsigned long long epoch,
                                            double& total) {
    constexpr int Q = 5;  // 160 CTAs per pass
    const int lane = threadIdx.x & 31;
    double s = 0.0;
    bool ok = true;
    const long long t0 = clock64();
    for (int q0 = 0; q0 < ncta && ok; q0 += 32 * Q) {
        double v[Q];
        for (;;) {
            bool ready = true;
#pragma unroll
            for (int i = 0; i < Q; ++i) {
                const int q = q0 + 32 * i + lane;
                v[i] = 0.0;
                if (q < ncta) {
                    unsigned long long e;
                    v[i] = peek(p + q, e);
                    ready = ready && e == epoch;
                }
            }
            if (__all_sync(0xffffffffu, ready)) break;
            ok = __all_sync(0xffffffffu, clock64() - t0 < (1LL << 31));
            if (!ok) break;
        }
#pragma unroll
        for (int i = 0; i < Q; ++i) s += v[i];
    }
    total = warp_sum(s);
    return ok;
}

// One thread: the value published at p with this epoch.
__device__ __noinline__ bool await(const ulonglong2* p, unsigned long long epoch, double& v) {
    unsigned long long e;
    v = peek(p, e);
    if (e == epoch) return true;
    const long long t0 = clock64();
    while (v = peek(p, e), e != epoch)
        if (clock64() - t0 > (1LL << 31)) return false;
    return true;
}
// One warp: wait until the flags first .. last have reached this epoch.
__device__ __noinline__ bool await_flags(const unsigned long long* flags, int first, int last,
                                         unsigned long long epoch) {
    const long long t0 = clock64();
    bool ok = true;
    for (int r = first + (threadIdx.x & 31); r <= last && ok; r += 32) {
        for (;;) {
            unsigned long long e;
            asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(e) : "l"(flags + r) : "memory");
            if (e >= epoch) break;
            ok = clock64() - t0 < (1LL << 31);
            if (!ok) break;
        }
    }
    return __all_sync(0xffffffffu, ok);
}
// Value c of a 16-byte load in the arithmetic of the update (complex64: scaled
// by 2^-896, see widen_scaled), f w, and the updated values rounded and packed.
template <typename S> struct Upd;
template <> struct Upd<bf2> {
    static __device__ __forceinline__ void start(const bf2* y, double f, float2 (&u)[4]) {
        const uint4 r = *reinterpret_cast<const uint4*>(y);
#pragma unroll
        for (int c = 0; c < 4; ++c) u[c] = cscale(get(r, c), float(f));
    }
    static __device__ __forceinline__ float2 get(const uint4& r, int c) {
        const unsigned v = c == 0 ? r.x : c == 1 ? r.y : c == 2 ? r.z : r.w;
        return to_f(*reinterpret_cast<const bf2*>(&v));
    }
    static __device__ __forceinline__ uint4 pack(const float2 (&u)[4]) {
        unsigned w[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const bf2 h = __float22bfloat162_rn(u[c]);
            w[c] = *reinterpret_cast<const unsigned*>(&h);
        }
        return make_uint4(w[0], w[1], w[2], w[3]);
    }
    static __device__ __forceinline__ double norm2(const uint4& r, int c) {
        const float2 f = get(r, c);
        return cabs2(make_double2(f.x, f.y));
    }
};
template <> struct Upd<float2> {
    static __device__ __forceinline__ void start(const double2* y, double f, double2 (&u)[2]) {
#pragma unroll
        for (int c = 0; c < 2; ++c) u[c] = cscale(cscale(y[c], kScaleDown * f), kScaleDown);
    }
    static __device__ __forceinline__ double2 get(const uint4& r, int c) {
        return c ? make_double2(widen_scaled(r.z), widen_scaled(r.w))
                 : make_double2(widen_scaled(r.x), widen_scaled(r.y));
    }
    static __device__ __forceinline__ uint4 pack(const double2 (&u)[2]) {
        return make_uint4(__float_as_uint(float(u[0].x * kScaleUp)), __float_as_uint(float(u[0].y * kScaleUp)),
                          __float_as_uint(float(u[1].x * kScaleUp)), __float_as_uint(float(u[1].y * kScaleUp)));
    }
    static __device__ __forceinline__ double norm2(const uint4& r, int c) {
        return cabs2(c ? make_double2(__uint_as_float(r.z), __uint_as_float(r.w))
                       : make_double2(__uint_as_float(r.x), __uint_as_float(r.y)));
    }
};
template <> struct Upd<double2> {
    static __device__ __forceinline__ void start(const double2* y, double f, double2 (&u)[1]) {
        u[0] = cscale(y[0], f);
    }
    static __device__ __forceinline__ double2 get(const uint4& r, int) {
        return *reinterpret_cast<const double2*>(&r);
    }
    static __device__ __forceinline__ uint4 pack(const double2 (&u)[1]) {
        return *reinterpret_cast<const uint4*>(&u[0]);
    }
    static __device__ __forceinline__ double norm2(const uint4& r, int) { return cabs2(get(r, 0)); }
};
// u -= h v
__device__ __forceinline__ void sub_mul(float2& u, float2 h, float2 v) {
    u = ffma2(v, make_float2(-h.x, -h.x), u);
    u = ffma2(make_float2(v.y, v.x), make_float2(h.y, -h.y), u);
}
__device__ __forceinline__ void sub_mul(double2& u, double2 h, double2 v) {
    u.x = fma(-h.x, v.x, fma(h.y, v.y, u.x));
    u.y = fma(-h.x, v.y, fma(-h.y, v.x, u.y));
}

// Row coefficients of a node: six neighbour directions, in the precision of
// the vectors, from the operator buffer.
template <typename S> struct RowCoef;
template <> struct RowCoef<bf2> {
    bf2 c[6];
};
template <> struct RowCoef<float2> {
    float2 c[6];
};
template <> struct RowCoef<double2> {
    double2 c[6];
};
__device__ __forceinline__ void load_coef(const OpView<float>& op, long long n, bool, RowCoef<bf2>& k) {
    const uint2* p = op.cb + 3 * n;
    const uint2 a = __ldg(p), b = __ldg(p + 1), d = __ldg(p + 2);
    const unsigned w[6] = {a.x, a.y, b.x, b.y, d.x, d.y};
#pragma unroll
    for (int i = 0; i < 6; ++i) k.c[i] = *reinterpret_cast<const bf2*>(&w[i]);
}
__device__ __forceinline__ void load_coef(const OpView<float>& op, long long n, bool, RowCoef<float2>& k) {
    const float4* p = op.cf + 3 * n;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const float4 v = __ldg(p + q);
        k.c[2 * q] = make_float2(v.x, v.y);
        k.c[2 * q + 1] = make_float2(v.z, v.w);
    }
}
// complex128: R_n e_nd s_d from the FP64 edge coefficients and node records
__device__ __forceinline__ void load_coef(const OpView<double>& op, long long n, bool adj,
                                          RowCoef<double2>& k) {
    const Node p = decode(n, op.nx, op.ny);
    const long long sy = op.nx, sz = (long long)op.nx * op.ny;
    const double r = op.rec[n].y;
    const bool fixed = node_fixed(op.soft, p.i, p.j, p.k, op.nx, op.ny, op.nz);
    auto edge = [&](int d, bool has, int i, int j, int kk, long long m) {
        k.c[d] = make_double2(0.0, 0.0);
        if (!has || (adj ? node_fixed(op.soft, i, j, kk, op.nx, op.ny, op.nz) : fixed)) return;
        const double2 e = op.e64[6 * n + d];
        const double4 nb = op.rec[m];
        k.c[d] = cscale(cmul(adj ? cconj(e) : e, make_double2(nb.z, nb.w)), r);
    };
    edge(0, p.i > 0, p.i - 1, p.j, p.k, n - 1);
    edge(1, p.i < op.nx - 1, p.i + 1, p.j, p.k, n + 1);
    edge(2, p.j > 0, p.i, p.j - 1, p.k, n - sy);
    edge(3, p.j < op.ny - 1, p.i, p.j + 1, p.k, n + sy);
    edge(4, p.k > 0, p.i, p.j, p.k - 1, n - sz);
    edge(5, p.k < op.nz - 1, p.i, p.j, p.k + 1, n + sz);
}
// sigma (u_n + sum_d c_d u_d), rounded to the vector precision (the arithmetic
// of k_row_cb_clamped / k_row_cf_clamped: a missing neighbour has a zero
// coefficient and some finite value)
__device__ __forceinline__ bf2 row_value(const RowCoef<bf2>& k, const bf2 (&u)[7], float sj) {
    float rr = 0.f, ii = 0.f, ri = 0.f, ir = 0.f;
#pragma unroll
    for (int d = 0; d < 6; ++d) bf_mac(rr, ii, ri, ir, *reinterpret_cast<const unsigned*>(&k.c[d]), *reinterpret_cast<const unsigned*>(&u[d]));
    const float2 un = to_f(u[6]);
    return narrow<bf2>(cscale(make_float2(un.x + (rr - ii), un.y + (ri + ir)), sj));
}
__device__ __forceinline__ float2 row_value(const RowCoef<float2>& k, const float2 (&u)[7], float sj) {
    float2 y = u[6];
#pragma unroll
    for (int d = 0; d < 6; ++d) {
        y.x = fmaf(k.c[d].x, u[d].x, fmaf(-k.c[d].y, u[d].y, y.x));
        y.y = fmaf(k.c[d].x, u[d].y, fmaf(k.c[d].y, u[d].x, y.y));
    }
    return cscale(y, sj);
}
__device__ __forceinline__ double2 row_value(const RowCoef<double2>& k, const double2 (&u)[7], double sj) {
    double2 y = u[6];
#pragma unroll
    for (int d = 0; d < 6; ++d) {
        y.x = fma(k.c[d].x, u[d].x, fma(-k.c[d].y, u[d].y, y.x));
        y.y = fma(k.c[d].x, u[d].y, fma(k.c[d].y, u[d].x, y.y));
    }
    return cscale(y, sj);
}

}  // namespace

// Entry (j + 1, j) of the Hessenberg matrix, and its copy for the harmonic Ritz step.
__device__ __forceinline__ void set_subdiagonal(const GState& g, int b, int j, double beta) {
    const int m = g.m;
    g.H[((long long)b * m + j) * (m + 1) + j + 1] = make_double2(beta, 0.0);
    if (g.kr > 0) {
        double* gr = g.hb + (long long)b * g.hb_len + hb_graw(m) + 2LL * j * (m + 1) + 2 * (j + 1);
        gr[0] = beta;
        gr[1] = 0.0;
    }
}

// adj: rows of the adjoint operator (complex128 only; the others read the
// adjoint's own coefficient array). smem: dynamic shared memory of the launch.
template <typename R, typename S, bool MS, int UN>
__global__ void __launch_bounds__(kCycThreads, 1) k_cycle(OpView<R> op, S* V, GState g, int nrhs, int adj,
                                                          int smem) {
    using M2 = typename MathT<S>::T2;
    using MT = typename MathT<S>::T;
    using G = Geo<S, UN>;
    using W = typename DotW<S>::T;
    constexpr int NT = kCycThreads, NL = G::NL, NPT = G::NODES;
    extern __shared__ __align__(128) char cyc_smem[];
    __shared__ int who[4];  // right-hand side, rank, CTAs of it, failed wait
    __shared__ double wred[kCycWarps];
    __shared__ double raw_norm, h_norm;  // ||u_j||^2; sum |h|^2 of the previous column
    const int m = g.m;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // The CTAs are shared out over the right-hand sides still active, in
    // proportion to their scenes' sizes (contiguous blocks; every CTA derives
    // the same split from the status words, which only change between
    // launches or on a failed wait).
    if (threadIdx.x == 0) {
        // (32-bit arithmetic: cycle_shape takes at most kCycMaxCtas * cycle_line nodes)
        unsigned total = 0, active = 0;
#pragma unroll 1
        for (int b = 0; b < nrhs; ++b)
            if (g.status[b] == ST_ACTIVE) {
                total += MS ? unsigned(g.slots[b].n) : 1u;
                ++active;
            }
        who[0] = -1;
        who[3] = 0;
        unsigned before = 0, seen = 0;
#pragma unroll 1
        for (int b = 0; b < nrhs; ++b)
            if (g.status[b] == ST_ACTIVE) {
                const unsigned own = MS ? unsigned(g.slots[b].n) : 1u;
                const unsigned first = cycle_first_cta(gridDim.x, active, seen, before, total);
                before += own;
                ++seen;
                const unsigned end = cycle_first_cta(gridDim.x, active, seen, before, total);
                if (blockIdx.x >= first && blockIdx.x < end) {
                    who[0] = b;
                    who[1] = int(blockIdx.x - first);
                    who[2] = int(end - first);
                }
            }
    }
    __syncthreads();
    const int b = who[0];
    if (b < 0) return;
    const int rank = who[1], ncta = who[2];
    if constexpr (MS) op = slot_view<R>(g.slots[b]);
    const CycleBasis<S> cb = cycle_basis(V, g, b);
    const int kc = cb.kc;
    // node range of this CTA: at most G::MAX nodes in every launch of a solve
    // (cycle_shape). More would leave nodes out: such a right-hand side ends
    // with an error, set by the least-squares kernel so that the status words
    // do not change while other CTAs derive their split from them.
    const int N = int(op.n);
    const int per = cycle_cta_nodes(N, ncta);
    if (per > G::MAX) {
        if (rank == 0 && threadIdx.x == 0) {
            g.len[b] = -1;
            g.ended[b] = 1;
        }
        return;
    }
    const int lo = min(N, rank * per), len = min(N, lo + per) - lo;
    const int units = (len + NL - 1) / NL;

    const CycFixed<S> fix(m, G::MAX);
    double* ssum = reinterpret_cast<double*>(cyc_smem + fix.dots);
    double2* hs = reinterpret_cast<double2*>(cyc_smem + fix.hs);
    M2* hm = reinterpret_cast<M2*>(cyc_smem + fix.hm);
    double* sig = reinterpret_cast<double*>(cyc_smem + fix.sig);
    int* seg_table = reinterpret_cast<int*>(cyc_smem + fix.segs);
    W* ws = reinterpret_cast<W*>(cyc_smem + fix.w);
    // slices of slots 0 .. res-1 in shared memory; the coefficients too when
    // the whole basis fits, or (complex128, whose rows cost more to form than
    // slices to read: stencil 11000 -> 2500 SM cycles at 48^3) whenever they do
    char* sp = cyc_smem + fix.total;
    unsigned room = unsigned(smem) - unsigned(fix.total);
    const unsigned coef_bytes = unsigned(G::COEF) * per, slice_bytes = unsigned(sizeof(S)) * per;
    const bool coef_res = coef_bytes + (sizeof(S) == 16 ? 0u : slice_bytes * (m + 1)) <= room;
    if (coef_res) room -= coef_bytes;
    S* cw = reinterpret_cast<S*>(sp);
    S* vs = reinterpret_cast<S*>(sp + (coef_res ? coef_bytes : 0u));
    const int res = int(min(unsigned(m + 1), room / slice_bytes));
    auto global_slice = [&](int t) { return (t < kc ? cb.C : cb.V) + (long long)t * g.nv + lo; };

    // published sums of this right-hand side's CTAs: rows 2t, 2t+1 of the dots
    // (re, im), and the norms; the value of CTA `rank` at [rank]
    ulonglong2* part = g.cyc_part + blockIdx.x - rank;
    ulonglong2* npart = g.cyc_norm + blockIdx.x - rank;
    ulonglong2* tot = g.cyc_tot + (long long)b * 2 * (m + 2);
    ulonglong2* ntot = tot + 2 * (m + 1) + 1;
    unsigned long long epoch = *g.cyc_epoch;  // advanced between launches

    // segments per vector group
    if (threadIdx.x < 32) seg_table[threadIdx.x] = cycle_segments(threadIdx.x < 1 ? 1 : threadIdx.x, per);
#pragma unroll 1
    for (int t = threadIdx.x; t <= kc; t += NT) sig[t] = g.sigma[(long long)b * (m + 1) + t];
#pragma unroll 1
    for (int t = 0; t <= kc && t < res; ++t) {
        const S* src = global_slice(t);
#pragma unroll 1
        for (int e = NL * threadIdx.x; e < len; e += NL * NT)
            *reinterpret_cast<uint4*>(vs + t * per + e) = *reinterpret_cast<const uint4*>(src + e);
    }
    if (coef_res)
#pragma unroll 1
        for (int e = threadIdx.x; e < len; e += NT) {
            RowCoef<S> k;
            load_coef(op, lo + e, adj != 0, k);
#pragma unroll
            for (int d = 0; d < 6; ++d) cw[d * per + e] = k.c[d];
        }
    __syncthreads();

    // ranks whose nodes the stencil of this CTA reads
    const int reach = op.nx * op.ny;
    const int nb_first = max(0, lo - reach) / per, nb_last = min(N - 1, lo + len - 1 + reach) / per;
    unsigned long long* flags = g.cyc_flag + blockIdx.x - rank;
    // scale applied to u_j by the stencil: sigma_j, or an estimate while the
    // norm of u_j is still to come (pending)
    bool pending = false, after_proj = false;
    double est_inv = 1.0 / sig[kc];

    for (int j = kc > 0 ? kc - 1 : 0; j < m; ++j) {
        // proj (recycled cycles): the first residual (slot kc) against C_0..C_kc-1
        const bool proj = kc > 0 && j == kc - 1;
        const int nd = proj ? kc : j + 1;  // dot products
        const int out = proj ? kc : j + 1;
        S* slot = cb.V + (long long)out * g.nv + lo;
        ++epoch;
        // ---- w = s K u_j (proj: w = the residual)
        if (proj) {
#pragma unroll 1
            for (int e = threadIdx.x; e < per; e += NT) ws[e] = dot_value(e < len ? slot[e] : S{});
        } else {
            const S* uj = cb.V + (long long)j * g.nv;
            const R sj = R(sig[j]);
            const int sy = op.nx, sz = op.nx * op.ny, last = N - 1;
            constexpr int SU = 2;
#pragma unroll(SU)
            for (int c = 0; c < NPT; ++c) {
                const int e = threadIdx.x + NT * c;
                S y = S{};
                if (e < len) {
                    const int n = lo + e;
                    RowCoef<S> k;
                    if (coef_res) {
#pragma unroll
                        for (int d = 0; d < 6; ++d) k.c[d] = cw[d * per + e];
                    } else {
                        load_coef(op, n, adj != 0, k);
                    }
                    const S u[7] = {uj[max(n - 1, 0)], uj[min(n + 1, last)], uj[max(n - sy, 0)],
                                    uj[min(n + sy, last)], uj[max(n - sz, 0)], uj[min(n + sz, last)], uj[n]};
                    y = row_value(k, u, sj);
                }
                if (e < per) ws[e] = dot_value(y);
            }
        }
        __syncthreads();
        // ---- dots with slots 0 .. nd-1: a warp per (kDotVecs vectors, segment)
        const int groups = (nd + kDotVecs - 1) / kDotVecs;
        const int segs = seg_table[groups];
        const int per_seg = (units + segs - 1) / segs;
#pragma unroll 1
        for (int task = warp; task < groups * segs; task += kCycWarps) {
            const int gr = task / segs, sg = task - gr * segs;
            const int q0 = sg * per_seg, q1 = min(units, q0 + per_seg);
            const uint4* vp[kDotVecs];
            MT acc[2 * kDotVecs];  // (bfloat16: at most 128 nodes per fp32 lane sum, see cycle_segments)
#pragma unroll
            for (int i = 0; i < kDotVecs; ++i) {
                const int t = min(gr * kDotVecs + i, nd - 1);  // (a repeated vector's sums are not used)
                vp[i] = reinterpret_cast<const uint4*>(t < res ? vs + t * per : global_slice(t));
                acc[2 * i] = acc[2 * i + 1] = 0;
            }
            uint4 v[kDotVecs];
#pragma unroll
            for (int i = 0; i < kDotVecs; ++i)
                v[i] = q0 + lane < q1 ? vp[i][q0 + lane] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll 1
            for (int q = q0 + lane; q < q1; q += 32) {
                uint4 next[kDotVecs];
#pragma unroll
                for (int i = 0; i < kDotVecs; ++i)
                    if (q + 32 < q1) next[i] = vp[i][q + 32];
                const UnitW<S> w(ws + NL * q);
#pragma unroll
                for (int i = 0; i < kDotVecs; ++i) {
                    unit_dot(v[i], w, acc[2 * i], acc[2 * i + 1]);
                    v[i] = next[i];
                }
            }
            double wide[2 * kDotVecs];
#pragma unroll
            for (int i = 0; i < 2 * kDotVecs; ++i) wide[i] = double(acc[i]);
            int idx;
            const double sum = warp_sum_dots(wide, idx);
            if ((lane & 3) == 0) ssum[2 * kDotVecs * task + idx] = sum;
        }
        __syncthreads();
        // published: the dots <u_t, w>, unscaled, and the norm of u_j
        const int rows = 2 * nd + (pending ? 1 : 0);
        for (int q = threadIdx.x; q < rows; q += NT) {
            double v = 0.0;
            if (q < 2 * nd) {
                const int t = q >> 1, gr = t / kDotVecs, i = t - gr * kDotVecs;
#pragma unroll 1
                for (int sg = 0; sg < segs; ++sg)
                    v += ssum[2 * (kDotVecs * (gr * segs + sg) + i) + (q & 1)];
                publish(part + (long long)q * gridDim.x + rank, v, epoch);
            } else {
#pragma unroll 1
                for (int w = 0; w < kCycWarps; ++w) v += wred[w];
                publish(npart + rank, v, epoch);
            }
        }
        // totals: row q by warp q / ncta of the CTA of rank q % ncta
        bool ok = true;
#pragma unroll 1
        for (int q = rank + warp * ncta; q < rows; q += kCycWarps * ncta) {
            double v;
            ok = warp_gather(q < 2 * nd ? part + (long long)q * gridDim.x : npart, ncta, epoch, v) && ok;
            if (lane == 0 && ok) publish(q < 2 * nd ? tot + q : ntot, v, epoch);
        }
#pragma unroll 1
        for (int q = threadIdx.x; q < rows; q += NT) {
            double v;
            ok = await(q < 2 * nd ? tot + q : ntot, epoch, v) && ok;
            if (q < 2 * nd) reinterpret_cast<double*>(hs)[q] = v;
            else raw_norm = v;
        }
        if (!ok) who[3] = 1;
        __syncthreads();
        if (who[3]) {
            if (threadIdx.x == 0) g.status[b] = ST_DEVICE_TIMEOUT;
            return;
        }
        // ---- what ||u_j|| decides (before any use of hs: the sums over a u_j
        // that is not finite are meaningless, see widen_scaled)
        double ratio = 1.0, sigma_j = sig[j];
        if (pending) {
            const double n2 = raw_norm, beta = sqrt(n2);
            sigma_j = 1.0 / beta;
            ratio = sigma_j * est_inv;
            est_inv = beta;
            const bool finite = isfinite(beta);
            bool stop;
            if (after_proj) {
                stop = !(beta > 1e-300 && finite);  // r lies in span(C): the projection alone solves this cycle
                if (rank == 0 && threadIdx.x == 0)
                    g.g[(long long)b * (m + 1) + kc] = make_double2(stop ? 0.0 : beta, 0.0);
            } else {
                // breakdown: beta against ||w|| of its step, ||w||^2 = beta^2 + sum |h|^2
                const double wnorm = sqrt(n2 + h_norm);
                stop = !finite || !(beta > 1e-30 * wnorm);
                if (rank == 0 && threadIdx.x == 0)
                    set_subdiagonal(g, b, j - 1, beta);
            }
            if (rank == 0 && threadIdx.x == 0) {
                if (!(stop && after_proj)) g.sigma[(long long)b * (m + 1) + j] = stop ? 0.0 : sigma_j;
                if (stop) {
                    g.len[b] = j;
                    g.ended[b] = 1;
                }
            }
            if (stop) return;
            after_proj = false;
        }
        if (threadIdx.x < nd) {
            const int t = threadIdx.x;
            const double st = !proj && t == j ? sigma_j : sig[t];
            const double2 h = cscale(hs[t], proj ? st : st * ratio);
            hs[t] = h;
            const double2 hd = cscale(h, st);
            hm[t] = cmake<M2>(hd.x, hd.y);
            if (rank == 0) {
                // raw Hessenberg column (the least-squares kernel applies the
                // rotations), and its copy for the harmonic Ritz step
                if (proj) {
                    g.alpha[(long long)b * g.kr + t] = h;
                } else {
                    g.H[((long long)b * m + j) * (m + 1) + t] = h;
                    if (g.kr > 0) {
                        double* gr = g.hb + (long long)b * g.hb_len + hb_graw(m) + 2LL * j * (m + 1) + 2 * t;
                        gr[0] = h.x;
                        gr[1] = h.y;
                    }
                }
            }
        }
        __syncthreads();
        if (threadIdx.x == 0 && !proj) {
            sig[j] = sigma_j;
            if (j + 1 < m) sig[j + 1] = sigma_j;  // the estimate for the next stencil
        }
        if (warp == kCycWarps - 1) {
            double s = 0.0;
            for (int t = lane; t < nd; t += 32) s += cabs2(hs[t]);
            s = warp_sum(s);
            if (lane == 0) h_norm = s;
        }
        // ---- u_{j+1} = w - sum_t h_t sigma_t u_t
        double acc = 0.0;
        if (NL * warp * 32 < len) {
            M2 u[UN][NL];
#pragma unroll
            for (int q = 0; q < UN; ++q) {
                const int e = NL * (threadIdx.x + NT * q);
                Upd<S>::start(ws + (e < per ? e : 0), ratio, u[q]);
            }
            const int nres = min(nd, res);
#pragma unroll 2
            for (int t = 0; t < nres; ++t) {
                const M2 h = hm[t];
#pragma unroll
                for (int q = 0; q < UN; ++q) {
                    const int e = NL * (threadIdx.x + NT * q);
                    const uint4 raw = *reinterpret_cast<const uint4*>(vs + t * per + (e < per ? e : 0));
#pragma unroll
                    for (int c = 0; c < NL; ++c) sub_mul(u[q][c], h, Upd<S>::get(raw, c));
                }
            }
            constexpr int LB = G::LOADS;
#pragma unroll 1
            for (int t0 = nres; t0 < nd; t0 += LB) {
                uint4 raw[LB][UN];
#pragma unroll
                for (int i = 0; i < LB; ++i) {
                    const S* ut = global_slice(t0 + i);
#pragma unroll
                    for (int q = 0; q < UN; ++q) {
                        const int e = NL * (threadIdx.x + NT * q);
                        raw[i][q] = t0 + i < nd && e < len ? *reinterpret_cast<const uint4*>(ut + e)
                                                           : make_uint4(0u, 0u, 0u, 0u);
                    }
                }
#pragma unroll
                for (int i = 0; i < LB; ++i) {
                    const M2 h = hm[t0 + i < nd ? t0 + i : 0];  // (a vector past the last reads as zero)
#pragma unroll
                    for (int q = 0; q < UN; ++q)
#pragma unroll
                        for (int c = 0; c < NL; ++c) sub_mul(u[q][c], h, Upd<S>::get(raw[i][q], c));
                }
            }
#pragma unroll
            for (int q = 0; q < UN; ++q) {
                const int e = NL * (threadIdx.x + NT * q);
                if (e < len) {
                    const uint4 o = Upd<S>::pack(u[q]);
                    *reinterpret_cast<uint4*>(slot + e) = o;
                    if (out < res) *reinterpret_cast<uint4*>(vs + out * per + e) = o;
#pragma unroll
                    for (int c = 0; c < NL; ++c) acc += Upd<S>::norm2(o, c);
                }
            }
        }
        acc = warp_sum(acc);
        if (lane == 0) wred[warp] = acc;
        pending = true;
        after_proj = proj;
        if (j == m - 1) break;
        __syncthreads();  // (every u_{j+1} store of this CTA comes before the fence below)
        if (warp == 0) {
            if (lane == 0) {
                __threadfence();
                asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(flags + rank), "l"(epoch) : "memory");
            }
            const bool got = await_flags(flags, nb_first, nb_last, epoch);
            __threadfence();  // the neighbours' u_{j+1} are visible from here on
            if (!got) who[3] = 1;
        }
        __syncthreads();
        if (who[3]) {
            if (threadIdx.x == 0) g.status[b] = ST_DEVICE_TIMEOUT;
            return;
        }
    }
    // the last subdiagonal entry ||u_m||
    ++epoch;
    __syncthreads();
    if (warp == 0) {
        const double s = warp_sum(lane < kCycWarps ? wred[lane] : 0.0);
        if (lane == 0) publish(npart + rank, s, epoch);
        if (rank == 0) {
            double n2;
            const bool ok = warp_gather(npart, ncta, epoch, n2);
            if (lane == 0) {
                if (!ok) g.status[b] = ST_DEVICE_TIMEOUT;
                const double beta = sqrt(n2);
                const bool stop = !isfinite(beta) || !(beta > 1e-30 * sqrt(n2 + h_norm));
                set_subdiagonal(g, b, m - 1, beta);
                g.sigma[(long long)b * (m + 1) + m] = stop ? 0.0 : 1.0 / beta;
                g.len[b] = m;
                g.ended[b] = 1;
            }
        }
    }
}

// Launch of the instance that cycle_shape picks.
template <typename R, typename S, bool MS>
cudaError_t cycle_plan(int m, const long long* sizes, int nrhs, int sms, CyclePlan& plan) {
    plan = CyclePlan{};
    constexpr int bytes = int(sizeof(S));
    const CycleShape shape = cycle_shape(bytes, MS, sizes, nrhs, sms);
    if (!shape.ctas) return cudaSuccess;
    const void* fn = nullptr;
    int max_nodes = 0;
    auto instance = [&](auto index) {
        constexpr int I = decltype(index)::value;
        if constexpr (I < cycle_instances(bytes, MS)) {
            using G = Geo<S, cycle_units(bytes, I)>;
            static_assert(G::MAX == cycle_capacity(bytes, I), "room of an instance");
            if (shape.instance == I)
                fn = reinterpret_cast<const void*>(k_cycle<R, S, MS, cycle_units(bytes, I)>), max_nodes = G::MAX;
        }
    };
    instance(std::integral_constant<int, 0>());
    instance(std::integral_constant<int, 1>());
    instance(std::integral_constant<int, 2>());
    instance(std::integral_constant<int, 3>());
    if (!fn) return cudaSuccess;
    const CycFixed<S> fix(m, max_nodes);
    const size_t smem = 225 * 1024;
    if (fix.total > smem) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kCycThreads, smem);
    if (e != cudaSuccess || per_sm < 1) return e;
    plan.fn = fn;
    plan.ctas = shape.ctas;
    plan.smem = smem;
    return cudaSuccess;
}

#define USV_PLAN(R, S, MS) \
    template cudaError_t cycle_plan<R, S, MS>(int, const long long*, int, int, CyclePlan&);
USV_PLAN(float, bf2, false)
USV_PLAN(float, bf2, true)
USV_PLAN(float, float2, false)
USV_PLAN(float, float2, true)
USV_PLAN(double, double2, false)
USV_PLAN(double, double2, true)
#undef USV_PLAN

}  // namespace usv
