// State and conventions shared by the restarted GMRES kernels (gmres.cu: one
// launch per Arnoldi pass; cycle.cu: the Arnoldi steps of a whole cycle in one
// launch).
#pragma once

#include "usv_internal.cuh"

#define USV_MAX_RESTART 112  // keeps the m x (m+1) least-squares tile in shared memory

namespace usv {

enum { ST_ACTIVE = 0, ST_CONVERGED = 1, ST_MAXITER = 2, ST_NONFINITE = 3,
       ST_DEVICE_TIMEOUT = 4,  // a bounded device-side wait ran out
       ST_TOO_LARGE = 5 };     // more nodes per CTA than a kernel has room for

// Per-RHS control words of a recycled (GCRO-DR) cycle, written by the host
// before each cycle.
enum {
    CW_KC = 0,      // recycled vectors used by this cycle (0 or k)
    CW_PAIR,        // pair buffer (U, C) used by this cycle
    CW_VBUF,        // Krylov buffer of this cycle
    CW_COMBINE,     // 1: build pair CW_DST at the start of this cycle
    CW_SRC_PAIR,    // pair used by the cycle whose data builds the new pair
    CW_SRC_VBUF,    // its Krylov buffer
    CW_SRC_KC,      // its recycled count
    CW_DST,         // pair buffer written by the combine
    CW_HARVEST,     // 1: this cycle's data feeds a harmonic Ritz step
    kCtl
};
constexpr int kPairBufs = 3;   // pairs in use: this cycle's, the source cycle's, the new one
constexpr int kVBufs = 2;      // Krylov buffers: this cycle's and the previous cycle's

struct GState {
    int m, nblk, chunk, full_cycles, maxiter;
    int nchunk;        // node chunks of `chunk` nodes; CTAs loop over them (grid <= nblk)
    int ps;            // partial-sum slots per CTA
    long long n;
    long long nv;      // Krylov vector stride: n rounded up to 64 (512-B aligned pairs)
    double rtol;
    double2* partial;  // [B][nblk][ps], one row per CTA of the launch
    double2* H;        // [B][m][m+1]  column j, rows 0..m
    double* gc;        // [B][m]
    double2* gs;       // [B][m]
    double2* g;        // [B][m+1]
    double2* y;        // [B][m]   (y_t * sigma_t)
    double* sigma;     // [B][m+1]
    double* bnorm;     // [B]
    double* atol;      // [B]
    double* wnorm;     // [B]
    double* gates;     // [B][4]
    double* hist;      // [B][hcap] ||r||/||Rb|| at each restart test
    int hcap;
    int* status;       // [B]
    int* cycles;       // [B]
    int* iters;        // [B]
    int* len;          // [B]
    int* ended;        // [B]
    unsigned* counter; // [B]
    // recycling (GCRO-DR), kr > 0 only
    int kr;            // recycled vectors k
    int hb_len;        // doubles per RHS in the host-read block
    long long vstride; // elements between the Krylov buffers (B (m+1) nv)
    long long pstride; // elements between pair buffers (B k nv)
    void* Ubuf;        // [kPairBufs][B][k][nv] U, K U = C
    void* Cbuf;        // [kPairBufs][B][k][nv] C, orthonormal
    int* ctl;          // [B][kCtl]
    double2* coef;     // [B][k + m + 1][2k] combine coefficients
    double* hb;        // [B][hb_len] read by the host after each cycle:
                       //   raw G columns [m][m+1] complex, bd [m+1][k] complex,
                       //   sigma [m+1], d [k], then len, kc
    double* dU;        // [kPairBufs][B][k] 1/||U_i||
    double2* alpha;    // [B][k] projection C^H r of the cycle's first residual
    int* klast;        // [B] recycled count of the last finished cycle
    int* started;      // [B]
    // cycle kernel (cycle.cu), values published with the step's number:
    ulonglong2* cyc_part;  // [2 (m + 2)][ctas] per-CTA dots (re, im rows)
    ulonglong2* cyc_norm;  // [ctas] per-CTA norms
    ulonglong2* cyc_tot;   // [B][2 (m + 2)] totals (last entry: the norm)
    unsigned long long* cyc_flag;   // [ctas] step whose vector a CTA has stored
    unsigned long long* cyc_epoch;  // step number before the next launch
    long long l2_keep; // bytes of a basis pass that the next pass is to find in L2
    int coef_keep;     // 1: the row coefficients as well
    int orth_forward;  // 1: k_orth walks the node chunks in the order of the dots
    const struct SceneSlot* slots;  // [B] multi-scene solves: the scene of each RHS
};

// Scene of one right-hand side of a multi-scene solve (usv_gmres_solve_scenes):
// the operator views, node count and chunk count of that scene and the node
// steps of the 256- and kDotsThreads-thread kernels. Kernels instantiated
// with MS = true read their scene from here (blockIdx.y = right-hand side);
// single-scene kernels take it from their arguments.
struct SceneSlot {
    OpView<double> op64;
    OpView<float> op32;
    long long n;
    int nchunk;
    Step step, step_d;
};
template <typename R> __device__ __forceinline__ const OpView<R>& slot_view(const SceneSlot& s);
template <> __device__ __forceinline__ const OpView<double>& slot_view<double>(const SceneSlot& s) {
    return s.op64;
}
template <> __device__ __forceinline__ const OpView<float>& slot_view<float>(const SceneSlot& s) {
    return s.op32;
}
// CTAs of the launch that work for right-hand side b: all of them for a
// single scene; for a multi-scene batch a share proportional to the RHS's
// scene size (the grid is sized for the largest scene), at least one.
template <bool MS> __device__ __forceinline__ int rhs_ctas(const GState& g, int b) {
    if constexpr (MS) {
        const long long c = ((long long)gridDim.x * g.slots[b].n + g.n - 1) / g.n;
        return int(c < 1 ? 1 : c);
    } else {
        return int(gridDim.x);
    }
}


// host-read block offsets (in doubles)
__host__ __device__ __forceinline__ int hb_graw(int) { return 0; }
__host__ __device__ __forceinline__ int hb_bd(int m) { return 2 * m * (m + 1); }
__host__ __device__ __forceinline__ int hb_sigma(int m, int k) { return hb_bd(m) + 2 * (m + 1) * k; }
__host__ __device__ __forceinline__ int hb_d(int m, int k) { return hb_sigma(m, k) + m + 1; }
__host__ __device__ __forceinline__ int hb_tail(int m, int k) { return hb_d(m, k) + k; }
__host__ __device__ __forceinline__ int hb_size(int m, int k) { return hb_tail(m, k) + 2; }

// Vectors of RHS b's current cycle: t < kc are the recycled C_t (and U_t for
// the solution update), the others Krylov slots of the cycle's buffer.
template <typename S> struct CycleBasis {
    S* V;        // Krylov slot 0
    const S* C;  // C_0 of the cycle's pair (kc > 0)
    const S* U;  // U_0 of the cycle's pair (kc > 0)
    int kc;
    int pair;
};
template <typename S>
__device__ __forceinline__ CycleBasis<S> cycle_basis(S* V, const GState& g, int b) {
    CycleBasis<S> cb;
    cb.V = V + (long long)b * (g.m + 1) * g.nv;
    cb.C = cb.U = cb.V;
    cb.kc = 0;
    cb.pair = 0;
    if (g.kr > 0) {
        const int* cw = g.ctl + b * kCtl;
        cb.V += cw[CW_VBUF] * g.vstride;
        cb.kc = cw[CW_KC];
        cb.pair = cw[CW_PAIR] > 0 ? cw[CW_PAIR] : 0;
        const long long po = cb.pair * g.pstride + (long long)b * g.kr * g.nv;
        cb.C = static_cast<const S*>(g.Cbuf) + po;
        cb.U = static_cast<const S*>(g.Ubuf) + po;
    }
    return cb;
}

// Arithmetic of the basis passes per storage type. bfloat16 values (8-bit
// mantissa) are combined in fp32: their products, the orthogonalisation
// update and per-lane partial sums (at most 128 nodes, 256 products per part:
// a 4096-node segment) are far more precise than the stored values; every
// reduction across lanes, CTAs and chunks stays FP64. complex64 and complex128 bases use FP64 throughout.
// (Widening to FP64 costs conversion-unit throughput: with bfloat16 the FP64
// dots saturated that unit in the Arnoldi kernel.)
template <typename C2> struct MathT {
    using T = double;
    using T2 = double2;
};
template <> struct MathT<bf2> {
    using T = float;
    using T2 = float2;
};
__device__ __forceinline__ float2 to_f(bf2 a) { return bf2_to_f2(a); }

// d = a * b + c on two fp32 lanes at once (PTX fma.rn.f32x2, sm_100)
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(d)
        : "l"(*reinterpret_cast<const unsigned long long*>(&a)),
          "l"(*reinterpret_cast<const unsigned long long*>(&b)),
          "l"(*reinterpret_cast<const unsigned long long*>(&c)));
    return *reinterpret_cast<const float2*>(&d);
}

// A float widened to double, scaled by 2^-896: the exponent field is moved,
// not rebiased, which is exact for every finite value (zeros and denormals
// included). Integer instructions: F2F.F64.F32 runs at 16 lanes per clock and
// SM and bounded the complex64 passes (2 per value and pass). The other factor
// of a product carries 2^896, or the sum is scaled back. Infinities and NaN
// turn finite here, so sums over a basis vector formed this way only count once
// its norm, from the unscaled values, has been found finite. The per-pass
// kernels know it before; in the cycle kernel it arrives with the sums of the
// newest vector, and they are dropped if it is not. w is converted by F2F, once
// per step.
__device__ __forceinline__ double widen_scaled(unsigned f) {
    const long long t = (long long)(int)f * (1LL << 29);
    return __hiloint2double(int(t >> 32) & int(0x8fffffff), int(t));
}
constexpr double kScaleUp = 0x1p896, kScaleDown = 0x1p-896;

// Dots of w with several basis vectors at once: the 16-byte loads of w (shared
// memory) serve kDotVecs vectors.
constexpr int kDotVecs = 4;  // vectors of one dots task (they share its loads of w)
// w in shared memory as the dots read it: packed bfloat16, or FP64.
template <typename S> struct DotW { using T = S; };
template <> struct DotW<float2> { using T = double2; };

// the stored row value as the dots read it
__device__ __forceinline__ bf2 dot_value(bf2 y) { return y; }
__device__ __forceinline__ double2 dot_value(double2 y) { return y; }
__device__ __forceinline__ double2 dot_value(float2 y) {
    return make_double2(double(y.x) * kScaleUp, double(y.y) * kScaleUp);
}

// w of one 16-byte load's nodes, from shared memory to registers
template <typename S> struct UnitW;
template <> struct UnitW<bf2> {
    uint4 y;
    __device__ __forceinline__ explicit UnitW(const bf2* p) : y(*reinterpret_cast<const uint4*>(p)) {}
};
template <> struct UnitW<float2> {
    double2 y[2];
    __device__ __forceinline__ explicit UnitW(const double2* p) : y{p[0], p[1]} {}
};
template <> struct UnitW<double2> {
    double2 y;
    __device__ __forceinline__ explicit UnitW(const double2* p) : y(p[0]) {}
};
// re, im += conj(v) w over the nodes of one 16-byte load
__device__ __forceinline__ void unit_dot(uint4 v, const UnitW<bf2>& w, float& re, float& im) {
    float rr = re, ii = 0.f, ri = im, ir = 0.f;
    bf_mac(rr, ii, ri, ir, v.x, w.y.x);
    bf_mac(rr, ii, ri, ir, v.y, w.y.y);
    bf_mac(rr, ii, ri, ir, v.z, w.y.z);
    bf_mac(rr, ii, ri, ir, v.w, w.y.w);
    re = rr + ii;
    im = ri - ir;
}
__device__ __forceinline__ void unit_dot(uint4 v, const UnitW<float2>& w, double& re, double& im) {
    // (w carries the 2^896 of widen_scaled)
    const double2 a = make_double2(widen_scaled(v.x), widen_scaled(v.y));
    const double2 b = make_double2(widen_scaled(v.z), widen_scaled(v.w));
    re = fma(a.x, w.y[0].x, fma(a.y, w.y[0].y, fma(b.x, w.y[1].x, fma(b.y, w.y[1].y, re))));
    im = fma(a.x, w.y[0].y, fma(-a.y, w.y[0].x, fma(b.x, w.y[1].y, fma(-b.y, w.y[1].x, im))));
}
__device__ __forceinline__ void unit_dot(uint4 v, const UnitW<double2>& w, double& re, double& im) {
    const double2 a = *reinterpret_cast<const double2*>(&v);
    re = fma(a.x, w.y.x, fma(a.y, w.y.y, re));
    im = fma(a.x, w.y.y, fma(-a.y, w.y.x, im));
}

// Warp sums of the kDotVecs complex dots v of all lanes; every fourth lane
// holds the total of value `index`.
__device__ __forceinline__ double warp_sum_dots(double (&v)[2 * kDotVecs], int& index) {
    const int lane = threadIdx.x & 31;
    index = ((lane & 16) ? 4 : 0) + ((lane & 8) ? 2 : 0) + ((lane & 4) ? 1 : 0);
#pragma unroll
    for (int h = kDotVecs, bit = 16; h > 0; h >>= 1, bit >>= 1) {
        const bool hi = lane & bit;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const double keep = hi ? v[i + h] : v[i];
            const double send = hi ? v[i] : v[i + h];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
        }
    }
    double t = v[0] + __shfl_xor_sync(0xffffffffu, v[0], 2);
    return t + __shfl_xor_sync(0xffffffffu, t, 1);
}

}  // namespace usv
