// Scene set-up on the device: obstacle material blend, sinc_neumann aperture
// deposition, source right-hand sides, the phase gradient through the source
// columns and the material VJP.
//
// Parity:
//   usv_materials_blend   warp_utils.py:11-23 (blend), 57-73 (sphere SDF, h)
//   usv_source_masses     sinc_aperture.py:36-72 (bilinear unit-mass deposition)
//                         and the overlap checks of warp_utils.py:105-113
//   usv_source_rhs        sinc_aperture.py:75-85, warp_utils.py:118-120
//   usv_source_phase_grad phase_response_basis.py:208-253 with G = A^-1 B diag(a)
//   usv_material_vjp      conservative_helmholtz.py:151-175
#include <cmath>
#include <vector>

#include "usv_internal.cuh"

namespace usv {

__global__ void __launch_bounds__(256)
k_blend(int nx, int ny, int nz, double dx, const double* sdf, double cx, double cy, double cz,
        double radius, double width, double rho_o, double c_o, const double* rho_m,
        const double* c_m, double rho0, double c0, double* rho, double* c) {
    const long long N = (long long)nx * ny * nz;
    const double inv_rho_o = 1.0 / rho_o;
    const double comp_o = 1.0 / (rho_o * c_o * c_o);
    for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < N;
         n += (long long)gridDim.x * blockDim.x) {
        double d;
        if (sdf) {
            d = sdf[n];
        } else {
            const Node p = decode(n, nx, ny);
            const double x = p.i * dx - cx, y = p.j * dx - cy, z = p.k * dx - cz;
            d = sqrt(x * x + y * y + z * z) - radius;
        }
        double h;
        if (width > 0) {
            double t = fmin(fmax(d / width, -1.0), 1.0);
            h = 0.5 * (1.0 + t + sin(M_PI * t) / M_PI);
        } else {
            h = d > 0 ? 1.0 : 0.0;
        }
        const double rm = rho_m ? rho_m[n] : rho0;
        const double cm = c_m ? c_m[n] : c0;
        const double inv_rho = inv_rho_o + (1.0 / rm - inv_rho_o) * h;
        const double comp = comp_o + (1.0 / (rm * cm * cm) - comp_o) * h;
        rho[n] = 1.0 / inv_rho;
        c[n] = sqrt(inv_rho / comp);
    }
}

// Aperture deposition: one CTA per emitter gathers, in the reference's
// summation order (corner-major, then quadrature order), the bilinear masses
// that land on each node of the emitter's bounding box. Deterministic, no
// atomics on the masses.
//
// The order makes each node one chain of additions, so the parallelism is one
// warp per node. The grid cell of every quadrature point is found once per
// CTA (two FP64 divides per point) and the points are listed by cell in
// shared memory, in quadrature order (one warp per cell compacts the matching
// keys); a node's warp walks the lists of its four cells, forms 32 weights at
// a time, one per lane, and adds them in order. A box of more than kDepCells
// cells (an aperture wider than about 40 nodes) has no room for the lists: its
// warps scan the keys for each cell instead. Bounded by instruction issue;
// 256 emitters of 16384 points (96^3 scene): 16.4 ms with one thread per node
// testing every point against its node, 0.58 ms with the scan, 0.36 ms with
// the lists.
constexpr int kDepThreads = 512;
constexpr int kDepWarps = kDepThreads / 32;
constexpr int kDepBlock = 16384;        // quadrature points per pass
constexpr int kDepCells = 2048;
constexpr int kDepQueue = 128 + 32;     // one scan step appends at most 128 points
struct DepShared {
    double2 term[kDepWarps][32];
    int key[kDepBlock];                 // (cell x - x0 + 1) + (cell y - y0 + 1) (bw + 1), -1: outside
    int first[kDepCells + 1];           // list of cell c: points[first[c]] .. points[first[c + 1] - 1]
    union {
        unsigned short points[kDepBlock];
        unsigned short queue[kDepWarps][kDepQueue];
    };
};

// Positions (quadrature order) of the keys equal to `want` among the 128 from
// `k` on, four per lane: put(index, rank) for each; returns their number.
template <typename Put>
__device__ __forceinline__ int match_keys(const int* key, int k, int nk4, int want, Put&& put) {
    const int lane = threadIdx.x & 31;
    int4 kv = make_int4(-1, -1, -1, -1);
    if (k + 4 * lane < nk4) kv = *reinterpret_cast<const int4*>(key + k + 4 * lane);
    const bool h0 = kv.x == want, h1 = kv.y == want, h2 = kv.z == want, h3 = kv.w == want;
    if (!__any_sync(0xffffffffu, h0 || h1 || h2 || h3)) return 0;
    const unsigned below = (1u << lane) - 1u;
    const unsigned m0 = __ballot_sync(0xffffffffu, h0), m1 = __ballot_sync(0xffffffffu, h1);
    const unsigned m2 = __ballot_sync(0xffffffffu, h2), m3 = __ballot_sync(0xffffffffu, h3);
    int pos = __popc(m0 & below) + __popc(m1 & below) + __popc(m2 & below) + __popc(m3 & below);
    if (h0) put(k + 4 * lane, pos++);
    if (h1) put(k + 4 * lane + 1, pos++);
    if (h2) put(k + 4 * lane + 2, pos++);
    if (h3) put(k + 4 * lane + 3, pos++);
    return __popc(m0) + __popc(m1) + __popc(m2) + __popc(m3);
}

__global__ void __launch_bounds__(kDepThreads)
k_deposit(int nx, int ny, double dx, const double* centers, const double* qx,
          const double* qy, const double* qw, int q, double diameter, double* masses) {
    extern __shared__ __align__(16) unsigned char dep_smem[];
    DepShared& sm = *reinterpret_cast<DepShared*>(dep_smem);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int m = blockIdx.x;
    const double cx = centers[3 * m], cy = centers[3 * m + 1];
    const int x0 = int(floor((cx - 0.5 * diameter) / dx)) - 1;
    const int y0 = int(floor((cy - 0.5 * diameter) / dx)) - 1;
    const int x1 = int(floor((cx + 0.5 * diameter) / dx)) + 2;
    const int y1 = int(floor((cy + 0.5 * diameter) / dx)) + 2;
    const int bw = x1 - x0 + 1, bh = y1 - y0 + 1;
    const int cells = (bw + 1) * (bh + 1);
    const bool lists = cells <= kDepCells;
    double* col = masses + (long long)m * nx * ny;
    double2* term = sm.term[warp];
    for (int corner = 0; corner < 4; ++corner) {
        const int a = corner >> 1, b = corner & 1;
        for (int k0 = 0; k0 < q; k0 += kDepBlock) {
            const int nk = min(kDepBlock, q - k0), nk4 = (nk + 3) & ~3;
            if (corner == 0 || q > kDepBlock) {
                __syncthreads();  // every warp is done with the previous block
                if (lists)
                    for (int c = threadIdx.x; c <= cells; c += kDepThreads) sm.first[c] = 0;
                __syncthreads();
                for (int k = threadIdx.x; k < nk4; k += kDepThreads) {
                    int v = -1;
                    if (k < nk) {
                        // a node takes the point from the cells at its own and
                        // the previous index, so the box is widened by one cell
                        const long long rx = (long long)int(floor((cx + qx[k0 + k]) / dx)) - x0 + 1;
                        const long long ry = (long long)int(floor((cy + qy[k0 + k]) / dx)) - y0 + 1;
                        if (rx >= 0 && rx <= bw && ry >= 0 && ry <= bh) v = int(rx + ry * (bw + 1));
                    }
                    sm.key[k] = v;
                    if (lists && v >= 0) atomicAdd(&sm.first[v + 1], 1);
                }
                __syncthreads();
                if (lists) {
                    if (warp == 0) {  // counts to list starts
                        int run = 0;
                        for (int c0 = 1; c0 <= cells; c0 += 32) {
                            const int c = c0 + lane;
                            int v = c <= cells ? sm.first[c] : 0;
#pragma unroll
                            for (int o = 1; o < 32; o <<= 1) {
                                const int u = __shfl_up_sync(0xffffffffu, v, o);
                                if (lane >= o) v += u;
                            }
                            if (c <= cells) sm.first[c] = run + v;
                            run += __shfl_sync(0xffffffffu, v, 31);
                        }
                    }
                    __syncthreads();
                    for (int c = warp; c < cells; c += kDepWarps) {
                        int pos = sm.first[c];
                        const int end = sm.first[c + 1];
                        for (int k = 0; k < nk4 && pos < end; k += 128)
                            pos += match_keys(sm.key, k, nk4, c, [&](int i, int rank) {
                                sm.points[pos + rank] = (unsigned short)i;
                            });
                    }
                    __syncthreads();
                }
            }
            for (int t = warp; t < bw * bh; t += kDepWarps) {
                const int ix = x0 + t % bw, iy = y0 + t / bw;
                if (ix < 0 || iy < 0 || ix >= nx || iy >= ny) continue;
                const int want = (t % bw + 1 - a) + (t / bw + 1 - b) * (bw + 1);
                double acc = col[(long long)iy * nx + ix];
                auto add = [&](const unsigned short* list, int count) {  // count <= 32
                    if (lane < count) {
                        const int k = k0 + list[lane];
                        const double px = (cx + qx[k]) / dx, py = (cy + qy[k]) / dx;
                        const double fx = px - floor(px), fy = py - floor(py);
                        term[lane] = make_double2(qw[k] * (a ? fx : 1.0 - fx), b ? fy : 1.0 - fy);
                    }
                    __syncwarp();
                    if (count == 32) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) acc = fma(term[i].x, term[i].y, acc);
                    } else {
                        for (int i = 0; i < count; ++i) acc = fma(term[i].x, term[i].y, acc);
                    }
                    __syncwarp();
                };
                if (lists) {
                    const int end = sm.first[want + 1];
                    for (int i = sm.first[want]; i < end; i += 32) add(sm.points + i, min(32, end - i));
                } else {
                    unsigned short* queue = sm.queue[warp];
                    int n = 0;  // queued points
                    for (int k = 0; k < nk4; k += 128) {
                        const int got = match_keys(sm.key, k, nk4, want, [&](int i, int rank) {
                            queue[n + rank] = (unsigned short)i;
                        });
                        if (got == 0) continue;
                        n += got;
                        __syncwarp();
                        int head = 0;
                        for (; n - head >= 32; head += 32) add(queue + head, 32);
                        if (head > 0) {  // fewer than 32 left: move them to the front
                            n -= head;
                            const unsigned short v = lane < n ? queue[head + lane] : (unsigned short)0;
                            __syncwarp();
                            if (lane < n) queue[lane] = v;
                            __syncwarp();
                        }
                    }
                    if (n > 0) add(queue, n);
                }
                if (lane == 0) col[(long long)iy * nx + ix] = acc;
                __syncwarp();
            }
        }
    }
}

// flags: bit0 a deposited node lies in the PML, bit1 on a soft face
__global__ void k_source_check(int nx, int ny, int m_emitters, const double* masses,
                               const double2* Tx, const double2* Ty, const double2* Tz,
                               unsigned soft, int nz, int* flag) {
    // (a node counts as soon as one emitter deposits there, so every mass is
    // tested by itself: one load per thread instead of a loop over emitters)
    const long long nxy = (long long)nx * ny, total = nxy * m_emitters;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total;
         q += (long long)gridDim.x * blockDim.x) {
        if (fabs(masses[q]) <= 0) continue;
        const int n = int(q % nxy);
        const int i = n % nx, j = n / nx;
        if (Tx[i].y + Ty[j].y + Tz[0].y > 0) atomicOr(flag, 1);
        if (node_fixed(soft, i, j, 0, nx, ny, nz)) atomicOr(flag, 2);
    }
}

// Right-hand sides: the first `plane_ctas` CTAs of a column form its z = 0
// plane (one thread per node), the others clear kRhsZero nodes each. Bounded
// by the 16 B per node written.
constexpr int kRhsZero = 4096;
__global__ void __launch_bounds__(256)
k_source_rhs(long long nxy, long long N, int m_emitters, const double* masses,
             const double2* coeff, double scale, double2* rhs, long long ld, int plane_ctas) {
    const int b = blockIdx.y;
    const double2* cb = coeff + (long long)b * m_emitters;
    double2* out = rhs + b * ld;
    if (int(blockIdx.x) >= plane_ctas) {
        const long long z0 = nxy + (long long)(blockIdx.x - plane_ctas) * kRhsZero + threadIdx.x;
#pragma unroll
        for (int u = 0; u < kRhsZero / 256; ++u)
            if (z0 + 256 * u < N) out[z0 + 256 * u] = make_double2(0.0, 0.0);
        return;
    }
    const long long n = blockIdx.x * 256LL + threadIdx.x;
    if (n >= nxy) return;
    double2 acc = make_double2(0.0, 0.0);
    // sixteen masses in flight per thread; added in emitter order
    for (int m0 = 0; m0 < m_emitters; m0 += 16) {
        double w[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) w[u] = m0 + u < m_emitters ? masses[(m0 + u) * nxy + n] : 0.0;
#pragma unroll
        for (int u = 0; u < 16; ++u)
            if (w[u] != 0.0) acc = cadd(acc, cscale(cb[m0 + u], scale * w[u]));
    }
    out[n] = acc;
}

__global__ void __launch_bounds__(256)
k_source_grad(long long nxy, const double* masses, const double2* lam, const double* phases,
              const double* amps, double scale, double* grad) {
    __shared__ double sh[32];
    const int m = blockIdx.x;
    double re = 0.0, im = 0.0;
    for (long long n = threadIdx.x; n < nxy; n += blockDim.x) {
        const double w = masses[m * nxy + n];
        re += w * lam[n].x;
        im += w * lam[n].y;
    }
    re = block_sum(re, sh);
    im = block_sum(im, sh);
    if (threadIdx.x == 0) {
        // r = (B^H lam)_m ; grad = Re(conj(a r) * i e^{i phi})
        const double a = amps ? amps[m] : 1.0;
        const double rr = a * scale * re, ri = a * scale * im;
        double sp, cp;
        sincos(phases[m], &sp, &cp);
        // conj(r) * (i e^{i phi}) = (rr - i ri)(-sp + i cp); real part:
        grad[m] += -rr * sp + ri * cp;
    }
}

// dL = -Re(lambda^H dA u): mass, edge (density) and open-face terms.
__global__ void __launch_bounds__(256)
k_material_vjp(OpView<double> op, const double* rho, const double* c, double omega,
               double dx, int open_mask, const double2* u, const double2* lam_in,
               double* g_rho, double* g_c) {
    for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < op.n;
         n += (long long)gridDim.x * blockDim.x) {
        const Node p = decode(n, op.nx, op.ny);
        auto lam_at = [&](long long m, int i, int j, int k) {
            return node_fixed(op.soft, i, j, k, op.nx, op.ny, op.nz) ? make_double2(0.0, 0.0)
                                                                      : lam_in[m];
        };
        const double r = rho[n], cc = c[n];
        const double2 un = u[n];
        const double2 ln = lam_at(n, p.i, p.j, p.k);
        const double2 tx = op.T[0][p.i], ty = op.T[1][p.j], tz = op.T[2][p.k];
        const double2 mass = cscale(cmul(cmul(tx, ty), tz), omega * omega / (r * cc * cc));
        const double2 prod = cmul(cmulc(ln, un), mass);
        double gr = prod.x / r;
        double gc = 2.0 * prod.x / cc;
        const double2 fyz = cmul(ty, tz), fxz = cmul(tx, tz), fxy = cmul(tx, ty);
        auto edge = [&](long long m, int i, int j, int k, double2 F) {
            const double s = r + rho[m];
            const double2 dr = cscale(F, -2.0 / (s * s));
            const double2 lm = lam_at(m, i, j, k);
            // (conj(l_lo) - conj(l_hi)) (u_hi - u_lo) is symmetric in lo/hi
            const double2 dl = make_double2(ln.x - lm.x, -(ln.y - lm.y));
            const double2 du = csub(u[m], un);
            gr += -cmul(cmul(dl, du), dr).x;
        };
        const long long sy = op.nx, sz = (long long)op.nx * op.ny;
        if (p.i > 0) edge(n - 1, p.i - 1, p.j, p.k, cmul(fyz, op.Q[0][p.i - 1]));
        if (p.i < op.nx - 1) edge(n + 1, p.i + 1, p.j, p.k, cmul(fyz, op.Q[0][p.i]));
        if (p.j > 0) edge(n - sy, p.i, p.j - 1, p.k, cmul(fxz, op.Q[1][p.j - 1]));
        if (p.j < op.ny - 1) edge(n + sy, p.i, p.j + 1, p.k, cmul(fxz, op.Q[1][p.j]));
        if (p.k > 0) edge(n - sz, p.i, p.j, p.k - 1, cmul(fxy, op.Q[2][p.k - 1]));
        if (p.k < op.nz - 1) edge(n + sz, p.i, p.j, p.k + 1, cmul(fxy, op.Q[2][p.k]));
        const int coord[3] = {p.i, p.j, p.k};
        const int dims[3] = {op.nx, op.ny, op.nz};
        for (int f = 0; f < 6; ++f) {
            if (!(open_mask & (1 << f))) continue;
            const int axis = f >> 1;
            if (coord[axis] != ((f & 1) ? dims[axis] - 1 : 0)) continue;
            const double2 area = cscale(axis == 0 ? fyz : (axis == 1 ? fxz : fxy), 1.0 / dx);
            const double2 term = cmul(make_double2(0.0, omega), cscale(area, 1.0 / (r * cc)));
            const double contrib = cmul(cmulc(ln, un), term).x;
            gr += contrib / r;
            gc += contrib / cc;
        }
        g_rho[n] = gr;
        g_c[n] = gc;
    }
}

static unsigned grid1(long long n) {
    long long b = (n + 255) / 256;
    if (b > 148LL * 32) b = 148LL * 32;
    return unsigned(b < 1 ? 1 : b);
}

}  // namespace usv

using namespace usv;

extern "C" {

int usv_materials_blend(const usv_scene* scene, const double* sdf, const double* center,
                        double radius, double width, double rho_obstacle, double c_obstacle,
                        const double* rho_medium, const double* c_medium, double rho0, double c0,
                        double* rho, double* c, void* stream) {
    if (!scene || !rho || !c) return USV_ERR_ARG;
    if (!sdf && (!center || !(radius >= 0))) return USV_ERR_ARG;
    if (!(width >= 0) || !std::isfinite(width) || !(rho_obstacle > 0) || !(c_obstacle > 0))
        return USV_ERR_ARG;
    const usv_scene& s = *scene;
    const long long N = (long long)s.nx * s.ny * s.nz;
    const double cx = center ? center[0] : 0, cy = center ? center[1] : 0,
                 cz = center ? center[2] : 0;
    k_blend<<<grid1(N), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        s.nx, s.ny, s.nz, s.dx, sdf, cx, cy, cz, radius, width, rho_obstacle, c_obstacle,
        rho_medium, c_medium, rho0, c0, rho, c);
    USV_CUDA_TRY(cudaGetLastError());
    return USV_OK;
}

// `masses` holds nx*ny*M doubles followed by one spare double used as the
// check-flag word; `op_buf` must be built for the same scene (PML tables).
int usv_source_masses(const usv_scene* scene, const void* op_buf,
                              const double* centers_host, const double* centers_dev,
                              int m_emitters, double diameter, const double* quad_x,
                              const double* quad_y, const double* quad_w, int q_points,
                              double* masses, void* stream) {
    if (!scene || !op_buf || !centers_host || !centers_dev || m_emitters < 1 || !quad_x ||
        !quad_y || !quad_w || q_points < 1 || !masses)
        return USV_ERR_ARG;
    const usv_scene& s = *scene;
    if (s.nx < 3 || s.ny < 3 || !(diameter > 0) || !std::isfinite(diameter)) return USV_ERR_ARG;
    const double ex = (s.nx - 1) * s.dx, ey = (s.ny - 1) * s.dx;
    for (int m = 0; m < m_emitters; ++m) {
        const double x = centers_host[3 * m], y = centers_host[3 * m + 1],
                     z = centers_host[3 * m + 2];
        if (!std::isfinite(x) || !std::isfinite(y) || !std::isfinite(z) || z != 0.0)
            return USV_ERR_ARG;
        if (x - diameter / 2 < s.dx || y - diameter / 2 < s.dx || x + diameter / 2 > ex - s.dx ||
            y + diameter / 2 > ey - s.dx)
            return USV_ERR_SOURCE_CLEARANCE;
    }
    cudaStream_t strm = static_cast<cudaStream_t>(stream);
    const long long nxy = (long long)s.nx * s.ny;
    USV_CUDA_TRY(cudaMemsetAsync(masses, 0, sizeof(double) * (nxy * m_emitters + 1), strm));
    USV_CUDA_TRY(cudaFuncSetAttribute(k_deposit, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      int(sizeof(DepShared))));
    k_deposit<<<m_emitters, kDepThreads, sizeof(DepShared), strm>>>(s.nx, s.ny, s.dx, centers_dev, quad_x,
                                                           quad_y, quad_w, q_points, diameter, masses);
    USV_CUDA_TRY(cudaGetLastError());
    const OpView<double> op = make_view<double>(s, op_buf, false);
    int* flag = reinterpret_cast<int*>(masses + nxy * m_emitters);
    k_source_check<<<grid1(nxy * m_emitters), 256, 0, strm>>>(s.nx, s.ny, m_emitters, masses, op.T[0],
                                                 op.T[1], op.T[2], op.soft, s.nz, flag);
    USV_CUDA_TRY(cudaGetLastError());
    int h = 0;
    USV_CUDA_TRY(cudaMemcpyAsync(&h, flag, sizeof(int), cudaMemcpyDeviceToHost, strm));
    USV_CUDA_TRY(cudaStreamSynchronize(strm));
    if (h & 1) return USV_ERR_SOURCE_PML;
    if (h & 2) return USV_ERR_SOURCE_SOFT;
    return USV_OK;
}

int usv_source_rhs(const usv_scene* scene, const double* masses, int m_emitters,
                   const double* coeff, double rho_ref, void* rhs, int nrhs, int64_t ld,
                   void* stream) {
    if (!scene || !masses || m_emitters < 1 || !coeff || !rhs || nrhs < 1 || nrhs > 65535 ||
        !(rho_ref > 0))
        return USV_ERR_ARG;
    const usv_scene& s = *scene;
    const long long N = (long long)s.nx * s.ny * s.nz, nxy = (long long)s.nx * s.ny;
    if (ld < N) return USV_ERR_ARG;
    const double scale = -2.0 * M_PI / (rho_ref * s.dx * s.dx * s.dx);
    const long long plane_ctas = (nxy + 255) / 256;
    const long long zero_ctas = (N - nxy + kRhsZero - 1) / kRhsZero;
    dim3 grid(unsigned(plane_ctas + zero_ctas), nrhs);
    k_source_rhs<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        nxy, N, m_emitters, masses, reinterpret_cast<const double2*>(coeff), scale,
        static_cast<double2*>(rhs), ld, int(plane_ctas));
    USV_CUDA_TRY(cudaGetLastError());
    return USV_OK;
}

int usv_source_phase_grad(const usv_scene* scene, const double* masses, int m_emitters,
                          const void* lam, const double* phases, const double* amplitudes,
                          double rho_ref, double* grad, void* stream) {
    if (!scene || !masses || m_emitters < 1 || !lam || !phases || !grad || !(rho_ref > 0))
        return USV_ERR_ARG;
    const usv_scene& s = *scene;
    const double scale = -2.0 * M_PI / (rho_ref * s.dx * s.dx * s.dx);
    k_source_grad<<<m_emitters, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        (long long)s.nx * s.ny, masses, static_cast<const double2*>(lam), phases, amplitudes,
        scale, grad);
    USV_CUDA_TRY(cudaGetLastError());
    return USV_OK;
}

int usv_material_vjp(const usv_scene* scene, const void* op_buf, const double* rho,
                     const double* c, const void* field, const void* adjoint, double* grad_rho,
                     double* grad_c, void* stream) {
    if (!scene || !op_buf || !rho || !c || !field || !adjoint || !grad_rho || !grad_c)
        return USV_ERR_ARG;
    const usv_scene& s = *scene;
    int open_mask = 0;
    for (int f = 0; f < 6; ++f)
        if (s.face_kind[f] == USV_FACE_OPEN) open_mask |= 1 << f;
    const OpView<double> op = make_view<double>(s, op_buf, false);
    k_material_vjp<<<grid1(op.n), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        op, rho, c, s.omega, s.dx, open_mask, static_cast<const double2*>(field),
        static_cast<const double2*>(adjoint), grad_rho, grad_c);
    USV_CUDA_TRY(cudaGetLastError());
    return USV_OK;
}

}  // extern "C"
