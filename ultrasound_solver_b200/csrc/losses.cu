// Focal losses and their field cotangents on the device (FP64), for
// dL = Re(g^H du) (the reference's convention, which is also torch's).
//
//   USV_LOSS_FOCAL_PRESSURE  FocalPressureLoss.evaluate
//        L = -w_t mean_targets |u_t| + 0.5 w_b mean |u|^2
//        (phase_adjoint_optimizer.py:210-270)
//   USV_LOSS_FOCAL_CONTRAST  FocalContrastLoss.evaluate
//        L = -w_t mean_targets |u_t| + w_s (max + T (log sum exp((|u|-max)/T)
//            - log n)) over the background mask (phase_adjoint_optimizer.py:283-364)
//   USV_LOSS_CONTRAST_RATIO  L = -|u_t|^2 / mean_mask |u|^2 (mean over targets
//        of |u_t|^2; the mask is the focal shell)
//
// A pass leaves one partial per CTA; every CTA of the next pass adds all of
// them itself (the same values in the same order everywhere), so no pass has a
// finishing launch: two launches (three with the soft maximum) instead of five
// (seven). At most kLossCtas CTAs keep that re-reading small. On a 63,000-node
// field the launches are the cost: a step of basis field, focal contrast with
// cotangent and phase gradient took 88.9 us, now 79.5 (64 complex64 columns; the
// rest is the host's calls). Results are deterministic; repeated target indices accumulate in target
// order like the reference.
#include <cmath>

#include "usv_internal.cuh"

namespace usv {

constexpr int kLossChunk = 4096;  // fewest nodes per CTA (and the unit of the workspace size)
constexpr int kLossCtas = 592;
constexpr int kLossTargets = 64;  // more targets are added by a launch of their own

struct LossArgs {
    int mode;
    double target_weight, background_weight, temperature, eps;
    long long n;
    int n_targets;
    long long chunk;  // nodes per CTA
};

// partial[cta] = {sum |u|^2, sum_mask |u|^2, max_mask |u|, count_mask}
__global__ void __launch_bounds__(256) k_loss_pass1(LossArgs a, const double2* u, const unsigned char* mask,
                                                    double4* partial) {
    __shared__ double sh[32];
    const long long n0 = blockIdx.x * a.chunk, n1 = min(n0 + a.chunk, a.n);
    double s_all = 0.0, s_m = 0.0, mx = 0.0, cnt = 0.0;
#pragma unroll 4
    for (long long i = n0 + threadIdx.x; i < n1; i += 256) {
        const double a2 = cabs2(u[i]);
        s_all += a2;
        if (!mask || mask[i]) {
            s_m += a2;
            mx = fmax(mx, sqrt(a2));
            cnt += 1.0;
        }
    }
    s_all = block_sum(s_all, sh);
    s_m = block_sum(s_m, sh);
    cnt = block_sum(cnt, sh);
    mx = block_max(mx, sh);
    if (threadIdx.x == 0) partial[blockIdx.x] = make_double4(s_all, s_m, mx, cnt);
}

// {sum |u|^2, sum_mask |u|^2, max_mask |u|, count_mask} over all CTAs of pass 1
__device__ __forceinline__ double4 loss_stat(const double4* partial, int ctas, double* sh) {
    double a = 0.0, b = 0.0, c = 0.0, d = 0.0;
    for (int q = threadIdx.x; q < ctas; q += blockDim.x) {
        const double4 p = partial[q];
        a += p.x;
        b += p.y;
        c = fmax(c, p.z);
        d += p.w;
    }
    a = block_sum(a, sh);
    b = block_sum(b, sh);
    d = block_sum(d, sh);
    c = block_max(c, sh);
    return make_double4(a, b, c, d);
}

// partial2[cta] = sum_mask exp((|u| - max)/T)
__global__ void __launch_bounds__(256) k_loss_pass2(LossArgs a, const double2* u, const unsigned char* mask,
                                                    const double4* partial, int ctas, double* partial2) {
    __shared__ double sh[32];
    const double mx = loss_stat(partial, ctas, sh).z;
    const long long n0 = blockIdx.x * a.chunk, n1 = min(n0 + a.chunk, a.n);
    double s = 0.0;
#pragma unroll 4
    for (long long i = n0 + threadIdx.x; i < n1; i += 256)
        if (!mask || mask[i]) s += exp((sqrt(cabs2(u[i])) - mx) / a.temperature);
    s = block_sum(s, sh);
    if (threadIdx.x == 0) partial2[blockIdx.x] = s;
}

// Target terms of the cotangent for target t.
__device__ __forceinline__ void add_target(const LossArgs& a, const double2* u, long long i, double shell,
                                           double2* cot) {
    const double2 v = u[i];
    double2 g;
    if (a.mode == USV_LOSS_CONTRAST_RATIO) {
        g = cscale(v, -2.0 / (shell * a.n_targets));
    } else {
        const double amp = sqrt(cabs2(v));
        g = cscale(v, -a.target_weight / a.n_targets / (amp + a.eps));
    }
    cot[i] = cadd(cot[i], g);
}

// The loss value (CTA 0) from the partials and the target samples, and each
// CTA's nodes of the field cotangent (cot may be NULL): background / mask terms
// elementwise, then the targets among them.
__global__ void __launch_bounds__(256) k_loss_cot(LossArgs a, const double2* u, const unsigned char* mask,
                                                  const long long* targets, const double4* partial,
                                                  const double* partial2, int ctas, double* out,
                                                  double2* cot) {
    __shared__ double sh[32];
    const double4 stat = loss_stat(partial, ctas, sh);
    double sexp = 0.0;
    if (a.mode == USV_LOSS_FOCAL_CONTRAST) {
        for (int q = threadIdx.x; q < ctas; q += blockDim.x) sexp += partial2[q];
        sexp = block_sum(sexp, sh);
    }
    double mean_amp = 0.0, mean_pow = 0.0;
    for (int t = threadIdx.x; t < a.n_targets; t += blockDim.x) {
        const double p = cabs2(u[targets[t]]);
        mean_amp += sqrt(p);
        mean_pow += p;
    }
    mean_amp = block_sum(mean_amp, sh) / a.n_targets;
    mean_pow = block_sum(mean_pow, sh) / a.n_targets;
    const double shell = stat.y / stat.w;  // mean_mask |u|^2
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        double loss;
        if (a.mode == USV_LOSS_FOCAL_PRESSURE) {
            loss = -a.target_weight * mean_amp;
            if (a.background_weight > 0) loss += 0.5 * a.background_weight * stat.x / double(a.n);
        } else if (a.mode == USV_LOSS_FOCAL_CONTRAST) {
            loss = -a.target_weight * mean_amp;
            loss += a.background_weight * (stat.z + a.temperature * (log(sexp) - log(stat.w)));
        } else {
            loss = -mean_pow / shell;
        }
        out[0] = loss;
        out[1] = mean_amp;
        out[2] = mean_pow;
    }
    if (!cot) return;
    const long long n0 = blockIdx.x * a.chunk, n1 = min(n0 + a.chunk, a.n);
#pragma unroll 2
    for (long long i = n0 + threadIdx.x; i < n1; i += 256) {
        const double2 v = u[i];
        double2 g = make_double2(0.0, 0.0);
        const bool in = !mask || mask[i];
        if (a.mode == USV_LOSS_FOCAL_PRESSURE) {
            if (a.background_weight > 0) g = cscale(v, a.background_weight / double(a.n));
        } else if (a.mode == USV_LOSS_FOCAL_CONTRAST) {
            if (in) {
                const double amp = sqrt(cabs2(v));
                const double p = exp((amp - stat.z) / a.temperature) / sexp;
                g = cscale(v, a.background_weight * p / (amp + a.eps));
            }
        } else if (in) {
            // d(-P/S)/du_i = P/S^2 dS,  S = sum_mask |u|^2 / count
            g = cscale(v, 2.0 * mean_pow / (shell * shell * stat.w));
        }
        cot[i] = g;
    }
    if (a.n_targets > kLossTargets) return;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int t = 0; t < a.n_targets; ++t)
            if (targets[t] >= n0 && targets[t] < n1) add_target(a, u, targets[t], shell, cot);
}

// Target terms of many targets, added in target order by one thread.
__global__ void __launch_bounds__(256) k_loss_targets(LossArgs a, const double2* u, const long long* targets,
                                                      const double4* partial, int ctas, double2* cot) {
    __shared__ double sh[32];
    const double4 stat = loss_stat(partial, ctas, sh);
    if (threadIdx.x == 0)
        for (int t = 0; t < a.n_targets; ++t) add_target(a, u, targets[t], stat.y / stat.w, cot);
}

}  // namespace usv

using namespace usv;

extern "C" {

int usv_loss_workspace_bytes(int64_t n, size_t* bytes) {
    if (n < 1 || !bytes) return USV_ERR_ARG;
    const long long nblk = (n + kLossChunk - 1) / kLossChunk;
    *bytes = sizeof(double4) * nblk + sizeof(double) * nblk + sizeof(double) * 8;
    return USV_OK;
}

int usv_loss(int mode, const void* field, int64_t n, const unsigned char* mask,
             const int64_t* targets, int n_targets, double target_weight,
             double background_weight, double temperature, double eps, double* value,
             void* cotangent, void* workspace, size_t workspace_bytes, void* stream) {
    if (!field || n < 1 || !targets || n_targets < 1 || !value || !workspace) return USV_ERR_ARG;
    if (mode < USV_LOSS_FOCAL_PRESSURE || mode > USV_LOSS_CONTRAST_RATIO) return USV_ERR_ARG;
    if (mode == USV_LOSS_FOCAL_CONTRAST && !(temperature > 0)) return USV_ERR_ARG;
    size_t need = 0;
    usv_loss_workspace_bytes(n, &need);
    if (workspace_bytes < need) return USV_ERR_WORKSPACE;
    long long chunk = (n + kLossCtas - 1) / kLossCtas;
    chunk = chunk < kLossChunk ? kLossChunk : (chunk + 255) / 256 * 256;
    const int ctas = int((n + chunk - 1) / chunk);  // at most n / kLossChunk, what the workspace holds
    double4* p1 = static_cast<double4*>(workspace);
    double* p2 = reinterpret_cast<double*>(p1 + ctas);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const double2* u = static_cast<const double2*>(field);
    const long long* tg = reinterpret_cast<const long long*>(targets);
    double2* cot = static_cast<double2*>(cotangent);
    LossArgs a{mode, target_weight, background_weight, temperature, eps, n, n_targets, chunk};
    k_loss_pass1<<<ctas, 256, 0, s>>>(a, u, mask, p1);
    if (mode == USV_LOSS_FOCAL_CONTRAST) k_loss_pass2<<<ctas, 256, 0, s>>>(a, u, mask, p1, ctas, p2);
    k_loss_cot<<<cot ? ctas : 1, 256, 0, s>>>(a, u, mask, tg, p1, p2, ctas, value, cot);
    if (cot && n_targets > kLossTargets) k_loss_targets<<<1, 256, 0, s>>>(a, u, tg, p1, ctas, cot);
    USV_CUDA_TRY(cudaGetLastError());
    return USV_OK;
}

}  // extern "C"
