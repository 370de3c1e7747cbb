// hmc.cu -- device-resident pieces around the likelihood for HMC sampling of
// many patches at once: the scene-parameter transform, proposal construction
// with on-device spline amplitudes, lnp and its gradient, and the leapfrog /
// Metropolis updates.  Every launch is asynchronous on the caller's stream and
// reads its scalars from device memory, so a whole trajectory (16 leapfrog
// steps = ~100 launches) is captured once into a CUDA graph and replayed.
//
// Host-side counterparts in the reference: Galaxy.proposal with scipy
// RectBivariateSpline amplitudes (forcepho/sources.py:607-681),
// FastPosterior.evaluate / stack_grad (forcepho/model.py:302-387),
// BoundedTransform (forcepho/model.py:596-637); the sampler itself is
// littlemcmc's NUTS driven by fitting.run_lmc (forcepho/fitting.py:254-341),
// replaced here by fixed-length HMC with a diagonal mass matrix.

#include <math.h>

#include "fp_common.cuh"

namespace {

constexpr int HMC_THREADS = 128;
constexpr int MAXDEG = 5;

// The span l of x in the knots t of n coefficients and degree k: t[l] <= x <
// t[l+1], k <= l <= n-1, x == t[n] in the last one.  The lanes of `mask` compare
// `width` knots at a time; `lane` counts them from 0.
__device__ __forceinline__ int knot_span(const double *__restrict__ t, int n, int k, double x, unsigned mask, int lane,
                                         int width)
{
    int below = 0;
    for (int i0 = 0; i0 <= n; i0 += width) {
        const int i = i0 + lane;
        below += __popc(__ballot_sync(mask, i <= n && t[i] <= x) & mask);
    }
    return max(k, min(n - 1, below - 1));
}

// Nonzero B-spline basis functions of degree k at x, and their derivatives, on
// the knot vector t with x in span l.  Cox-de Boor recurrence (de Boor, "A
// Practical Guide to Splines", ch. X).  DEG > 0: k = DEG is known, and the
// arrays stay in registers.
template <int DEG>
__device__ __forceinline__ void bspline_basis(const double *__restrict__ t, int l, int deg, double x, double *N,
                                              double *dN)
{
    const int k = DEG > 0 ? DEG : deg;
    double left[MAXDEG + 1], right[MAXDEG + 1], lower[MAXDEG + 1];
    N[0] = 1.0;
#pragma unroll
    for (int j = 1; j <= k; ++j) {
        left[j] = x - t[l + 1 - j];
        right[j] = t[l + j] - x;
        double saved = 0.0;
#pragma unroll
        for (int r = 0; r < j; ++r) {
            const double tmp = N[r] / (right[r + 1] + left[j - r]);
            N[r] = saved + right[r + 1] * tmp;
            saved = left[j - r] * tmp;
        }
        N[j] = saved;
        if (j == k - 1) {
#pragma unroll
            for (int r = 0; r <= j; ++r) lower[r] = N[r];
        }
    }
    if (k == 1) lower[0] = 1.0;
    // d/dx N_{i,k} = k (N_{i,k-1} / (t_{i+k} - t_i) - N_{i+1,k-1} / (t_{i+k+1} - t_{i+1}))
    // with N_{i,k-1} for i = l-k+1 .. l held in lower[0..k-1]
#pragma unroll
    for (int r = 0; r <= k; ++r) {
        const int i = l - k + r;
        double d = 0.0;
        if (r >= 1) {
            const double den = t[i + k] - t[i];
            if (den > 0.0) d += lower[r - 1] / den;
        }
        if (r <= k - 1) {
            const double den = t[i + k + 1] - t[i + 1];
            if (den > 0.0) d -= lower[r] / den;
        }
        dN[r] = k * d;
    }
}

__device__ __forceinline__ double sigm(double z) { return 1.0 / (1.0 + exp(-z)); }

// --------------------------------------------------------------------------
// transform + proposal: one warp per (patch, source)
// --------------------------------------------------------------------------
// Latency bounds it: a thread per source ran the transforms, two knot searches,
// the recurrences' divisions and 160 coefficient loads one after another, 20-24
// us whatever the batch.  Here the lanes share the parameters, the knots (one
// ballot per 16), the two axes (half a warp each) and the radii: 5.2 us for 12
// sources, 5.5 us for 60.
constexpr int PREPARE_WARPS = 2;

template <int DEG>
__global__ void __launch_bounds__(32 * PREPARE_WARPS)
prepare_kernel(const fp_hmc_patch *__restrict__ hp, const double *z, const double *__restrict__ lower,
               const double *__restrict__ upper, fp_spline_table tab, fp_source *__restrict__ props, double *theta,
               double *__restrict__ jac)
{
    const int p = blockIdx.x, lane = threadIdx.x & 31;
    const int s = blockIdx.y * PREPARE_WARPS + (threadIdx.x >> 5);
    const fp_hmc_patch P = hp[p];
    if (s >= P.n_sources) return;               // the whole warp
    const int nb = P.n_bands, nper = nb + NPARAMS - 1;
    const int64_t j0 = P.param_offset + (int64_t)s * nper;
    fp_source *src = props + (size_t)p * MAXSOURCES + s;
    const auto value = [&](int k, double *J) {
        const double zz = z[j0 + k];
        double q = zz;
        *J = 1.0;
        if (lower != nullptr) {
            const double rng = upper[j0 + k] - lower[j0 + k];
            const double sg = sigm(zz);
            q = lower[j0 + k] + rng * sg;
            *J = rng * sg * (1.0 - sg);
        }
        return q;
    };
    // sersic for the lower half of the warp, rhalf for the upper: read ahead of
    // the writes, as theta may lie where z does
    const int half = lane >> 4;
    double J;
    const double shape = value(nb + 4 + half, &J);
    __syncwarp();
    for (int k = lane; k < nper; k += 32) {
        const double q = value(k, &J);
        theta[j0 + k] = q;
        jac[j0 + k] = J;
        if (k < nb) src->fluxes[k] = (float)q;
        else (&src->ra)[k - nb] = (float)q;     // ra, dec, q, pa, nsersic, rh
    }
    for (int b = nb + lane; b < MAXBANDS; b += 32) src->fluxes[b] = 0.f;

    // A_r(sersic, rhalf) and its partial derivatives from the tensor-product
    // spline: the lower half of the warp forms the basis in sersic, the upper
    // half in rhalf.  x is clamped to the knots' range first, as FITPACK's
    // bispev/parder do (so does scipy).
    const int ncx = tab.nx - tab.kx - 1, ncy = tab.ny - tab.ky - 1;
    const double *t = half ? tab.ty : tab.tx;
    const int n = half ? ncy : ncx, k = half ? tab.ky : tab.kx;
    double N[MAXDEG + 1], dN[MAXDEG + 1];
    const double x = fmin(fmax(shape, t[k]), t[n]);
    const int l = knot_span(t, n, k, x, half ? 0xffff0000u : 0x0000ffffu, lane & 15, 16);
    bspline_basis<DEG>(t, l, k, x, N, dN);
    const int ix = __shfl_sync(0xffffffffu, l, 0) - tab.kx, iy = __shfl_sync(0xffffffffu, l, 16) - tab.ky;
    constexpr int TOP = DEG > 0 ? DEG : MAXDEG;
    double Nx[TOP + 1], dNx[TOP + 1], Ny[TOP + 1], dNy[TOP + 1];
#pragma unroll
    for (int u = 0; u <= TOP; ++u) {
        Nx[u] = __shfl_sync(0xffffffffu, N[u], 0);
        dNx[u] = __shfl_sync(0xffffffffu, dN[u], 0);
        Ny[u] = __shfl_sync(0xffffffffu, N[u], 16);
        dNy[u] = __shfl_sync(0xffffffffu, dN[u], 16);
    }
    if (lane >= MAXRADII) return;
    double a = 0.0, an = 0.0, ar = 0.0;
    if (lane < tab.n_radii) {
        const double *c = tab.coef + (size_t)lane * ncx * ncy;
#pragma unroll
        for (int u = 0; u <= TOP; ++u) {
            if (DEG == 0 && u > tab.kx) break;
            const double *row = c + (size_t)(ix + u) * ncy + iy;
            double sv = 0.0, sd = 0.0;
#pragma unroll
            for (int v = 0; v <= TOP; ++v) {
                if (DEG == 0 && v > tab.ky) break;
                sv += row[v] * Ny[v];
                sd += row[v] * dNy[v];
            }
            a += Nx[u] * sv;
            an += dNx[u] * sv;
            ar += Nx[u] * sd;
        }
    }
    src->mixture_amplitudes[lane] = (float)a;
    src->damplitude_dnsersic[lane] = (float)an;
    src->damplitude_drh[lane] = (float)ar;
}

// --------------------------------------------------------------------------
// lnp and dlnp/dz: one CTA per patch
// --------------------------------------------------------------------------
__device__ double block_sum(double v, double *sh)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) sh[w] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += sh[i];
    return t;   // valid in thread 0
}

__global__ void __launch_bounds__(HMC_THREADS)
lnprob_kernel(const fp_hmc_patch *__restrict__ hp, const double *__restrict__ z, const double *__restrict__ jac,
              const double *__restrict__ chi2, const fp_response *__restrict__ resp, int transformed, int sampling,
              double *__restrict__ lnp, double *__restrict__ grad)
{
    __shared__ double sh[HMC_THREADS / 32];
    const int p = blockIdx.x;
    const fp_hmc_patch P = hp[p];
    const int nb = P.n_bands, nper = nb + NPARAMS - 1;
    const int n = P.n_sources * nper;
    const fp_response *R = resp + (size_t)p * MAXBANDS;
    double logj = 0.0;
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        const int s = j / nper, k = j - s * nper;
        double g;
        if (k < nb) {
            g = (double)R[k].dchi2_dparam[s * NPARAMS];
        } else {
            g = 0.0;
            for (int b = 0; b < nb; ++b) g += (double)R[b].dchi2_dparam[s * NPARAMS + 1 + (k - nb)];
        }
        const int64_t jj = P.param_offset + j;
        double gz = -0.5 * g * jac[jj];
        if (transformed && sampling) {
            gz += 1.0 - 2.0 * sigm(z[jj]);
            logj += log(fabs(jac[jj]));
        }
        grad[jj] = gz;
    }
    const double lj = block_sum(logj, sh);
    if (threadIdx.x == 0) {
        double c = 0.0;
        for (int b = 0; b < nb; ++b) c += chi2[(size_t)p * MAXBANDS + b];
        lnp[p] = -0.5 * c + lj;
    }
}

// --------------------------------------------------------------------------
// vector-Jacobian product of the band chi2s: one CTA per patch
// --------------------------------------------------------------------------
// out[theta] = sum over bands of g[row] dchi2[row]/dtheta, from the rows that
// fetch_kernel copied: a flux moves its own band, a shape parameter every band.
__global__ void __launch_bounds__(HMC_THREADS)
vjp_kernel(const fp_hmc_patch *__restrict__ hp, const fp_result_row *__restrict__ rows,
           const int32_t *__restrict__ first_row, const double *__restrict__ g, int64_t g_stride,
           const float *__restrict__ grads, double *__restrict__ out)
{
    const int p = blockIdx.x;
    const fp_hmc_patch P = hp[p];
    const int nb = P.n_bands, nper = nb + NPARAMS - 1;
    const int64_t r0 = first_row[p];
    for (int j = threadIdx.x; j < P.n_sources * nper; j += blockDim.x) {
        const int s = j / nper, k = j - s * nper;
        const int b0 = k < nb ? k : 0, b1 = k < nb ? k + 1 : nb;
        const int col = s * NPARAMS + (k < nb ? 0 : 1 + (k - nb));
        double acc = 0.0;
        for (int b = b0; b < b1; ++b)
            acc += g[(r0 + b) * g_stride] * (double)grads[rows[r0 + b].grad_offset + col];
        out[P.param_offset + j] = acc;
    }
}

// --------------------------------------------------------------------------
// leapfrog and Metropolis: one CTA per patch; scalars from device memory
// --------------------------------------------------------------------------
// start of a trajectory: momentum from the pre-drawn normals, save (z, grad, lnp),
// H0 = -lnp + p^T M^-1 p / 2, then the first half kick and drift
__global__ void __launch_bounds__(HMC_THREADS)
begin_kernel(const fp_hmc_patch *__restrict__ hp, const fp_hmc_state st)
{
    __shared__ double sh[HMC_THREADS / 32];
    const int p = blockIdx.x;
    const fp_hmc_patch P = hp[p];
    const int n = P.n_sources * (P.n_bands + NPARAMS - 1);
    const int64_t traj = *st.traj % st.n_traj;
    const double eps = st.eps[p];
    double kin = 0.0;
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        const int64_t jj = P.param_offset + j;
        const double im = st.inv_mass[jj];
        const double mom = st.normals[traj * st.n_params + jj] / sqrt(im);
        kin += mom * mom * im;
        st.z0[jj] = st.z[jj];
        st.grad0[jj] = st.grad[jj];
        const double ph = mom + 0.5 * eps * st.grad[jj];
        st.p[jj] = ph;
        st.z[jj] += eps * im * ph;
    }
    const double k = block_sum(kin, sh);
    if (threadIdx.x == 0) {
        st.lnp0[p] = st.lnp[p];
        st.h0[p] = -st.lnp[p] + 0.5 * k;
    }
}

// between two gradient evaluations: full kick then drift
__global__ void __launch_bounds__(HMC_THREADS)
step_kernel(const fp_hmc_patch *__restrict__ hp, const fp_hmc_state st)
{
    const int p = blockIdx.x;
    const fp_hmc_patch P = hp[p];
    const int n = P.n_sources * (P.n_bands + NPARAMS - 1);
    const double eps = st.eps[p];
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        const int64_t jj = P.param_offset + j;
        const double ph = st.p[jj] + eps * st.grad[jj];
        st.p[jj] = ph;
        st.z[jj] += eps * st.inv_mass[jj] * ph;
    }
}

// end of a trajectory: last half kick, H1, accept with prob min(1, exp(H0 - H1))
// using the pre-drawn uniform, otherwise restore (z, grad, lnp)
__global__ void __launch_bounds__(HMC_THREADS)
end_kernel(const fp_hmc_patch *__restrict__ hp, int n_patches, const fp_hmc_state st)
{
    __shared__ double sh[HMC_THREADS / 32];
    __shared__ int s_acc;
    const int p = blockIdx.x;
    const fp_hmc_patch P = hp[p];
    const int n = P.n_sources * (P.n_bands + NPARAMS - 1);
    const int64_t traj = *st.traj % st.n_traj;
    const double eps = st.eps[p];
    double kin = 0.0;
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        const int64_t jj = P.param_offset + j;
        const double ph = st.p[jj] + 0.5 * eps * st.grad[jj];
        st.p[jj] = ph;
        kin += ph * ph * st.inv_mass[jj];
    }
    const double k = block_sum(kin, sh);
    if (threadIdx.x == 0) {
        const double h1 = -st.lnp[p] + 0.5 * k;
        const double du = st.uniforms[traj * n_patches + p];
        const double dh = st.h0[p] - h1;
        const int acc = isfinite(h1) && (log(du) < dh);
        s_acc = acc;
        st.accepted[p] += acc;
        st.energy_error[p] = dh;
        if (!acc) st.lnp[p] = st.lnp0[p];
    }
    __syncthreads();
    if (!s_acc) {
        for (int j = threadIdx.x; j < n; j += blockDim.x) {
            const int64_t jj = P.param_offset + j;
            st.z[jj] = st.z0[jj];
            st.grad[jj] = st.grad0[jj];
        }
    }
}

// advances the trajectory counter after end_kernel (a separate launch, so every
// CTA of end_kernel has read the current value)
__global__ void bump_kernel(int64_t *traj) { *traj += 1; }

}  // namespace

extern "C" int fp_hmc_prepare(const fp_hmc_patch *d_hp, int n_patches, const double *d_z, const double *d_lower,
                              const double *d_upper, const fp_spline_table *tab, fp_source *d_proposals,
                              double *d_theta, double *d_jac, void *stream)
{
    if (!d_hp || n_patches < 1 || !d_z || !tab || !d_proposals || !d_theta || !d_jac || (!d_lower != !d_upper))
        return fp_set_error(FP_ERR_ARGUMENT, "fp_hmc_prepare: bad arguments");
    if (tab->n_radii < 1 || tab->n_radii > MAXRADII || tab->kx < 1 || tab->kx > MAXDEG || tab->ky < 1 ||
        tab->ky > MAXDEG || tab->nx < 2 * tab->kx + 2 || tab->ny < 2 * tab->ky + 2 || !tab->tx || !tab->ty ||
        !tab->coef)
        return fp_set_error(FP_ERR_ARGUMENT, "fp_hmc_prepare: bad spline table");
    const dim3 blocks((unsigned)n_patches, (MAXSOURCES + PREPARE_WARPS - 1) / PREPARE_WARPS);
    if (tab->kx == 3 && tab->ky == 3)           // the bicubic splines of the amplitude table
        prepare_kernel<3><<<blocks, 32 * PREPARE_WARPS, 0, (cudaStream_t)stream>>>(d_hp, d_z, d_lower, d_upper, *tab,
                                                                                   d_proposals, d_theta, d_jac);
    else
        prepare_kernel<0><<<blocks, 32 * PREPARE_WARPS, 0, (cudaStream_t)stream>>>(d_hp, d_z, d_lower, d_upper, *tab,
                                                                                   d_proposals, d_theta, d_jac);
    return fp_check_cuda(cudaGetLastError(), "prepare_kernel launch");
}

extern "C" int fp_hmc_lnprob(const fp_hmc_patch *d_hp, int n_patches, const double *d_z, const double *d_jac,
                             const double *d_chi2, const fp_response *d_response, int transformed, int sampling,
                             double *d_lnp, double *d_grad, void *stream)
{
    if (!d_hp || n_patches < 1 || !d_z || !d_jac || !d_chi2 || !d_response || !d_lnp || !d_grad)
        return fp_set_error(FP_ERR_ARGUMENT, "fp_hmc_lnprob: bad arguments");
    lnprob_kernel<<<n_patches, HMC_THREADS, 0, (cudaStream_t)stream>>>(d_hp, d_z, d_jac, d_chi2, d_response,
                                                                       transformed, sampling, d_lnp, d_grad);
    return fp_check_cuda(cudaGetLastError(), "lnprob_kernel launch");
}

extern "C" int fp_chi2_vjp(const fp_hmc_patch *d_hp, int n_patches, const fp_result_row *d_rows,
                           const int32_t *d_first_row, const double *d_g, int64_t g_stride, const float *d_grads,
                           double *d_out, void *stream)
{
    if (!d_hp || n_patches < 1 || !d_rows || !d_first_row || !d_g || g_stride < 0 || !d_grads || !d_out)
        return fp_set_error(FP_ERR_ARGUMENT, "fp_chi2_vjp: bad arguments");
    vjp_kernel<<<n_patches, HMC_THREADS, 0, (cudaStream_t)stream>>>(d_hp, d_rows, d_first_row, d_g, g_stride, d_grads,
                                                                    d_out);
    return fp_check_cuda(cudaGetLastError(), "vjp_kernel launch");
}

extern "C" int fp_hmc_leapfrog(const fp_hmc_patch *d_hp, int n_patches, const fp_hmc_state *state, int stage,
                               void *stream)
{
    if (!d_hp || n_patches < 1 || !state || state->n_traj < 1)
        return fp_set_error(FP_ERR_ARGUMENT, "fp_hmc_leapfrog: bad arguments");
    cudaStream_t st = (cudaStream_t)stream;
    if (stage == FP_HMC_BEGIN) {
        begin_kernel<<<n_patches, HMC_THREADS, 0, st>>>(d_hp, *state);
    } else if (stage == FP_HMC_STEP) {
        step_kernel<<<n_patches, HMC_THREADS, 0, st>>>(d_hp, *state);
    } else if (stage == FP_HMC_END) {
        end_kernel<<<n_patches, HMC_THREADS, 0, st>>>(d_hp, n_patches, *state);
        if (int rc = fp_check_cuda(cudaGetLastError(), "end_kernel launch")) return rc;
        bump_kernel<<<1, 1, 0, st>>>(state->traj);
    } else {
        return fp_set_error(FP_ERR_ARGUMENT, "fp_hmc_leapfrog: unknown stage %d", stage);
    }
    return fp_check_cuda(cudaGetLastError(), "leapfrog launch");
}
