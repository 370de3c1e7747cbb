// transfer.cu -- a batch's proposals from, and its results to, pinned host
// memory, one launch each way.
//
// The kernels read and write the host buffers directly (pinned memory is
// addressable from the device), and move only what exists: a patch's own
// source records rather than MAXSOURCES of them, and of each (patch, band) row
// the n_sources x NPARAMS derivatives.  A copy of the whole slots and two row
// gathers followed by two copies took 22 + 9 + 11 us of a 213 us evaluation of
// 128 small stamps; the two launches here take 7.3 + 6.0 us
// (48 field patches: 13.5 + 9.8 + 10.1 us against 11.2 + 8.4).

#include "fp_common.cuh"

namespace {

constexpr int TRANSFER_THREADS = 128;

// one CTA per patch: its records, 8 bytes a thread (264 = 33 x 8)
__global__ void __launch_bounds__(TRANSFER_THREADS)
upload_kernel(const fp_source *__restrict__ h_records, const int32_t *__restrict__ counts,
              fp_source *__restrict__ proposals)
{
    constexpr int WORDS = sizeof(fp_source) / 8;
    static_assert(sizeof(fp_source) % 8 == 0, "records are copied 8 bytes at a time");
    const int64_t base = (int64_t)blockIdx.x * MAXSOURCES * WORDS;
    const int n = min(counts[blockIdx.x], MAXSOURCES) * WORDS;
    const uint2 *src = reinterpret_cast<const uint2 *>(h_records) + base;
    uint2 *dst = reinterpret_cast<uint2 *>(proposals) + base;
    for (int i = threadIdx.x; i < n; i += TRANSFER_THREADS) dst[i] = src[i];
}

// one CTA per (patch, band) row
__global__ void __launch_bounds__(TRANSFER_THREADS)
fetch_kernel(const double *__restrict__ chi2, const fp_response *__restrict__ resp,
             const fp_result_row *__restrict__ rows, double *__restrict__ h_chi2, float *__restrict__ h_grad)
{
    const fp_result_row r = rows[blockIdx.x];
    const int n = min(r.n_sources, MAXSOURCES) * NPARAMS;
    const float *src = resp[r.row].dchi2_dparam;
    for (int i = threadIdx.x; i < n; i += TRANSFER_THREADS) h_grad[r.grad_offset + i] = src[i];
    if (threadIdx.x == 0) h_chi2[blockIdx.x] = chi2[r.row];
}

}  // namespace

extern "C" int fp_upload_proposals(const fp_source *h_records, const int32_t *d_counts, int n_patches,
                                   fp_source *d_proposals, void *stream)
{
    if (!h_records || !d_counts || n_patches < 1 || !d_proposals)
        return fp_set_error(FP_ERR_ARGUMENT, "fp_upload_proposals: bad arguments");
    if ((((uintptr_t)h_records) | ((uintptr_t)d_proposals)) & 7)
        return fp_set_error(FP_ERR_ARGUMENT, "fp_upload_proposals: records must be 8-byte aligned");
    upload_kernel<<<n_patches, TRANSFER_THREADS, 0, (cudaStream_t)stream>>>(h_records, d_counts, d_proposals);
    return fp_check_cuda(cudaGetLastError(), "upload_kernel launch");
}

extern "C" int fp_fetch_results(const double *d_chi2, const fp_response *d_response, const fp_result_row *d_rows,
                                int64_t n_rows, double *h_chi2, float *h_grad, void *stream)
{
    if (!d_chi2 || !d_response || !d_rows || n_rows < 0 || n_rows > INT32_MAX || !h_chi2 || !h_grad)
        return fp_set_error(FP_ERR_ARGUMENT, "fp_fetch_results: bad arguments");
    if (n_rows == 0) return FP_OK;
    fetch_kernel<<<(unsigned)n_rows, TRANSFER_THREADS, 0, (cudaStream_t)stream>>>(d_chi2, d_response, d_rows, h_chi2,
                                                                                 h_grad);
    return fp_check_cuda(cudaGetLastError(), "fetch_kernel launch");
}
