// fw_fused.cu -- entry of the fused, temporally blocked FP32 form: checks
// that the configuration has a fused kernel and dispatches per model (the
// kernels are in fw_fused_kernel.cuh and fw_fused_tma.cuh, instantiated in
// fw_fused_{ap,ms,fk}.cu), and the weight repacking for the TMA kernel.
#include "fw_internal.cuh"

namespace fw {

namespace {

// out[p * NWO + q] = w[plane(q) * n + p], plane(q) skipping the centre.
template <int NWO, int CENTRE>
__global__ void k_pack(const float *__restrict__ w, int64_t n,
                       float *__restrict__ out)
{
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n;
         p += (int64_t)gridDim.x * blockDim.x) {
        float v[NWO];
#pragma unroll
        for (int q = 0; q < NWO; ++q) v[q] = w[(int64_t)(q < CENTRE ? q : q + 1) * n + p];
        float4 *o = reinterpret_cast<float4 *>(out + p * NWO);
#pragma unroll
        for (int q = 0; q < NWO / 4; ++q)
            o[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    }
}

}  // namespace

int step_fused(const fw_step_args *a, int64_t n_begin, int64_t n_steps,
               cudaStream_t stream)
{
    if (a->precision != FW_F32) {
        set_error("fw_step (fused): float32 only");
        return FW_ERR_UNSUPPORTED;
    }
    if (a->ni > (1 << 30) || a->nj > (1 << 30)) {
        set_error("fw_step (fused): grid too large");
        return FW_ERR_ARG;
    }
    switch (a->model) {
    case FW_MODEL_AP: return step_fused_ap(a, n_begin, n_steps, stream);
    case FW_MODEL_MS: return step_fused_ms(a, n_begin, n_steps, stream);
    case FW_MODEL_FK: return step_fused_fk(a, n_begin, n_steps, stream);
    case FW_MODEL_BK: return step_fused_bk(a, n_begin, n_steps, stream);
    }
    set_error("fw_step (fused): model %d has no fused form", a->model);
    return FW_ERR_UNSUPPORTED;
}

int pack_weights(int32_t stencil, const float *w, int64_t n, float *out,
                 cudaStream_t stream)
{
    if (!w || !out || n <= 0) {
        set_error("fw_pack_weights: null pointer or empty grid");
        return FW_ERR_ARG;
    }
    if (((uintptr_t)out & 15) != 0) {
        set_error("fw_pack_weights: output must be 16-byte aligned");
        return FW_ERR_ARG;
    }
    const int threads = 256;
    const int blocks = grid_for(n, threads);
    if (stencil == FW_STENCIL_ISO5)
        k_pack<4, 2><<<blocks, threads, 0, stream>>>(w, n, out);
    else if (stencil == FW_STENCIL_ANISO9)
        k_pack<8, 4><<<blocks, threads, 0, stream>>>(w, n, out);
    else {
        set_error("fw_pack_weights: 2D stencils only");
        return FW_ERR_UNSUPPORTED;
    }
    FW_CHECK_LAUNCH("k_pack");
    return FW_OK;
}

namespace {

// k_pack for padded rows, with the centre plane beside: one pass over the
// weights (40 B read, 36 written a node) where padding all planes first moved
// them twice.
template <int NWO, int CENTRE>
__global__ void __launch_bounds__(256)
    k_pack_rows(const float *__restrict__ w, int64_t ni, int64_t nj, int64_t pitch,
                float *__restrict__ out, float *__restrict__ centre)
{
    const int64_t n = ni * nj;
    for (int64_t i = blockIdx.y; i < ni; i += gridDim.y)
        for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < pitch;
             j += (int64_t)gridDim.x * blockDim.x) {
            float v[NWO], c = 0.f;
#pragma unroll
            for (int q = 0; q < NWO; ++q) v[q] = 0.f;
            if (j < nj) {
                const int64_t p = i * nj + j;
#pragma unroll
                for (int q = 0; q < NWO; ++q)
                    v[q] = w[(int64_t)(q < CENTRE ? q : q + 1) * n + p];
                c = w[(int64_t)CENTRE * n + p];
            }
            const int64_t o = i * pitch + j;
            float4 *d = reinterpret_cast<float4 *>(out + o * NWO);
#pragma unroll
            for (int q = 0; q < NWO / 4; ++q)
                d[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
            centre[o] = c;
        }
}

}  // namespace

int pack_rows(int32_t stencil, const float *w, int64_t ni, int64_t nj, int64_t pitch,
              float *out, float *centre, cudaStream_t stream)
{
    if (!w || !out || !centre || ni < 1 || nj < 1 || pitch < nj ||
        ((uintptr_t)out & 15) != 0) {
        set_error("fw_pack_rows: null or misaligned pointer, empty grid or pitch < nj");
        return FW_ERR_ARG;
    }
    const dim3 grid((unsigned)grid_for(pitch, 256, 64),
                    (unsigned)(ni < 4096 ? ni : 4096));
    if (stencil == FW_STENCIL_ISO5)
        k_pack_rows<4, 2><<<grid, 256, 0, stream>>>(w, ni, nj, pitch, out, centre);
    else if (stencil == FW_STENCIL_ANISO9)
        k_pack_rows<8, 4><<<grid, 256, 0, stream>>>(w, ni, nj, pitch, out, centre);
    else {
        set_error("fw_pack_rows: 2D stencils only");
        return FW_ERR_UNSUPPORTED;
    }
    FW_CHECK_LAUNCH("k_pack_rows");
    return FW_OK;
}

// ---- what a run does around its steps ------------------------------------------

namespace {

// 16 nodes a thread and round: their flags in one load, and the potentials
// only of groups that hold a non-myocyte.  Bound by memory: 42 us on 4096^2
// nodes at 20 % fibrosis, where index, gather and compare of whole arrays
// took 250 us and four host synchronisations.
template <class T>
__global__ void __launch_bounds__(256)
    k_nonmyo(const int8_t *__restrict__ myo, const T *__restrict__ u0,
             const T *__restrict__ u1, int64_t n, bool vec, int32_t *flag)
{
    const int64_t groups = (n + 15) / 16;
    bool bad = false;
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < groups;
         g += (int64_t)gridDim.x * blockDim.x) {
        const int64_t p0 = g * 16;
        alignas(16) int8_t m[16];
        if (vec && p0 + 16 <= n) {
            *reinterpret_cast<int4 *>(m) = *reinterpret_cast<const int4 *>(myo + p0);
        } else {
            for (int q = 0; q < 16; ++q) m[q] = p0 + q < n ? myo[p0 + q] : 1;
        }
#pragma unroll
        for (int q = 0; q < 16; ++q)
            if (!m[q]) bad |= !(u0[p0 + q] == u1[p0 + q]);
    }
    if (bad) *flag = 1;
}

constexpr int kRowsMax = 64;
struct RowsK {
    fw_rows c[kRowsMax];
};

// blockIdx.y: the copy; a warp a row at a time, in the widest words that
// both sides' alignment allows.
template <class W>
__device__ __forceinline__ void copy_words(const fw_rows &c)
{
    const int64_t words = c.row_bytes / (int64_t)sizeof(W);
    const int lane = threadIdx.x & 31;
    for (int64_t r = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
         r < c.rows; r += (int64_t)gridDim.x * (blockDim.x >> 5)) {
        const W *s = reinterpret_cast<const W *>((const char *)c.src + r * c.src_pitch);
        W *d = reinterpret_cast<W *>((char *)c.dst + r * c.dst_pitch);
        int64_t q = lane;
        for (; q + 96 < words; q += 128) {   // four loads under way a lane
            const W a = s[q], b = s[q + 32], c2 = s[q + 64], e = s[q + 96];
            d[q] = a;
            d[q + 32] = b;
            d[q + 64] = c2;
            d[q + 96] = e;
        }
        for (; q < words; q += 32) d[q] = s[q];
    }
}

__global__ void __launch_bounds__(256) k_rows(const __grid_constant__ RowsK k)
{
    const fw_rows &c = k.c[blockIdx.y];
    const uint64_t a = (uint64_t)c.src | (uint64_t)c.dst | (uint64_t)c.row_bytes |
                       (uint64_t)c.src_pitch | (uint64_t)c.dst_pitch;
    if (a % 16 == 0) copy_words<int4>(c);
    else if (a % 4 == 0) copy_words<int32_t>(c);
    else copy_words<int8_t>(c);
}

}  // namespace

int nonmyo_differ(const int8_t *myo, const void *u0, const void *u1,
                  int32_t precision, int64_t n, int32_t *flag, cudaStream_t stream)
{
    if (!myo || !u0 || !u1 || !flag || n < 1 ||
        (precision != FW_F64 && precision != FW_F32)) {
        set_error("fw_nonmyo_differ: null pointer, empty grid or unknown precision");
        return FW_ERR_ARG;
    }
    const bool vec = ((uintptr_t)myo & 15) == 0;
    const int blocks = grid_for((n + 15) / 16, 256);
    if (precision == FW_F64)
        k_nonmyo<double><<<blocks, 256, 0, stream>>>(myo, (const double *)u0,
                                                     (const double *)u1, n, vec, flag);
    else
        k_nonmyo<float><<<blocks, 256, 0, stream>>>(myo, (const float *)u0,
                                                    (const float *)u1, n, vec, flag);
    FW_CHECK_LAUNCH("k_nonmyo");
    return FW_OK;
}

int copy_rows(const fw_rows *copies, int32_t n, cudaStream_t stream)
{
    if (n < 0 || (n > 0 && !copies)) {
        set_error("fw_copy_rows: NULL copies");
        return FW_ERR_ARG;
    }
    for (int32_t i = 0; i < n; ++i) {
        const fw_rows &c = copies[i];
        if (!c.src || !c.dst || c.rows < 0 || c.row_bytes < 0 ||
            c.src_pitch < c.row_bytes || c.dst_pitch < c.row_bytes) {
            set_error("fw_copy_rows: copy %d has a null pointer or a pitch below "
                      "its rows", i);
            return FW_ERR_ARG;
        }
    }
    for (int32_t i = 0; i < n; i += kRowsMax) {
        RowsK k;
        const int m = n - i < kRowsMax ? n - i : kRowsMax;
        int64_t rows = 0;
        for (int q = 0; q < m; ++q) {
            k.c[q] = copies[i + q];
            if (k.c[q].rows > rows) rows = k.c[q].rows;
        }
        if (rows == 0) continue;
        const dim3 grid((unsigned)grid_for(rows, 8, 512), (unsigned)m);
        k_rows<<<grid, 256, 0, stream>>>(k);
        FW_CHECK_LAUNCH("k_rows");
    }
    return FW_OK;
}

}  // namespace fw
