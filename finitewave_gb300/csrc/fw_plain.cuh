// fw_plain.cuh -- kernels and host loop of the plain form of the monodomain
// step (one launch per time step) and of the stand-alone ionic pass, as
// templates over the model M, the stencil ST and the precision T.  Each
// translation unit that instantiates them picks its own FMA policy: the
// float64 path of the reference's +,-,*,/-only models is compiled with
// --fmad=false so that it is bitwise the reference's.
//
// Per time step n (core/model/cardiac_model.py:164-178):
//   1. k_stim      once per stimulus whose step window contains n, on u_cur
//   2. k_step      all nodes: trackers read u_cur (after stimuli, before the
//                  update, as tracker_next does after the kernels but before
//                  the swap); myocytes get u_nxt = diffusion + ionic
//   3. k_probe     when a probe tracker of state variables is active at n:
//                  u_cur and the state (already advanced, as the reference's
//                  trackers see them); probes of u alone are sampled inside
//                  k_step
//   the caller's buffers then swap roles.
#pragma once

#include "fw_internal.cuh"
#include "fw_models.cuh"

namespace fw {
namespace {


constexpr int kThreads = 256;

template <class T>
struct StimK {
    const int8_t *mesh;
    const int8_t *mask;
    T *u;
    int64_t lo[3], ext[3];
    int64_t stride[3];
    int64_t count;
    double value, u_max;
    int kind, has_umax;
};

// StimVoltage*/StimCurrent* .stimulate (cpuwave2D/stimulation/*.py) over the
// stimulus box, restricted to mesh == 1 and the optional mask.
template <class T>
__global__ void k_stim(StimK<T> s)
{
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
         t < s.count; t += (int64_t)gridDim.x * blockDim.x) {
        int64_t c2 = t % s.ext[2];
        int64_t r = t / s.ext[2];
        int64_t c1 = r % s.ext[1];
        int64_t c0 = r / s.ext[1];
        int64_t p = (s.lo[0] + c0) * s.stride[0] + (s.lo[1] + c1) * s.stride[1] +
                    (s.lo[2] + c2) * s.stride[2];
        if (s.mesh[p] != 1) continue;
        if (s.mask && !s.mask[p]) continue;
        if (s.kind == FW_STIM_VOLTAGE) {
            s.u[p] = (T)s.value;
        } else {
            T x = s.u[p] + (T)s.value;
            if (s.has_umax && x > (T)s.u_max) x = (T)s.u_max;
            s.u[p] = x;
        }
    }
}

// Thresholds, parameters and dt are held in the kernel's precision T,
// rounded on the host: a float32 kernel then does no float64 conversions
// (GB300's float64 pipe is a small fraction of its float32 rate).
template <class T>
struct AtK {
    T thr;
    int32_t *act;
};

template <class T>
struct LatK {
    T thr;
    uint8_t *activated;
    int32_t *steps;
    int32_t *count;
    int32_t cap;
};

// A probe tracker's sample of the potential: out[c] = u[cells[c]].
struct UProbe {
    const int64_t *cells;
    double *out;
    int32_t n_cells;
};

template <class M, class T>
struct StepK {
    const int8_t *myo;
    const T *w;
    // FW_STENCIL_ANISO19_XY: the weights as distinct rows of 12 values
    // (planes 0-8, 11, 12, padding) and each node's row, or NULL
    const T *wrow;
    const int32_t *widx;
    const T *u;
    T *un;
    void *state[M::NS];
    T params[M::NP + M::ND];
    T dt;
    int64_t n, si, sj;
    // nodes in list order, myocytes first (NULL: every node in grid order);
    // the first n_myo of them step.  The launch's first `rest` CTAs show the
    // other nodes to the local activation trackers and, with rest_at, to the
    // activation trackers
    const int32_t *list;
    int32_t n_myo, rest;
    bool rest_at;
    int64_t step;
    int32_t n_at, n_lat;
    AtK<T> at[FW_MAX_AT];
    LatK<T> lat[FW_MAX_LAT];
    int32_t *status;
    // probes of the potential alone, sampled by the launch's last CTA
    int32_t n_up;
    UProbe up[FW_MAX_PROBE];
};

// isfinite on the bits: the comparison would take a turn of the float64 pipe
__device__ __forceinline__ bool finite_bits(double x)
{
    return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000;
}
__device__ __forceinline__ bool finite_bits(float x) { return isfinite(x); }

// True wherever x > y: the same comparison on the bits as integers, which
// most nodes fail, so that the float64 pipe is asked only about the others.
__device__ __forceinline__ bool maybe_above(double x, double y)
{
    long long a = __double_as_longlong(x), b = __double_as_longlong(y);
    a ^= (a >> 63) & 0x7fffffffffffffffll;
    b ^= (b >> 63) & 0x7fffffffffffffffll;
    return a > b;
}
__device__ __forceinline__ bool maybe_above(float, float) { return true; }

template <class M, class T>
__device__ __forceinline__ void track(const StepK<M, T> &k, int64_t p, T uc)
{
    for (int a = 0; a < k.n_at; ++a) {
        // (act_t < 0) & (u > threshold)  (activation_time_2d_tracker.py:61-63)
        if (maybe_above(uc, k.at[a].thr) && uc > k.at[a].thr && k.at[a].act[p] < 0)
            k.at[a].act[p] = (int32_t)k.step;
    }
    for (int l = 0; l < k.n_lat; ++l) {
        // cross_threshold (local_activation_time_2d_tracker.py:71-89)
        const LatK<T> &L = k.lat[l];
        uint8_t act = L.activated[p];
        if (uc >= L.thr && !act) {
            L.activated[p] = 1;
            int32_t c = L.count[p];
            if (c < L.cap)
                L.steps[(int64_t)c * k.n + p] = (int32_t)k.step;
            else if (k.status)
                atomicOr(k.status, FW_DEV_LAT_OVERFLOW);
            L.count[p] = c + 1;
        } else if (uc < L.thr && act) {
            L.activated[p] = 0;
        }
    }
}

// The trackers at the nodes that do not step, which follow the myocytes in
// the list: kRestNodes nodes a thread and round, whose loads are all under
// way before the first is used.
constexpr int kRestNodes = 4;
template <int N, class M, class T>
__device__ __forceinline__ void rest_nodes(const StepK<M, T> &k, int64_t t0)
{
    int64_t p[N];
    T u[N];
    bool look[N];   // a tracker has something to record
#pragma unroll
    for (int q = 0; q < N; ++q) p[q] = k.list[t0 + q * (int64_t)blockDim.x];
#pragma unroll
    for (int q = 0; q < N; ++q) {
        u[q] = k.u[p[q]];
        look[q] = k.rest_at;
    }
    for (int l = 0; l < k.n_lat; ++l) {
        uint8_t act[N];
#pragma unroll
        for (int q = 0; q < N; ++q) act[q] = k.lat[l].activated[p[q]];
#pragma unroll
        for (int q = 0; q < N; ++q)
            look[q] |= act[q] ? u[q] < k.lat[l].thr : u[q] >= k.lat[l].thr;
    }
#pragma unroll
    for (int q = 0; q < N; ++q)
        if (look[q]) track(k, p[q], u[q]);
}
// part `part` of `parts` of them
template <class M, class T>
__device__ __forceinline__ void track_rest(const StepK<M, T> &k, int part, int parts)
{
    const int64_t round = (int64_t)blockDim.x * kRestNodes;
    int64_t t0 = k.n_myo + part * round + threadIdx.x;
    for (; t0 + (kRestNodes - 1) * (int64_t)blockDim.x < k.n; t0 += parts * round)
        rest_nodes<kRestNodes>(k, t0);
    for (int q = 0; q < kRestNodes && t0 < k.n; ++q, t0 += blockDim.x)
        rest_nodes<1>(k, t0);
}

// Minimum resident CTAs per SM asked of the compiler for the float32
// k_step: models may set M::kMinBlocksF32 (the detailed models trade
// registers for the occupancy their memory latency needs); 1 otherwise.
template <class M, class T, class = void>
struct MinBlocks {
    static constexpr int value = 1;
};
template <class M>
struct MinBlocks<M, float, decltype(void(M::kMinBlocksF32))> {
    static constexpr int value = M::kMinBlocksF32;
};

// A model whose step is bound by arithmetic visits the myocytes through the
// node list: a warp of grid order spends a full warp's issue slots (and, in
// float64, a full warp's turn of the float64 pipe, two lanes a clock per SM)
// whatever the number of myocytes among its nodes.  Measured with 10-20 %
// fibrosis, list and one-warp CTAs against grid order and 256 threads:
// Aliev-Panfilov float64 600 x 601 30 against 35 us a step, TP06 float64
// 192 x 190 150 against 169 (reference-order update); with 256 threads on
// both sides, Courtemanche float32 511 x 387 12.8 against 13.6, TP06 float32
// 192^3 shell (19 % myocytes) 83 against 105.
// Below kListMinNodes (four warps an SM) the step's time is the latency of
// its loads, to which the list adds one: Aliev-Panfilov float64 100 x 100
// is 4 % slower with it.
constexpr int64_t kListMinNodes = 152 * 4 * 32;
template <class M, class T, class = void>
struct UseList {
    static constexpr bool value = sizeof(T) == 8;
};
template <class M, class T>
struct UseList<M, T, decltype(void(M::kMinBlocksF32))> {
    static constexpr bool value = true;
};

// Threads per CTA.  float64 steps are bound by the float64 pipe, so what
// counts is that every SM gets the same number of warps: one-warp CTAs, as
// many as the grid has, go to whichever SM is free.  Listed float32 steps
// launch kListThreadsF32 of the kThreads that the kernel is compiled for (its
// registers and the threads an SM holds stay as they are): the same fill, in
// halves, leaves less of the last round empty.  Us a step with 256, 128 and
// 64: Courtemanche 511 x 387 12.8, 12.0, 12.1, 700 x 700 24.2, 22.4, 22.4;
// TP06 500 x 501 10.6, 9.9, 9.9, 256 x 256 x 40 106, 104, 103, 100 x 100 x 20
// 9.5, 8.5, 8.7, 192^3 shell 83.0, 83.2, 83.9; with 32 TP06 500 x 501 takes
// 11.8 (an SM holds 32 CTAs at most).
constexpr int kListThreadsF32 = 128;
template <class T>
constexpr int step_threads()
{
    return sizeof(T) == 8 ? 32 : kThreads;
}

// Threads that show the other nodes to the trackers (track_rest), as CTAs
// before those that step: 512 an SM, so that myocytes step beside them while
// their loads are under way.  Us a step with one local activation tracker, in
// grid order, with the other nodes one a thread behind the myocytes, and so:
// TP06 float32 236^3 shell (7 % myocytes) 185, 211, 132, 192^3 shell (16 %)
// 132, 133, 89, Aliev-Panfilov float64 192^3 shell 327, 300, 139, 600 x 601
// (79 %) 41.4, 28.8, 29.0, TP06 float32 600 x 601 18.9, 10.7, 10.5; with 256
// an SM 186, 110, 139, 29.0, 10.5, with 1024 131, 94, 139, 29.0, 10.5.
constexpr int kRestThreads = 152 * 512;

// CTAs of a step.  Listed and float64 steps run one node per thread; the
// others loop over the grid with the resident CTAs.  Detailed float32 steps
// without a list as well: TP06 236^3 shell (7 % myocytes) 140 us a step, 175
// with one node per thread, Courtemanche 160^3 shell 108 against 126, TP06
// 200 x 200 x 40 60.8 against 59.4.
template <class T>
constexpr int step_blocks(bool listed)
{
    return listed || sizeof(T) == 8 ? 1 << 26 : 152 * 8;
}

template <class M, int ST, class T, bool LIST>
__global__ void __launch_bounds__(step_threads<T>(), (MinBlocks<M, T>::value))
    k_step(StepK<M, T> k)
{
    const Params<T, M::NP + M::ND> P = load_params<T, M::NP + M::ND>(k.params);
    const T dt = k.dt;
    const int64_t n = LIST ? (int64_t)k.n_myo : k.n;
    // Steps of one call follow one another with programmatic serialisation:
    // the next one's CTAs take their places, read their parameters and wait
    // here while this one's last CTAs run.  A float64 step lets them come
    // only when a CTA is done: placed earlier, in the slots that this step's
    // CTAs leave, they would not spread evenly over the SMs, whose float64
    // pipes set the time.  Us a step early and late: TP06 192 x 190 68 and 61,
    // in grid order 100 x 100 57.8 and 33.4, Aliev-Panfilov 100 x 100 3.9 and
    // 3.6, 130 x 140 5.9 and 3.9, 150 x 151 without a list 13.4 and 4.2,
    // Fenton-Karma 150 x 151 without a list 35 and 11.  With and without the
    // overlap: Courtemanche float32 511 x 387 12.8 and 14.5, Aliev-Panfilov
    // float32 256 x 240 x 60 59.8 and 61.8 and 320 x 300 4.0 and 5.8 (ECG
    // samples included), float64 600 x 601 with 20 % fibrosis 28.5 and 30.9.
    constexpr bool kLate = sizeof(T) == 8;
    if constexpr (!kLate) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (k.n_up && blockIdx.x == gridDim.x - 1) {
        for (int a = 0; a < k.n_up; ++a)
            for (int c = threadIdx.x; c < k.up[a].n_cells; c += blockDim.x)
                k.up[a].out[c] = (double)k.u[k.up[a].cells[c]];
        return;
    }
    int cta = (int)blockIdx.x, ctas = (int)gridDim.x - (k.n_up ? 1 : 0);
    if constexpr (LIST) {
        if (cta < k.rest) {
            track_rest(k, cta, k.rest);
            return;
        }
        cta -= k.rest;
        ctas -= k.rest;
    }
    const int64_t stride = (int64_t)ctas * blockDim.x;
    for (int64_t t = cta * (int64_t)blockDim.x + threadIdx.x; t < n; t += stride) {
        const int64_t p = LIST ? (int64_t)k.list[t] : t;
        T uc = k.u[p];
        if (k.n_at | k.n_lat) track(k, p, uc);
        if (!LIST && !k.myo[p]) continue;
        T un;
        if constexpr (ST == FW_STENCIL_ANISO19_XY) {
            if (k.wrow)
                un = diffuse_row_xy<T>(k.u, k.wrow + (int64_t)k.widx[p] * 12, p,
                                       k.si, k.sj);
            else
                un = diffuse_node<ST, T>(k.u, k.w, p, k.n, k.si, k.sj);
        } else {
            un = diffuse_node<ST, T>(k.u, k.w, p, k.n, k.si, k.sj);
        }
        auto st = M::template load<T>(k.state, p);
        un = M::template update<T>(uc, un, st, P, dt);
        M::template store<T>(k.state, p, st);
        k.un[p] = un;
        if (!finite_bits(un) && k.status) atomicOr(k.status, FW_DEV_NONFINITE);
    }
    if constexpr (kLate) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

struct ProbeOne {
    const int64_t *cells;
    double *out;
    int64_t sample;
    int64_t capacity;
    int32_t n_cells, n_vars;
    int32_t var_ids[FW_MAX_PROBE_VARS];
};

template <class T>
struct ProbeK {
    const T *u;
    void *state[FW_MAX_STATE];
    uint32_t f64_mask;
    uint32_t pair_mask;
    int32_t n;
    ProbeOne pr[FW_MAX_PROBE];
    int32_t *status;
};

template <class T>
__global__ void k_probe(ProbeK<T> k)
{
    for (int t = 0; t < k.n; ++t) {
        const ProbeOne &P = k.pr[t];
        if (P.sample >= P.capacity) {
            if (threadIdx.x == 0 && k.status)
                atomicOr(k.status, FW_DEV_PROBE_OVERFLOW);
            continue;
        }
        int total = P.n_cells * P.n_vars;
        for (int q = threadIdx.x; q < total; q += blockDim.x) {
            int v = q / P.n_cells, c = q % P.n_cells;
            int64_t p = P.cells[c];
            int id = P.var_ids[v];
            double x;
            if (id == 0)
                x = (double)k.u[p];
            else if ((k.f64_mask >> (id - 1)) & 1u)
                x = ((const double *)k.state[id - 1])[p];
            else if ((k.pair_mask >> (id - 1)) & 1u) {
                const float2 c = ((const float2 *)k.state[id - 1])[p];
                x = (double)c.x + (double)c.y;
            }
            else
                x = (double)((const T *)k.state[id - 1])[p];
            P.out[(P.sample * P.n_vars + v) * (int64_t)P.n_cells + c] = x;
        }
    }
}

// ECG leads (ecg_2d_tracker.py:114-153, ecg_3d_tracker.py:99-140): per
// myocyte the diffusion increment diffuse(u) - u weighted by 1 / (d dr),
// d the squared distance to the lead; per-thread partial sums in T, a block
// reduction in float64, one float64 atomic add per block and lead.
template <class T>
struct EcgK {
    const T *u;
    const T *w;
    const int8_t *myo;
    int64_t n, si, sj, nj, nk;
    int32_t dim, n_leads;
    T xyz[FW_MAX_ECG_LEADS][3];
    T dr;
    double *out;
};

template <int ST, class T>
__global__ void __launch_bounds__(kThreads) k_ecg(EcgK<T> k)
{
    T acc[FW_MAX_ECG_LEADS];
#pragma unroll
    for (int c = 0; c < FW_MAX_ECG_LEADS; ++c) acc[c] = (T)0;
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < k.n;
         p += (int64_t)gridDim.x * blockDim.x) {
        if (!k.myo[p]) continue;
        const T diff = diffuse_node<ST, T>(k.u, k.w, p, k.n, k.si, k.sj) - k.u[p];
        T fi, fj, fk;
        if (k.n <= INT32_MAX) {   // 32-bit divisions
            const uint32_t nk = k.dim == 2 ? 1u : (uint32_t)k.nk;
            const uint32_t ij = (uint32_t)p / nk, i = ij / (uint32_t)k.nj;
            fi = (T)i;
            fj = (T)(ij - i * (uint32_t)k.nj);
            fk = (T)((uint32_t)p - ij * nk);
        } else if (k.dim == 2) {
            fi = (T)(p / k.nj);
            fj = (T)(p % k.nj);
            fk = (T)0;
        } else {
            const int64_t plane = k.nj * k.nk, r = p % plane;
            fi = (T)(p / plane);
            fj = (T)(r / k.nk);
            fk = (T)(r % k.nk);
        }
#pragma unroll
        for (int c = 0; c < FW_MAX_ECG_LEADS; ++c) {
            if (c >= k.n_leads) break;
            const T dx = k.xyz[c][0] - fi, dy = k.xyz[c][1] - fj,
                    dz = k.xyz[c][2] - fk;
            const T d = dx * dx + dy * dy + dz * dz;
            if (d > (T)0) acc[c] += diff / (d * k.dr);
        }
    }
    // Warp sums of all leads at once: at each exchange a lane keeps half of
    // its leads and adds the partner's part of them, 4 + 2 + 1 float64
    // additions down to one lead a lane, then two more -- 9 turns of the
    // float64 pipe, 16 cycles each, where a tree per lead took 40.  With the
    // 32-bit divisions above, 1000 float32 steps of 320 x 300 nodes with a
    // sample every 10 take 3990 us, 4780 before.
    static_assert(FW_MAX_ECG_LEADS == 8, "three halvings");
    __shared__ double red[FW_MAX_ECG_LEADS][kThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double v[FW_MAX_ECG_LEADS];
#pragma unroll
    for (int c = 0; c < FW_MAX_ECG_LEADS; ++c) v[c] = (double)acc[c];
#pragma unroll
    for (int h = 4, o = 16; h >= 1; h >>= 1, o >>= 1) {
        const bool upper = (lane & o) != 0;   // keeps leads h .. 2h - 1
#pragma unroll
        for (int c = 0; c < h; ++c) {
            const double mine = upper ? v[c + h] : v[c], other = upper ? v[c] : v[c + h];
            v[c] = mine + __shfl_xor_sync(0xffffffffu, other, o);
        }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
    // lane 4 q holds lead q, its bits being the halves it kept
    if ((lane & 3) == 0) red[lane >> 2][warp] = v[0];
    __syncthreads();
    if (threadIdx.x < FW_MAX_ECG_LEADS && (int)threadIdx.x < k.n_leads) {
        double s = 0.0;
        for (int q = 0; q < kThreads / 32; ++q) s += red[threadIdx.x][q];
        atomicAdd(&k.out[threadIdx.x], s);
    }
}

template <int ST, class T>
int launch_ecg(const T *u, const T *w, const int8_t *myo, const Grid &g,
               int dim, const double (*coords)[3], int n_leads, double dr,
               double *out, cudaStream_t stream)
{
    if (n_leads < 1 || n_leads > FW_MAX_ECG_LEADS) {
        set_error("ECG: %d leads (1..%d)", n_leads, FW_MAX_ECG_LEADS);
        return FW_ERR_ARG;
    }
    EcgK<T> k;
    k.u = u;
    k.w = w;
    k.myo = myo;
    k.n = g.n;
    k.si = g.si;
    k.sj = g.sj;
    k.nj = g.nj;
    k.nk = g.nk;
    k.dim = dim;
    k.n_leads = n_leads;
    for (int c = 0; c < FW_MAX_ECG_LEADS; ++c)
        for (int a = 0; a < 3; ++a)
            k.xyz[c][a] = c < n_leads ? (T)coords[c][a] : (T)0;
    k.dr = (T)dr;
    k.out = out;
    k_ecg<ST, T><<<grid_for(g.n, kThreads, 152 * 8), kThreads, 0, stream>>>(k);
    FW_CHECK_LAUNCH("k_ecg");
    return FW_OK;
}

// Spiral-wave tips (spiral_wave_core_2d_tracker.py:88-249): the cell
// (i, j)-(i+1, j+1) holds a tip when the threshold isoline crosses it in
// both the previous and the current potential; the tip is the intersection
// of the two bilinear isolines inside the cell (_correct_tip_pos), found in
// float64.
template <class T>
struct TipK {
    const T *u_prev;
    const T *u;
    int64_t ni, nj, nk;   // slice (i, j) planes; k the z index (nk = 1 in 2D)
    double thr;
    fw_tip *out;
    int32_t *count;
    int64_t capacity;
    int32_t sample;
    int32_t *status;
};

template <class T>
__global__ void __launch_bounds__(kThreads) k_tips(TipK<T> k)
{
    const int64_t di = k.ni - 10, dj = k.nj - 10;
    if (di <= 0 || dj <= 0) return;
    const int64_t cells = di * dj * k.nk;
    const T thr = (T)k.thr;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
         t < cells; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t kk = t % k.nk;
        const int64_t r = t / k.nk;
        const int64_t j = 5 + r % dj, i = 5 + r / dj;
        // element (i, j) of z layer kk; rows of a layer are nj * nk apart
        const int64_t si = k.nj * k.nk, sj = k.nk;
        const int64_t p = i * si + j * sj + kk;
        // neighbours: (i+1, j) = p + si, (i, j+1) = p + sj
        const T *up = k.u_prev, *uc = k.u;
        auto crosses = [&](const T *u) {
            const T a = u[p], b = u[p + si], c = u[p + sj], d = u[p + si + sj];
            if (a >= thr && (b < thr || c < thr || d < thr)) return 1;
            if (a < thr && (b >= thr || c >= thr || d >= thr)) return 1;
            return 0;
        };
        int counter = crosses(up);
        if (counter == 1) counter += crosses(uc);
        if (counter != 2) continue;
        // _correct_tip_pos (spiral_wave_core_2d_tracker.py:98-146)
        const double u00 = up[p], u01 = up[p + sj], u10 = up[p + si],
                     u11 = up[p + si + sj];
        const double n00 = uc[p], n01 = uc[p + sj], n10 = uc[p + si],
                     n11 = uc[p + si + sj];
        const double th = k.thr;
        const double AC = u00 - u01 + u11 - u10;
        const double GC = u01 - u00;
        const double BC = u10 - u00;
        const double DC = u00 - th;
        const double AD = n00 - n01 + n11 - n10;
        const double GD = n01 - n00;
        const double BD = n10 - n00;
        const double DD = n00 - th;
        const double Q = BC * AD - BD * AC;
        const double R = GC * AD - GD * AC;
        const double S = DC * AD - DD * AC;
        const double QOnR = Q / R;
        const double SOnR = S / R;
        const double Tq = AC * QOnR;
        const double U = AC * SOnR - BC + GC * QOnR;
        const double V = GC * SOnR - DC;
        const double disc = U * U - 4. * Tq * V;
        if (disc < 0) continue;
        const double T2 = 2. * Tq;
        if (T2 == 0.) continue;
        const double sq = sqrt(disc);
        const double xn = (-U - sq) / T2, xp = (-U + sq) / T2;
        const double yn = -QOnR * xn - SOnR, yp = -QOnR * xp - SOnR;
        double cx, cy;
        if (0 <= xn && xn <= 1 && 0 <= yn && yn <= 1) {
            cx = xn;
            cy = yn;
        } else if (0 <= xp && xp <= 1 && 0 <= yp && yp <= 1) {
            cx = xp;
            cy = yp;
        } else {
            continue;
        }
        const int32_t slot = atomicAdd(k.count, 1);
        if (slot < k.capacity) {
            fw_tip &o = k.out[slot];
            o.sample = k.sample;
            o.k = (int32_t)kk;
            o.i = (int32_t)i;
            o.j = (int32_t)j;
            o.x = (double)j + cy;
            o.y = (double)i + cx;
        } else if (k.status) {
            atomicOr(k.status, FW_DEV_TIP_OVERFLOW);
        }
    }
}

template <int ST, class T>
__global__ void k_diffuse(T *un, const T *u, const T *w, const int64_t *idx,
                          int64_t n_idx, int64_t n, int64_t si, int64_t sj)
{
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n_idx;
         t += (int64_t)gridDim.x * blockDim.x) {
        int64_t p = idx[t];
        un[p] = diffuse_node<ST, T>(u, w, p, n, si, sj);
    }
}

template <class M, class T>
struct IonicK {
    T *un;
    const T *u;
    void *state[M::NS];
    T params[M::NP + M::ND];
    T dt;
    const int64_t *idx;
    int64_t n_idx;
};

template <class M, class T>
__global__ void k_ionic(IonicK<M, T> k)
{
    const Params<T, M::NP + M::ND> P = load_params<T, M::NP + M::ND>(k.params);
    const T dt = k.dt;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
         t < k.n_idx; t += (int64_t)gridDim.x * blockDim.x) {
        int64_t p = k.idx[t];
        auto st = M::template load<T>(k.state, p);
        k.un[p] = M::template update<T>(k.u[p], k.un[p], st, P, dt);
        M::template store<T>(k.state, p, st);
    }
}

bool in_window(const fw_window &w, int64_t n)
{
    return w.stride > 0 && n >= w.first && n <= w.last && n % w.stride == 0;
}

template <class T>
int launch_stim(const fw_step_args *a, const fw_stim &s, T *u,
                cudaStream_t stream)
{
    StimK<T> k;
    int dim = stencil_dim(a->stencil);
    Grid g = make_grid(a->ni, a->nj, a->nk, dim);
    int64_t shape[3] = {g.ni, g.nj, g.nk};
    k.mesh = a->mesh;
    k.mask = s.mask;
    k.u = u;
    k.count = 1;
    for (int d = 0; d < 3; ++d) {
        int64_t lo = d < dim ? s.lo[d] : 0, hi = d < dim ? s.hi[d] : 1;
        if (lo < 0) lo = 0;
        if (hi > shape[d]) hi = shape[d];
        if (hi <= lo) return FW_OK;
        k.lo[d] = lo;
        k.ext[d] = hi - lo;
        k.count *= hi - lo;
    }
    k.stride[0] = g.si;
    k.stride[1] = dim == 2 ? 1 : g.sj;
    k.stride[2] = 1;
    k.value = s.value;
    k.u_max = s.u_max;
    k.kind = s.kind;
    k.has_umax = s.has_umax;
    k_stim<T><<<grid_for(k.count, kThreads), kThreads, 0, stream>>>(k);
    FW_CHECK_LAUNCH("k_stim");
    return FW_OK;
}

template <class M, int ST, class T>
int run_plain(const fw_step_args *a, int64_t n_begin, int64_t n_steps,
              cudaStream_t stream)
{
    int dim = stencil_dim(ST);
    Grid g = make_grid(a->ni, a->nj, a->nk, dim);
    StepK<M, T> k;
    k.myo = a->myo;
    k.w = (const T *)a->weights;
    k.wrow = (const T *)a->weight_rows;
    k.widx = a->weight_row_index;
    if (k.wrow && (ST != FW_STENCIL_ANISO19_XY || !k.widx ||
                   ((uintptr_t)k.wrow & 15) != 0)) {
        set_error("fw_step: weight_rows needs FW_STENCIL_ANISO19_XY, a row "
                  "index and 16-byte aligned rows");
        return FW_ERR_ARG;
    }
    for (int i = 0; i < M::NS; ++i) k.state[i] = a->state[i];
    fill_params<M, T>(k.params, a->params, a->dt);
    k.dt = (T)a->dt;
    k.n = g.n;
    k.si = g.si;
    k.sj = g.sj;
    k.status = a->status;

    ProbeK<T> pk;
    pk.status = a->status;
    for (int i = 0; i < FW_MAX_STATE; ++i) pk.state[i] = a->state[i];
    pk.f64_mask = pk.pair_mask = 0;
    for (int i = 0; i < M::NS; ++i) {
        if (fw_state_is_f64(a->model, a->precision, i)) pk.f64_mask |= 1u << i;
        if (fw_state_is_pair(a->model, a->precision, i)) pk.pair_mask |= 1u << i;
    }

    const bool listed = UseList<M, T>::value && a->node_list &&
                        g.n >= kListMinNodes;
    const int threads = sizeof(T) == 4 && listed ? kListThreadsF32 : step_threads<T>();
    k.list = listed ? a->node_list : nullptr;
    k.n_myo = (int32_t)a->n_list_myo;
    // (without a myocyte in the list, none)
    const int64_t stepped = listed ? a->n_list_myo : g.n;
    const int blocks = stepped ? grid_for(stepped, threads, step_blocks<T>(listed)) : 0;
    const int blocks_rest = grid_for(g.n - a->n_list_myo, threads * kRestNodes,
                                     kRestThreads / threads);
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(threads);
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    // activation trackers (bits) that have looked at the non-myocytes of each
    // potential buffer since a stimulus last wrote it; nothing else does
    uint32_t seen[2] = {0, 0}, active;
    static_assert(FW_MAX_AT <= 32, "one bit a tracker");
    for (int64_t s = 0; s < n_steps; ++s) {
        const int64_t n = n_begin + s;
        T *cur = (T *)a->u[s & 1];
        T *nxt = (T *)a->u[(s + 1) & 1];
        for (int i = 0; i < a->n_stims; ++i) {
            const fw_stim &st = a->stims[i];
            if (n >= st.first && n <= st.last) {
                int rc = launch_stim<T>(a, st, cur, stream);
                if (rc) return rc;
                seen[s & 1] = 0;
            }
        }
        k.u = cur;
        k.un = nxt;
        k.step = n;
        k.n_at = 0;
        active = 0;
        for (int i = 0; i < a->n_at; ++i)
            if (in_window(a->at[i].win, n)) {
                active |= 1u << i;
                k.at[k.n_at++] = AtK<T>{(T)a->at[i].threshold,
                                        a->at[i].act_step};
            }
        k.n_lat = 0;
        for (int i = 0; i < a->n_lat; ++i)
            if (in_window(a->lat[i].win, n)) {
                const fw_lat_tracker &L = a->lat[i];
                k.lat[k.n_lat++] = LatK<T>{(T)L.threshold, L.activated,
                                        L.cross_steps, L.cross_count,
                                        L.capacity};
            }
        // probes of the potential alone ride on the step; those of the state,
        // which the step advances, follow it
        pk.n = 0;
        k.n_up = 0;
        for (int i = 0; i < a->n_probe; ++i) {
            const fw_probe_tracker &P = a->probe[i];
            if (!in_window(P.win, n)) continue;
            const int64_t sample = P.sample_offset + (n - P.win.first) / P.win.stride;
            if (P.n_vars == 1 && P.var_ids[0] == 0 && sample < P.capacity) {
                k.up[k.n_up++] = UProbe{P.cells, P.out + sample * P.n_cells, P.n_cells};
                continue;
            }
            ProbeOne &o = pk.pr[pk.n++];
            o.cells = P.cells;
            o.out = P.out;
            o.sample = sample;
            o.capacity = P.capacity;
            o.n_cells = P.n_cells;
            o.n_vars = P.n_vars;
            for (int v = 0; v < FW_MAX_PROBE_VARS; ++v) o.var_ids[v] = P.var_ids[v];
        }
        // the trackers also watch the nodes that do not step: the local
        // activation ones each time (a node may differ between the buffers
        // and cross back), the others, which record the first time only, once
        // for each buffer and stimulus.
        k.rest_at = (active & ~seen[s & 1]) != 0;
        k.rest = listed && (k.n_lat || k.rest_at) ? blocks_rest : 0;
        if (k.rest_at) seen[s & 1] |= active;
        const int ctas = blocks + k.rest + (k.n_up ? 1 : 0);
        attr.val.programmaticStreamSerializationAllowed = s > 0;
        cfg.gridDim = dim3((unsigned)ctas);
        auto kern = k_step<M, ST, T, false>;
        if constexpr (UseList<M, T>::value) {
            if (listed) kern = k_step<M, ST, T, true>;
        }
        if (ctas) {
            FW_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kern, k));
            FW_CHECK_LAUNCH("k_step");
        }
        if (pk.n) {
            pk.u = cur;
            k_probe<T><<<1, 128, 0, stream>>>(pk);
            FW_CHECK_LAUNCH("k_probe");
        }
        for (int i = 0; i < a->n_ecg; ++i) {
            const fw_ecg_tracker &E = a->ecg[i];
            if (!in_window(E.win, n)) continue;
            const int64_t smp = E.sample_offset + (n - E.win.first) / E.win.stride;
            if (smp < 0 || smp >= E.capacity) {
                set_error("fw_step: ECG sample %lld outside its capacity %lld",
                          (long long)smp, (long long)E.capacity);
                return FW_ERR_ARG;
            }
            int rc = launch_ecg<ST, T>(cur, k.w, a->myo, g, dim, E.coords,
                                       E.n_leads, E.dr,
                                       E.out + smp * E.n_leads, stream);
            if (rc) return rc;
        }
        for (int i = 0; i < a->n_tip; ++i) {
            const fw_tip_tracker &P = a->tip[i];
            if (!in_window(P.win, n)) continue;
            TipK<T> tk;
            tk.u_prev = (const T *)P.u_prev;
            tk.u = cur;
            tk.ni = g.ni;
            tk.nj = g.nj;
            tk.nk = g.nk;
            tk.thr = P.threshold;
            tk.out = P.out;
            tk.count = P.count;
            tk.capacity = P.capacity;
            tk.sample = (int32_t)(P.sample_offset + (n - P.win.first) / P.win.stride);
            tk.status = a->status;
            const int64_t cells = (g.ni > 10 && g.nj > 10)
                                      ? (g.ni - 10) * (g.nj - 10) * g.nk : 0;
            if (cells > 0) {
                k_tips<T><<<grid_for(cells, kThreads, 152 * 8), kThreads, 0,
                            stream>>>(tk);
                FW_CHECK_LAUNCH("k_tips");
            }
            FW_CUDA_CHECK(cudaMemcpyAsync(P.u_prev, cur, g.n * sizeof(T),
                                          cudaMemcpyDeviceToDevice, stream));
        }
    }
    return FW_OK;
}

template <class M, class T>
int run_ionic(void *u_new, const void *u, void *const *state,
              const int64_t *idx, int64_t n_idx, double dt,
              const double *params, cudaStream_t stream)
{
    IonicK<M, T> k;
    k.un = (T *)u_new;
    k.u = (const T *)u;
    for (int i = 0; i < M::NS; ++i) k.state[i] = state[i];
    fill_params<M, T>(k.params, params, dt);
    k.dt = (T)dt;
    k.idx = idx;
    k.n_idx = n_idx;
    if (n_idx > 0) k_ionic<M, T><<<grid_for(n_idx, kThreads), kThreads, 0, stream>>>(k);
    FW_CHECK_LAUNCH("k_ionic");
    return FW_OK;
}

struct PlainDispatch {
    const fw_step_args *a;
    int64_t n_begin, n_steps;
    cudaStream_t stream;
    template <class M, int ST, class T>
    int run() const { return run_plain<M, ST, T>(a, n_begin, n_steps, stream); }
};

struct IonicDispatch {
    void *u_new;
    const void *u;
    void *const *state;
    const int64_t *idx;
    int64_t n_idx;
    double dt;
    const double *params;
    cudaStream_t stream;
    template <class M, class T>
    int run() const
    {
        return run_ionic<M, T>(u_new, u, state, idx, n_idx, dt, params, stream);
    }
};

}  // namespace
}  // namespace fw
