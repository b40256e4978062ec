// bfb_aux.cu -- agents (secretion/uptake), checksum and precision conversion.
#include "bfb_aux.cuh"

#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>

#include <algorithm>
#include <type_traits>

#include "bfb_upload.h"

namespace bfb {

// ---------------------------------------------------------------------------
// Conversions
// ---------------------------------------------------------------------------
__global__ void d2f_kernel(const double *__restrict__ s, float *__restrict__ d, long long n) {
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
        d[e] = __double2float_rn(s[e]);
}
__global__ void f2d_kernel(const float *__restrict__ s, double *__restrict__ d, long long n) {
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
        d[e] = (double)s[e];
}
static unsigned grid_for(long long n) { return (unsigned)std::min<long long>((n + 255) / 256, 148LL * 32); }

template <typename TS, typename TD>
__global__ void convert_rows_kernel(const TS *__restrict__ s, TD *__restrict__ d, long long rows, int L, int sp,
                                    int dp) {
    const long long n = rows * L;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const long long r = e / L, q = e - r * L;
        if constexpr (sizeof(TD) == 4)
            d[r * dp + q] = __double2float_rn(s[r * sp + q]);
        else
            d[r * dp + q] = (double)s[r * sp + q];
    }
}

int launch_convert_d2f_rows(const double *src, float *dst, long long rows, int L, int sp, int dp, cudaStream_t s) {
    if (sp == L && dp == L) return launch_convert_d2f(src, dst, rows * L, s);
    if (rows * L <= 0) return BFB_OK;
    convert_rows_kernel<double, float><<<grid_for(rows * L), 256, 0, s>>>(src, dst, rows, L, sp, dp);
    BFB_CUDA(cudaGetLastError());
    return BFB_OK;
}
int launch_convert_f2d_rows(const float *src, double *dst, long long rows, int L, int sp, int dp, cudaStream_t s) {
    if (sp == L && dp == L) return launch_convert_f2d(src, dst, rows * L, s);
    if (rows * L <= 0) return BFB_OK;
    convert_rows_kernel<float, double><<<grid_for(rows * L), 256, 0, s>>>(src, dst, rows, L, sp, dp);
    BFB_CUDA(cudaGetLastError());
    return BFB_OK;
}

int launch_convert_d2f(const double *src, float *dst, long long n, cudaStream_t s) {
    if (n <= 0) return BFB_OK;
    d2f_kernel<<<grid_for(n), 256, 0, s>>>(src, dst, n);
    BFB_CUDA(cudaGetLastError());
    return BFB_OK;
}
int launch_convert_f2d(const float *src, double *dst, long long n, cudaStream_t s) {
    if (n <= 0) return BFB_OK;
    f2d_kernel<<<grid_for(n), 256, 0, s>>>(src, dst, n);
    BFB_CUDA(cudaGetLastError());
    return BFB_OK;
}

// ---------------------------------------------------------------------------
// Agent binning and constants.
//
// Binning restates Basic_Agent::assign_position -> update_voxel_index ->
// Cartesian_Mesh::nearest_voxel_local_index at one rank
// (BioFVM_basic_agent.cpp:112-153, BioFVM_parallel.cpp:418-522,
//  BioFVM_mesh.cpp:204-213):
//   invalid position (outside the closed box)  -> position rejected, the
//                                                agent keeps voxel 0
//   v = (int)floor((p - lo)/h) clamped to [0, (int)((hi - lo)/h) - 1]
//   index = x*lny*lnz + y*lnz + z with lny/lnz the truncated extents,
//   clamped to [0, V-1].
// Constants restate set_internal_uptake_constants (BioFVM_basic_agent.cpp:
// 155-176) with the reference build's fused axpy:
//   c = (dt*volume)/dV, t1 = (S*rho*)*c, t2 = fma(c, U, fma(c, S, 1)).
// ---------------------------------------------------------------------------
struct BinGeom {
    double lo[3], hi[3], h[3];
    int V;
    double dV;
};

__device__ __forceinline__ int bin_axis(double p, double lo, double hi, double h) {
    int v = (int)floor(__ddiv_rn(__dsub_rn(p, lo), h));
    const int g = (int)__ddiv_rn(__dsub_rn(hi, lo), h);
    if (v >= g) v = g - 1;
    if (v < 0) v = 0;
    return v;
}

// The voxel of each agent, and the (key, list index) pairs to sort: the voxel,
// or V for an inactive agent, so that those sort past every segment.
__global__ void bin_agents_kernel(int n, const double *__restrict__ pos, const uint8_t *__restrict__ active, BinGeom g,
                                  int *__restrict__ voxel, int *__restrict__ key, int *__restrict__ idx) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= n) return;
    const double x = pos[3 * (size_t)a], y = pos[3 * (size_t)a + 1], z = pos[3 * (size_t)a + 2];
    int v = 0;  // a freshly created agent's current_voxel_index
    const bool valid = !(x < g.lo[0] || x > g.hi[0] || y < g.lo[1] || y > g.hi[1] || z < g.lo[2] || z > g.hi[2]);
    if (valid) {
        const int xi = bin_axis(x, g.lo[0], g.hi[0], g.h[0]);
        const int yi = bin_axis(y, g.lo[1], g.hi[1], g.h[1]);
        const int zi = bin_axis(z, g.lo[2], g.hi[2], g.h[2]);
        const int lny = (int)__ddiv_rn(__dsub_rn(g.hi[1], g.lo[1]), g.h[1]);
        const int lnz = (int)__ddiv_rn(__dsub_rn(g.hi[2], g.lo[2]), g.h[2]);
        v = xi * lny * lnz + yi * lnz + zi;
        if (v < 0) v = 0;
        if (v >= g.V) v = g.V - 1;
    }
    voxel[a] = v;
    key[a] = !active || active[a] ? v : g.V;
    idx[a] = a;
}

__global__ void key_agents_kernel(int n, const int *__restrict__ voxel, const uint8_t *__restrict__ active, int V,
                                  int *__restrict__ key, int *__restrict__ idx) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= n) return;
    key[a] = !active || active[a] ? voxel[a] : V;
    idx[a] = a;
}

// Of the sorted keys: head[r] = 1 where a voxel's segment starts, and
// counts[1] = the number of active agents (keys below V; zeroed before).
__global__ void segment_heads_kernel(int n, const int *__restrict__ key, int V, uint8_t *__restrict__ head,
                                     int *__restrict__ counts) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const int k = key[r];
    head[r] = k < V && (r == 0 || key[r - 1] != k);
    if (k < V && (r == n - 1 || key[r + 1] >= V)) counts[1] = r + 1;
}

// seg_voxel of each segment and the end of the last one; counts = {segments, active agents}.
__global__ void segment_ends_kernel(const int *__restrict__ key, const int *__restrict__ counts,
                                    int *__restrict__ seg_start, int *__restrict__ seg_voxel) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x, n_occ = counts[0];
    if (s < n_occ) seg_voxel[s] = key[seg_start[s]];
    if (s == n_occ) seg_start[s] = counts[1];
}

// The constants of the sorted agents, from the rates ...
template <typename T>
__global__ void agent_constants_kernel(const int *__restrict__ counts, int S, const int *__restrict__ order,
                                       const double *__restrict__ vol, const double *__restrict__ sec,
                                       const double *__restrict__ upt, const double *__restrict__ sat, double dt,
                                       double dV, T *__restrict__ o1, T *__restrict__ o2) {
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (long long)counts[1] * S) return;
    const int r = (int)(e / S), d = (int)(e - (long long)r * S);
    const int a = order[r];
    const size_t q = (size_t)a * S + d;
    const double c = __ddiv_rn(__dmul_rn(dt, vol[a]), dV);
    o1[e] = (T)__dmul_rn(__dmul_rn(sec[q], sat[q]), c);
    o2[e] = (T)__fma_rn(c, upt[q], __fma_rn(c, sec[q], 1.0));
}
// ... or as given.
template <typename T>
__global__ void gather_constants_kernel(const int *__restrict__ counts, int S, const int *__restrict__ order,
                                        const double *__restrict__ t1, const double *__restrict__ t2,
                                        T *__restrict__ o1, T *__restrict__ o2) {
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (long long)counts[1] * S) return;
    const int r = (int)(e / S), d = (int)(e - (long long)r * S);
    const size_t q = (size_t)order[r] * S + d;
    o1[e] = (T)t1[q];
    o2[e] = (T)t2[q];
}

// BioFVM_basic_agent.cpp:291-296 for all agents of one voxel, in list order.
template <typename T>
__global__ void cells_kernel(T *f, int S, int nz, int Lp, int n_occ, const int *__restrict__ seg_start,
                             const int *__restrict__ seg_voxel, const T *__restrict__ t1, const T *__restrict__ t2) {
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (long long)n_occ * S) return;
    const int s = (int)(e / S), d = (int)(e % S);
    const size_t fe = voxel_elem(seg_voxel[s], d, nz, S, Lp);
    const int a0 = seg_start[s], a1 = seg_start[s + 1];
    pdl_wait();  // the segments are complete (bfb_set_agents waits for them); the field is the sweep's
    T x = f[fe];
    for (int a = a0; a < a1; ++a) {
        const size_t q = (size_t)a * S + d;
        if constexpr (sizeof(T) == 8)
            x = __ddiv_rn(__dadd_rn(x, t1[q]), t2[q]);
        else
            x = __fdiv_rn(__fadd_rn(x, t1[q]), t2[q]);
    }
    pdl_launch_dependents();
    f[fe] = x;
}

void agents_free(bfb_env_s *env) {
    cudaFree(env->ag_ws);
    env->ag_ws = nullptr;
    env->ag_ws_bytes = 0;
    env->n_agents = env->n_occ = env->n_active = 0;
    env->rates_known = false;
}

namespace {

// The scratch of one agents_build call, in the env's agent block.
struct AgentScratch {
    double *pos, *t1, *t2;  // positions; constants as given (in the rates' place)
    uint8_t *active, *head;
    int *key, *key_sorted, *idx, *counts;
    void *tmp;
    size_t sort_bytes, select_bytes;
};

// Lays the env's agent arrays and the scratch for n agents out in its agent
// block, which is kept between calls and grows when it must. A program sets its
// agents once per mechanics step; allocating and freeing seventeen arrays on
// each call (every cudaFree waits for the device) took most of a call's time:
// 40,000 agents x 4 substrates 4.3 -> 0.41 ms a call, 100,000 x 8 12 -> 1.3,
// now bound by the rates crossing the host link from pageable memory. An empty
// set gives the block back, and so does one that needs under a quarter of a
// block of more than kAgentBlockKeep bytes (a smaller one is not worth the
// wait for the device that freeing it takes).
constexpr size_t kAgentBlockKeep = 16 << 20;
int agents_layout(bfb_env_s *env, int n, bool rates, AgentScratch *w) {
    const size_t N = (size_t)n, nS = N * env->S;
    int end_bit = 1;
    while (end_bit < 31 && (1LL << end_bit) <= env->V) ++end_bit;
    env->ag_end_bit = end_bit;  // keys 0 .. V
    w->sort_bytes = w->select_bytes = 0;
    BFB_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, w->sort_bytes, (const int *)nullptr, (int *)nullptr,
                                             (const int *)nullptr, (int *)nullptr, n, 0, end_bit, env->stream));
    BFB_CUDA(cub::DeviceSelect::Flagged(nullptr, w->select_bytes, thrust::counting_iterator<int>(0),
                                        (const uint8_t *)nullptr, (int *)nullptr, (int *)nullptr, n, env->stream));
    char *base = nullptr;
    size_t off = 0;
    auto take = [&](auto **p, size_t bytes) {
        *p = reinterpret_cast<std::remove_reference_t<decltype(*p)>>(base ? base + off : nullptr);
        off += (std::max<size_t>(bytes, 1) + 255) / 256 * 256;
    };
    auto lay = [&]() {
        off = 0;
        take(&env->agent_voxel, sizeof(int) * N);
        take(&env->seg_start, sizeof(int) * (N + 1));
        take(&env->seg_voxel, sizeof(int) * N);
        take(&env->ag_order, sizeof(int) * N);
        take((char **)&env->ag_t1, env->elem * nS);
        take((char **)&env->ag_t2, env->elem * nS);
        if (rates) {
            take(&env->ag_vol, sizeof(double) * N);
            take(&env->ag_sec, sizeof(double) * nS);
            take(&env->ag_upt, sizeof(double) * nS);
            take(&env->ag_sat, sizeof(double) * nS);
            take(&w->pos, sizeof(double) * 3 * N);
        } else {
            take(&w->t1, sizeof(double) * nS);
            take(&w->t2, sizeof(double) * nS);
        }
        take(&w->active, N);
        take(&w->head, N);
        take(&w->key, sizeof(int) * N);
        take(&w->key_sorted, sizeof(int) * N);
        take(&w->idx, sizeof(int) * N);
        take(&w->counts, sizeof(int) * 2);
        take((char **)&w->tmp, std::max(w->sort_bytes, w->select_bytes));
    };
    lay();
    if (off > env->ag_ws_bytes || (env->ag_ws_bytes > kAgentBlockKeep && off < env->ag_ws_bytes / 4)) {
        const size_t want = off + off / 4;  // agents divide
        agents_free(env);
        BFB_CUDA(cudaMalloc(&env->ag_ws, want));
        env->ag_ws_bytes = want;
    }
    base = static_cast<char *>(env->ag_ws);
    lay();
    return BFB_OK;
}

// Sorts the active agents by voxel (stable: list order within a voxel) and
// builds the per-voxel segments the cells kernel walks, from w.key / w.idx.
int agents_sort(bfb_env_s *env, int n, AgentScratch &w) {
    cudaStream_t s = env->stream;
    BFB_CUDA(cudaMemsetAsync(w.counts, 0, 2 * sizeof(int), s));
    BFB_CUDA(cub::DeviceRadixSort::SortPairs(w.tmp, w.sort_bytes, w.key, w.key_sorted, w.idx, env->ag_order, n, 0,
                                             env->ag_end_bit, s));
    segment_heads_kernel<<<(n + 255) / 256, 256, 0, s>>>(n, w.key_sorted, (int)env->V, w.head, w.counts);
    BFB_CUDA(cudaGetLastError());
    BFB_CUDA(cub::DeviceSelect::Flagged(w.tmp, w.select_bytes, thrust::counting_iterator<int>(0), w.head,
                                        env->seg_start, w.counts, n, s));
    segment_ends_kernel<<<(n + 256) / 256, 256, 0, s>>>(w.key_sorted, w.counts, env->seg_start, env->seg_voxel);
    BFB_CUDA(cudaGetLastError());
    return BFB_OK;
}

// Waits for the build and takes the counts the launches are sized by.
int agents_finish(bfb_env_s *env, Uploads &up, const AgentScratch &w) {
    int counts[2] = {0, 0};
    BFB_CUDA(cudaMemcpyAsync(counts, w.counts, sizeof(counts), cudaMemcpyDeviceToHost, env->stream));
    BFB_CUDA(up.wait());
    env->n_occ = counts[0];
    env->n_active = counts[1];
    return BFB_OK;
}

// Drops the agent set once no kernel reads it any more.
int agents_drop(bfb_env_s *env) {
    if (int st = env_quiesce(env)) return st;
    env->n_agents = env->n_occ = env->n_active = 0;
    env->rates_known = false;
    return BFB_OK;
}

}  // namespace

int agents_build(bfb_env_s *env, int n, const double *pos, const double *volume, const double *sec,
                 const double *upt, const double *sat, const uint8_t *active, double dt) {
    int st = agents_drop(env);
    if (!st && n == 0) agents_free(env);
    if (st || n == 0) return st;
    const int S = env->S;
    const size_t nS = (size_t)n * S;
    cudaStream_t s = env->stream;
    AgentScratch w;
    if ((st = agents_layout(env, n, true, &w))) return st;
    Uploads up(s);  // the caller's arrays: no return before their copies are done
    BFB_CUDA(up.copy(w.pos, pos, sizeof(double) * 3 * n));
    if (active) BFB_CUDA(up.copy(w.active, active, n));
    BinGeom g;
    for (int a = 0; a < 3; ++a) {
        g.lo[a] = env->bbox[a];
        g.hi[a] = env->bbox[3 + a];
        g.h[a] = env->dx;
    }
    g.V = (int)env->V;
    g.dV = (env->dx * env->dx) * env->dx;
    bin_agents_kernel<<<(n + 127) / 128, 128, 0, s>>>(n, w.pos, active ? w.active : nullptr, g, env->agent_voxel, w.key,
                                                      w.idx);
    BFB_CUDA(cudaGetLastError());
    env->n_agents = n;
    if ((st = agents_sort(env, n, w))) return st;
    // the rates cross the host link while the sort runs
    BFB_CUDA(up.copy(env->ag_vol, volume, sizeof(double) * n));
    BFB_CUDA(up.copy(env->ag_sec, sec, sizeof(double) * nS));
    BFB_CUDA(up.copy(env->ag_upt, upt, sizeof(double) * nS));
    BFB_CUDA(up.copy(env->ag_sat, sat, sizeof(double) * nS));
    const unsigned gb = (unsigned)((nS + 255) / 256);
    if (env->precision == BFB_FP64)
        agent_constants_kernel<double><<<gb, 256, 0, s>>>(w.counts, S, env->ag_order, env->ag_vol, env->ag_sec,
                                                          env->ag_upt, env->ag_sat, dt, g.dV, (double *)env->ag_t1,
                                                          (double *)env->ag_t2);
    else
        agent_constants_kernel<float><<<gb, 256, 0, s>>>(w.counts, S, env->ag_order, env->ag_vol, env->ag_sec,
                                                         env->ag_upt, env->ag_sat, dt, g.dV, (float *)env->ag_t1,
                                                         (float *)env->ag_t2);
    BFB_CUDA(cudaGetLastError());
    if ((st = agents_finish(env, up, w))) return st;
    env->rates_known = true;
    return BFB_OK;
}

int agents_build_constants(bfb_env_s *env, int n, const int *voxel, const double *t1, const double *t2,
                           const uint8_t *active) {
    int st = agents_drop(env);
    if (!st && n == 0) agents_free(env);
    if (st || n == 0) return st;
    const int S = env->S;
    const size_t nS = (size_t)n * S;
    cudaStream_t s = env->stream;
    AgentScratch w;
    if ((st = agents_layout(env, n, false, &w))) return st;
    Uploads up(s);
    BFB_CUDA(up.copy(env->agent_voxel, voxel, sizeof(int) * n));
    env->n_agents = n;
    for (int a = 0; a < n; ++a)
        if ((!active || active[a]) && (voxel[a] < 0 || voxel[a] >= env->V))
            return fail(BFB_ERR_INVALID_ARG, "agent voxel index out of range");
    if (active) BFB_CUDA(up.copy(w.active, active, n));
    key_agents_kernel<<<(n + 127) / 128, 128, 0, s>>>(n, env->agent_voxel, active ? w.active : nullptr, (int)env->V,
                                                      w.key, w.idx);
    BFB_CUDA(cudaGetLastError());
    if ((st = agents_sort(env, n, w))) return st;
    BFB_CUDA(up.copy(w.t1, t1, sizeof(double) * nS));
    BFB_CUDA(up.copy(w.t2, t2, sizeof(double) * nS));
    const unsigned gb = (unsigned)((nS + 255) / 256);
    if (env->precision == BFB_FP64)
        gather_constants_kernel<double><<<gb, 256, 0, s>>>(w.counts, S, env->ag_order, w.t1, w.t2,
                                                           (double *)env->ag_t1, (double *)env->ag_t2);
    else
        gather_constants_kernel<float><<<gb, 256, 0, s>>>(w.counts, S, env->ag_order, w.t1, w.t2, (float *)env->ag_t1,
                                                          (float *)env->ag_t2);
    BFB_CUDA(cudaGetLastError());
    return agents_finish(env, up, w);
}

int launch_cells(bfb_env_s *env, cudaStream_t s) {
    if (env->n_occ == 0) return BFB_OK;
    const long long tot = (long long)env->n_occ * env->S;
    const unsigned gb = (unsigned)((tot + 255) / 256);
    if (env->precision == BFB_FP64)
        BFB_CUDA(launch_pdl(cells_kernel<double>, gb, 256, 0, s, (double *)env->field, env->S, env->nz, env->Lp,
                            env->n_occ, env->seg_start, env->seg_voxel, (const double *)env->ag_t1,
                            (const double *)env->ag_t2));
    else
        BFB_CUDA(launch_pdl(cells_kernel<float>, gb, 256, 0, s, (float *)env->field, env->S, env->nz, env->Lp,
                            env->n_occ, env->seg_start, env->seg_voxel, (const float *)env->ag_t1,
                            (const float *)env->ag_t2));
    return BFB_OK;
}

// ---------------------------------------------------------------------------
// Checksum: fixed partition of voxels per block, one pass over the field,
// FP64 sums in a fixed order -> deterministic.
// A block sums voxels [v0, v1) (v0 a multiple of 4, so the block's first
// element is 16-byte aligned when the field is). The block's elements are cut
// into rows of W = R*S elements (W a multiple of the 16-byte vector width V);
// thread t reads vector t of every row, so one warp load covers 512
// consecutive bytes, every element is read once, and the element at position
// p = V*t + j of a row always belongs to substrate p mod S: the thread keeps
// one FP64 accumulator per vector lane j. The block then adds, per substrate
// d, the accumulators of positions d, d + S, ..., in order, and
// checksum_final_kernel adds the blocks' partial sums in block order.
// ---------------------------------------------------------------------------
constexpr int kSumBlocks = 296;  // 2 x 148 SMs
constexpr int kSumThreads = 256;
constexpr int kMaxSumS = 64;

template <typename T>
struct SumVec;
template <>
struct SumVec<float> {
    static constexpr int V = 4;
    using type = float4;
    __device__ static void add(const float4 &x, double (&a)[4]) {
        a[0] += (double)x.x, a[1] += (double)x.y, a[2] += (double)x.z, a[3] += (double)x.w;
    }
};
template <>
struct SumVec<double> {
    static constexpr int V = 2;
    using type = double2;
    __device__ static void add(const double2 &x, double (&a)[2]) { a[0] += x.x, a[1] += x.y; }
};

// W = R*S elements per row: the largest multiple of lcm(S, V) not above V*256
__host__ __device__ inline int sum_row_width(int S, int V) {
    int l = S;
    while (l % V) l += S;
    return (V * kSumThreads) / l * l;
}

template <typename T>
__global__ void __launch_bounds__(kSumThreads) checksum_partial_kernel(const T *__restrict__ f, long long V, int S,
                                                                       double *__restrict__ partials) {
    constexpr int VW = SumVec<T>::V;
    using VT = typename SumVec<T>::type;
    __shared__ double red[VW * kSumThreads];
    const int W = sum_row_width(S, VW);
    const int t = threadIdx.x;
    long long per = (V + gridDim.x - 1) / gridDim.x;
    per = (per + 3) / 4 * 4;
    const long long v0 = min(V, (long long)blockIdx.x * per), v1 = min(V, v0 + per);
    const long long e0 = v0 * S, ne = (v1 - v0) * S;  // the block's elements
    const T *__restrict__ base = f + e0;
    double acc[VW];
#pragma unroll
    for (int j = 0; j < VW; ++j) acc[j] = 0.0;
    const bool vec = (reinterpret_cast<uintptr_t>(base) & 15) == 0;
    const long long rows = ne / W;
    long long row = 0;
    if (vec && VW * t < W) {
        const VT *__restrict__ p = reinterpret_cast<const VT *>(base) + t;
        const long long stride = W / VW;  // vectors per row
        constexpr int kRowsInFlight = 8;  // 8 x 16 B per thread in flight
        for (; row + kRowsInFlight <= rows; row += kRowsInFlight) {
            VT x[kRowsInFlight];
#pragma unroll
            for (int u = 0; u < kRowsInFlight; ++u) x[u] = p[(row + u) * stride];
#pragma unroll
            for (int u = 0; u < kRowsInFlight; ++u) SumVec<T>::add(x[u], acc);
        }
        for (; row < rows; ++row) SumVec<T>::add(p[row * stride], acc);
    }
    if (!vec) row = 0;  // an unaligned field is read element by element
    // the rest (the last partial row, or all rows without 16-byte alignment)
    // element by element, each element to the accumulator of its row position
    if (VW * t < W)
        for (long long e = row * W + VW * t; e < ne; e += W)
#pragma unroll
            for (int j = 0; j < VW; ++j)
                if (e + j < ne) acc[j] += (double)base[e + j];
#pragma unroll
    for (int j = 0; j < VW; ++j) red[VW * t + j] = VW * t < W ? acc[j] : 0.0;
    __syncthreads();
    if (t < S) {
        double sum = 0.0;
        for (int q = t; q < W; q += S) sum += red[q];
        partials[(size_t)blockIdx.x * S + t] = sum;
    }
}

// The same sums over a field with padded rows (rows of L = nz*S elements, Lp
// apart): block b sums rows [r0, r1); thread t < W = R*S takes positions
// t, t + W, ... of every row, all of substrate t mod S; then, as above,
// thread d < S adds its substrate's W / S accumulators in order.
template <typename T>
__global__ void __launch_bounds__(kSumThreads) checksum_rows_kernel(const T *__restrict__ f, long long rows, int L,
                                                                    int Lp, int S, double *__restrict__ partials) {
    __shared__ double red[kSumThreads];
    const int W = kSumThreads / S * S;
    const int t = threadIdx.x;
    const long long per = (rows + gridDim.x - 1) / gridDim.x;
    const long long r0 = min(rows, (long long)blockIdx.x * per), r1 = min(rows, r0 + per);
    double acc = 0.0;
    if (t < W)
        for (long long r = r0; r < r1; ++r) {
            const T *__restrict__ row = f + (size_t)r * Lp;
            for (int q = t; q < L; q += W) acc += (double)row[q];
        }
    red[t] = t < W ? acc : 0.0;
    __syncthreads();
    if (t < S) {
        double sum = 0.0;
        for (int q = t; q < W; q += S) sum += red[q];
        partials[(size_t)blockIdx.x * S + t] = sum;
    }
}

__global__ void checksum_final_kernel(const double *__restrict__ partials, int nblocks, int S, double *__restrict__ out) {
    const int d = threadIdx.x;
    if (d >= S) return;
    double acc = 0.0;
    for (int b = 0; b < nblocks; ++b) acc += partials[(size_t)b * S + d];
    out[d] = acc;
}

int checksum_prepare(bfb_env_s *env) {
    if (env->partials) return BFB_OK;
    BFB_CUDA(cudaMalloc(&env->partials, sizeof(double) * (kSumBlocks * (size_t)env->S + env->S)));
    env->partial_blocks = kSumBlocks;
    return BFB_OK;
}

int launch_checksum(bfb_env_s *env, double *out_dev, cudaStream_t s) {
    if (env->S > kMaxSumS) return fail(BFB_ERR_UNSUPPORTED, "checksum supports at most 64 substrates");
    if (env->Lp != env->nz * env->S) {  // padded rows
        const long long rows = (long long)env->nx * env->ny;
        if (env->precision == BFB_FP64)
            checksum_rows_kernel<double><<<kSumBlocks, kSumThreads, 0, s>>>(
                (const double *)env->field, rows, env->nz * env->S, env->Lp, env->S, env->partials);
        else
            checksum_rows_kernel<float><<<kSumBlocks, kSumThreads, 0, s>>>(
                (const float *)env->field, rows, env->nz * env->S, env->Lp, env->S, env->partials);
        checksum_final_kernel<<<1, kMaxSumS, 0, s>>>(env->partials, kSumBlocks, env->S, out_dev);
        BFB_CUDA(cudaGetLastError());
        return BFB_OK;
    }
    if (env->precision == BFB_FP64)
        checksum_partial_kernel<double><<<kSumBlocks, kSumThreads, 0, s>>>((const double *)env->field, env->V, env->S,
                                                                         env->partials);
    else
        checksum_partial_kernel<float><<<kSumBlocks, kSumThreads, 0, s>>>((const float *)env->field, env->V, env->S,
                                                                        env->partials);
    checksum_final_kernel<<<1, kMaxSumS, 0, s>>>(env->partials, kSumBlocks, env->S, out_dev);
    BFB_CUDA(cudaGetLastError());
    return BFB_OK;
}

// ---------------------------------------------------------------------------
// Field comparison: max|a-b|, max|b|, sum (a-b)^2, sum b^2 (FP64 partials per
// block, summed in block order on the host).
// ---------------------------------------------------------------------------
template <typename TA, typename TB>
__global__ void compare_kernel(const TA *__restrict__ a, int la, const TB *__restrict__ b, int lb, long long rows, int L,
                               double *__restrict__ part) {
    __shared__ double s0[256], s1[256], s2[256], s3[256];
    double mx = 0, mb = 0, sd = 0, sb = 0;
    const long long N = rows * L;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < N; e += (long long)gridDim.x * blockDim.x) {
        const long long r = (la == L && lb == L) ? 0 : e / L, q = e - r * L;
        const double x = (double)a[r * la + q], y = (double)b[r * lb + q], df = x - y;
        mx = fmax(mx, fabs(df));
        mb = fmax(mb, fabs(y));
        sd += df * df;
        sb += y * y;
    }
    s0[threadIdx.x] = mx;
    s1[threadIdx.x] = mb;
    s2[threadIdx.x] = sd;
    s3[threadIdx.x] = sb;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            s0[threadIdx.x] = fmax(s0[threadIdx.x], s0[threadIdx.x + w]);
            s1[threadIdx.x] = fmax(s1[threadIdx.x], s1[threadIdx.x + w]);
            s2[threadIdx.x] += s2[threadIdx.x + w];
            s3[threadIdx.x] += s3[threadIdx.x + w];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        part[4 * blockIdx.x + 0] = s0[0];
        part[4 * blockIdx.x + 1] = s1[0];
        part[4 * blockIdx.x + 2] = s2[0];
        part[4 * blockIdx.x + 3] = s3[0];
    }
}

int compare_fields(const void *a, int pa, int la, const void *b, int pb, int lb, long long rows, int L, double *out4,
                   cudaStream_t s) {
    const int blocks = 592;
    double *part = nullptr;
    BFB_CUDA(cudaMalloc(&part, sizeof(double) * 4 * blocks));
    if (pa == BFB_FP64 && pb == BFB_FP64)
        compare_kernel<<<blocks, 256, 0, s>>>((const double *)a, la, (const double *)b, lb, rows, L, part);
    else if (pa == BFB_FP32 && pb == BFB_FP64)
        compare_kernel<<<blocks, 256, 0, s>>>((const float *)a, la, (const double *)b, lb, rows, L, part);
    else if (pa == BFB_FP64 && pb == BFB_FP32)
        compare_kernel<<<blocks, 256, 0, s>>>((const double *)a, la, (const float *)b, lb, rows, L, part);
    else
        compare_kernel<<<blocks, 256, 0, s>>>((const float *)a, la, (const float *)b, lb, rows, L, part);
    std::vector<double> h(4 * blocks);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(h.data(), part, sizeof(double) * 4 * blocks, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaFree(part);
    if (e != cudaSuccess) return cuda_fail(e, "compare_fields");
    out4[0] = out4[1] = out4[2] = out4[3] = 0;
    for (int q = 0; q < blocks; ++q) {
        out4[0] = std::max(out4[0], h[4 * q]);
        out4[1] = std::max(out4[1], h[4 * q + 1]);
        out4[2] += h[4 * q + 2];
        out4[3] += h[4 * q + 3];
    }
    return BFB_OK;
}

// Checksum kernels on caller-provided scratch: `partials` holds at least
// nblocks*S doubles; out_dev receives S doubles. Launches only, no allocation.
int launch_checksum_raw(const void *field, int precision, long long V, int S, double *partials, int nblocks,
                        double *out_dev, cudaStream_t s) {
    if (precision == BFB_FP64)
        checksum_partial_kernel<double><<<nblocks, kSumThreads, 0, s>>>((const double *)field, V, S, partials);
    else
        checksum_partial_kernel<float><<<nblocks, kSumThreads, 0, s>>>((const float *)field, V, S, partials);
    checksum_final_kernel<<<1, kMaxSumS, 0, s>>>(partials, nblocks, S, out_dev);
    BFB_CUDA(cudaGetLastError());
    return BFB_OK;
}

}  // namespace bfb
