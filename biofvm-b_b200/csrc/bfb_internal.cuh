// bfb_internal.cuh -- shared types of the B200 diffusion-decay library.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdint>
#include <string>
#include <vector>

#include <nvtx3/nvToolsExt.h>

#include "biofvm_b200.h"

namespace bfb {

// An NVTX range over a host scope: one per entry point that launches work and
// one per phase in bfb_profile_steps, so that profilers recording NVTX (ncu's
// --nvtx filters) can select them. Without a profiler attached the calls do
// nothing.
struct NvtxRange {
    explicit NvtxRange(const char *name) { nvtxRangePushA(name); }
    ~NvtxRange() { nvtxRangePop(); }
    NvtxRange(const NvtxRange &) = delete;
    NvtxRange &operator=(const NvtxRange &) = delete;
};

// ---------------------------------------------------------------------------
// Error plumbing: every C entry point returns a status and records a message.
// ---------------------------------------------------------------------------
void set_error(const std::string &msg);
int fail(int code, const std::string &msg);
int cuda_fail(cudaError_t e, const char *what);

// Waits for the env's stream, then reads its sticky device error flag:
// BFB_ERR_WATCHDOG once a kernel's bounded wait has run out (the field is then
// not trustworthy), BFB_OK otherwise.
int env_check_device_error(::bfb_env_s *env);

// Waits until no kernel reads the env's device arrays (factors, faces, bulk
// coefficients, agents) any more, before they are overwritten in place: for the
// env's stream, and where a batch was made over the env, whose steps run on
// streams of its own, for the device.
int env_quiesce(::bfb_env_s *env);

#define BFB_CUDA(call)                                        \
    do {                                                      \
        cudaError_t _e = (call);                              \
        if (_e != cudaSuccess) return ::bfb::cuda_fail(_e, #call); \
    } while (0)

// Programmatic dependent launch: the next kernel of the stream may be set up
// (CTAs placed, barriers initialised) while this one drains; it must call
// pdl_wait before it touches what earlier kernels wrote, which returns once
// they have completed and their writes are visible. Every kernel launched
// this way waits, so completion stays transitive along the stream. What an
// earlier kernel may still be writing when such a kernel starts is not read-only
// for its lifetime: pointers to it carry no __restrict__ and are not read by
// __ldg, either of which would let the compiler move a load above the wait or
// take it from the read-only path. A kernel
// lets the next one in (pdl_launch_dependents) when its tile is solved, not
// when it starts: waiting CTAs hold the shared memory that other envs' kernels
// beside them could use (three 101x103x99 x 5 FP64 envs stepped side by side
// with bulk terms: 773 us with the early call, 723 with the late one, 716
// without; a single env gains either way, about 1.5 us a launch: 64^3 x 4 FP32
// step 22.6 -> 17.7 us, 129x127x126 x 3 45 -> 39 us).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kernel)(KArgs...), unsigned blocks, unsigned threads, size_t smem, cudaStream_t s,
                       Args &&...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// ---------------------------------------------------------------------------
// Dirichlet faces on the device.
//   faces[f] holds the values of face f for every substrate:
//     f = 0/1 (x-lo/hi): [ny][nz][S]   f = 2/3 (y-lo/hi): [nx][nz][S]
//     f = 4/5 (z-lo/hi): [nx][ny][S]
//   mask[d] bit f set <=> face f is active for substrate d.
// A voxel on several faces (edges, corners) has the same value in every face
// array, because all are cut from one per-voxel array.
// ---------------------------------------------------------------------------
// The field element of voxel v = (i*ny + j)*nz + k, substrate d, with the
// (i, j) rows Lp elements apart.
__device__ __forceinline__ size_t voxel_elem(int v, int d, int nz, int S, int Lp) {
    const int row = v / nz;
    return (size_t)row * Lp + (size_t)(v - row * nz) * S + d;
}

template <typename T>
struct DirFaces {
    const T *face[6];
    const uint8_t *mask;  // [S]
    int nx, ny, nz, S;
    int any;              // 0: no active face for any substrate
};

// Bulk source/sink terms, applied before the x sweep (bulk_kernel).
//   A = S*T (rounded once), B = U + S (rounded once); rho <- (rho + dt*A) / (B*dt + 1)
template <typename T>
struct BulkTerms {
    const T *A;
    const T *B;
    T dt;
    int on;
};

// Launch shape of the three sweeps, chosen by bfb_autotune or set by
// bfb_set_tuning. Every shape computes the same numbers; only speed differs.
struct SweepTuning {
    int tma[3] = {1, 1, 1};     // TMA tiles (when the grid allows them) or cp.async tiles
    int warps[3] = {1, 1, 1};   // warps (= tiles) per CTA; one packs shared memory tightest
    int chunks[3] = {2, 2, 2};  // row groups per TMA tile (pipeline stages); 2 measured fastest
};

}  // namespace bfb

// ---------------------------------------------------------------------------
// The environment handle.
// ---------------------------------------------------------------------------
struct bfb_env_s {
    int device = 0;
    int precision = BFB_FP64;
    int nx = 0, ny = 0, nz = 0, S = 0;
    double dx = 0;
    double bbox[6] = {0, 0, 0, 0, 0, 0};  // x0, y0, z0, x1, y1, z1
    cudaStream_t stream = nullptr;       // stream all device work is issued on
    cudaStream_t own_stream = nullptr;   // created by bfb_create, used unless bfb_set_stream overrides
    size_t elem = 8;                     // bytes per field element
    int64_t V = 0;                       // voxels
    int64_t N = 0;                       // V * S (the packed, reference layout)
    // Row pitch of the device field: the nz*S values of an (i, j) row are
    // followed by padding up to a whole number of 16-byte vectors when nz*S*elem
    // is not one (so that every sweep can use the TMA tiles); Lp = nz*S
    // otherwise. rho(i,j,k,d) lives at (i*ny + j)*Lp + k*S + d, and the field
    // holds Np = nx*ny*Lp elements.
    int Lp = 0;
    int64_t Np = 0;

    void *field = nullptr;               // device, N elements
    void *staging = nullptr;             // device, N doubles (host double <-> env precision)

    // coefficients and cached factors
    std::vector<double> D, lambda;
    bool factors_valid = false;
    double factor_dt = 0;
    int freeze_factors = 1;
    // per axis: tables [4][n*S] (FP64: den, c, 1/den hi, lo; FP32: 1/den hi,
    // 1/den lo, c1/den, c) and tail values [4][S] for rows [m0, n-2]
    void *fac_tab[3] = {nullptr, nullptr, nullptr};
    void *fac_tail[3] = {nullptr, nullptr, nullptr};
    void *fac_head[3] = {nullptr, nullptr, nullptr};
    int fac_hpad[3] = {4, 4, 4};
    int fac_m0[3] = {1, 1, 1};
    int fac_fast[3] = {0, 0, 0};         // Factors::fast
    void *c1 = nullptr;                  // [S] (FP64)
    void *g = nullptr;                   // [2*S] (FP32): 1/(1 + c2) as hi, lo

    // Dirichlet
    std::vector<uint8_t> activation;     // [S]
    std::vector<uint8_t> face_mask;      // [6*S], already ANDed with activation
    void *faces[6] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    uint8_t *d_mask = nullptr;           // [S]
    int dir_any = 0;

    // bulk
    int bulk_on = 0;
    void *bulkA = nullptr, *bulkB = nullptr;

    // agents
    int n_agents = 0;
    int n_occ = 0;                       // occupied voxels with >= 1 active agent
    int *agent_voxel = nullptr;          // [n_agents], list order (current_voxel_index)
    int *seg_start = nullptr;            // [n_occ + 1]
    int *seg_voxel = nullptr;            // [n_occ]
    void *ag_t1 = nullptr, *ag_t2 = nullptr;  // [n_active][S] in voxel-sorted, list-stable order
    int n_active = 0;
    int *ag_order = nullptr;             // [n_active]: list index of each sorted agent
    // volumes and rates as given to bfb_set_agents (device, list order; valid
    // when rates_known), also for the adjoint's chain rule
    double *ag_vol = nullptr, *ag_sec = nullptr, *ag_upt = nullptr, *ag_sat = nullptr;
    bool rates_known = false;
    double agent_dt = 0;
    void *ag_ws = nullptr;               // the block holding all of the above (agents_layout)
    size_t ag_ws_bytes = 0;
    int ag_end_bit = 1;                  // key bits of the voxel sort
    bool batched = false;                // a batch was made over this env: its streams may read its arrays

    // scratch for reductions
    double *partials = nullptr;
    int partial_blocks = 0;

    // CUDA graph of bfb_simulate
    int use_graphs = 1;
    // bfb_simulate's graphs: graphs[n] replays n steps (made when first needed)
    static constexpr int kGraphSteps = 8;
    cudaGraphExec_t graphs[kGraphSteps + 1] = {};
    int graph_flags = -1;
    double graph_dt = 0;
    uint64_t graph_epoch = 0;            // the epoch the graphs (and the count of steps) belong to
    int graph_seen = 0;                  // steps asked for since then
    uint64_t epoch = 1;                  // bumps whenever captured state changes

    bfb::SweepTuning tuning;

    // TMA: tensor maps of the field for the x and y sweeps (made at creation
    // when the grid meets TMA's alignment rules), and the switch
    int use_tma = 1;
    CUtensorMap tmap[2];
    int tma_crow[2] = {0, 0};
    int tma_lines[2] = {32, 32};  // lines per warp tile of the maps' boxes
    int tma_ok[2] = {0, 0};
    // FP64: maps of 16-row boxes for the tensor-memory x/y sweeps (tuning tma = 2)
    CUtensorMap tmem_map[2];
    int tmem_ok[2] = {0, 0};

    // sticky device error flag (a bounded wait in a kernel ran out)
    int *d_err = nullptr;

    // x-slab of a larger grid (bfb_create_slab): planes [x0, x0 + nx) of
    // nx_global; 0 for a whole grid
    int nx_global = 0;
    int x0 = 0;

    // reverse-mode workspace (bfb_adjoint.cu): one device block, kept between
    // calls and grown on demand, freed by bfb_destroy
    void *adj_ws = nullptr;
    size_t adj_ws_bytes = 0;
};
