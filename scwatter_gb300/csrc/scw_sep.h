// Separable-form coefficient set and shared declarations of the GEMM-form evaluator.
#pragma once

#include <cuda_runtime.h>
#include <vector>

#include "scw_internal.h"
#include "scw_launch.h"

namespace scw {

constexpr int kMaxGroup = 8;   // z-planes contracted together in stage 1

// z-planes of one region handled by one stage-1 pass
struct PGroup {
    int region;
    int nk;
    int zi[kMaxGroup];
};

// A planned evaluation of a separable set: the z-planes, their stage-1 grouping, the device
// descriptor block (groups, exterior planes, z-values) and the scratch it needs.
struct SepEvalPlan {
    int kind = 0, Na = 0, Nb = 0, Nz = 0, method = 0;
    float a0 = 0, b0 = 0, c = 0, da = 0, db = 0, dz = 0;
    std::vector<float> zlist;
    std::vector<PGroup> groups;
    std::vector<int2> ext;
    int max_nk = 1;
    size_t off_e = 0, off_z = 0, desc_bytes = 0;
    int nrows = 0, ncols = 0, Mk = 0;
    size_t phi_bytes = 0, c_bytes = 0, t_bytes = 0, tab_bytes = 0, scratch_bytes = 0;
};
// A plan's descriptor block as stage 1's kernels get it: a device address, or (dev null) the block itself among the
// kernel parameters.  Uploading it first cost a copy of 1 us that the host took 11 us to submit and the first kernel
// waited 14 us for, as long as all of a small volume's kernels; a block that fits goes with the launches.
constexpr size_t kDescInline = 3584;       // 64 groups and 256 planes; all parameters of a kernel below 4 KB
struct SepDesc {
    const char* dev;
    alignas(16) char here[kDescInline];
    __device__ __forceinline__ const char* base() const { return dev ? dev : here; }
};
// kind 0: Nz xy planes (a = x, b = y); 1: xz plane at y = c; 2: yz plane at x = c
scw_status sep_eval_plan(const scw_sep_s* s, int kind, float a0, float b0, float c, float da, float db, float dz,
                         int Na, int Nb, int Nz, int method, SepEvalPlan& p);
void sep_eval_desc(const SepEvalPlan& p, char* host);
// launches only, on the set's context stream; d_desc null: the plan's block (at most kDescInline bytes) goes with them
// chained: each kernel may be set up while the one before it in the stream ends (launch_chained)
scw_status sep_eval_record(scw_sep_s* s, const SepEvalPlan& p, const char* d_desc, char* scratch, float* dE,
                           bool chained = false);


// output GEMM of stage 2: E[r][col][c] = sum_m T[r][c][m] F[m][col]
scw_status sep_synth(scw_ctx ctx, const float2* T, const float2* F, int nrows, int ncols, int Mk, float* out,
                     int method, bool chained);
// tensor-core version (eval_sep_tc.cu); SCW_ERR_UNSUPPORTED when the shape is outside it
scw_status sep_synth_tc(scw_ctx ctx, const float2* T, const float2* F, int nrows, int ncols, int Mk, float* out,
                        int method, bool chained);

}  // namespace scw

struct scw_sep_s {
    scw_ctx ctx = nullptr;
    int device = -1;                        // the context's: it may be gone when this is freed
    int M0 = 0, M1 = 0, MF = 0, Z = 0, J = 0;
    int Jp = 0;                            // J rounded up to even: row stride of Q / kz on the device (zero padded)
    int rule = 0;
    std::vector<double> kx, ky, zb;
    std::vector<float> z_layers;           // Z + 1 boundaries as float (region rule)
    double* dkx = nullptr;
    double* dky = nullptr;
    double* dzb = nullptr;
    double2* dExt = nullptr;               // inc[3][MF], refl[3][MF], trans[3][MF], kz_inc, kz_refl, kz_trans
    double2* dKz = nullptr;                // [Z][2][Jp] kz of the downward / upward modes
    // Interior amplitudes, in one of two forms:
    //   halves = 2: dQ [Z][2][3][MF][Jp], the downward and upward blocks Q_dn, Q_up as given;
    //   halves = 1 ("paired"): dQ [Z][3][MF][Jp] holds one block V and dBeta [Z][2][Jp] the mode
    //     amplitudes, with Q_dn = V diag(beta_dn) and Q_up = S V diag(beta_up), S = diag(+1, +1, -1)
    //     over (Ex, Ey, Ez) -- the structure of the solver's modes, whose E rows are the same
    //     eigenvector for the two roots +-gamma and whose H rows (hence Ez) change sign.
    int halves = 2;
    // contraction tile shape: 0 = the default rows per warp for the launch's planes per group (8 for one or two
    // planes, 4 for 3 to 8; half as many where that leaves SMs without a CTA), 1 = half as many always;
    // chosen by the batch autotuner
    int ctr_shape = 0;
    float2* dQ = nullptr;
    double2* dBeta = nullptr;
    bool own_Q = false;
    // host-streamed evaluation (scw_sep_eval_volume_host): copy streams, events, output slabs
    cudaStream_t up_stream = nullptr, down_stream = nullptr;
    std::vector<cudaEvent_t> events;
    // pipelined device volumes: stage 2 of one chunk of planes on hi_stream (high priority) while
    // stage 1 of the next runs on the context stream
    cudaStream_t hi_stream = nullptr;
    // the viewer's second and third plane run beside the first (scw_sep_gpu_cw_evaluate)
    cudaStream_t plane_stream[2] = {nullptr, nullptr};
    cudaEvent_t plane_event[4] = {nullptr, nullptr, nullptr, nullptr};   // start, xz done, yz done, C of both
    std::vector<cudaEvent_t> pevents;
    int pipe_chunks = 0;                   // chunks of a pipelined slab (0 or 1: one pass)
    int pipe_synth_div = 2;                // the pipelined output GEMM runs on sm_count / pipe_synth_div SMs
    void* dslab = nullptr;                 // output slab ring (device)
    size_t slab_bytes = 0;
    size_t chunk_bytes = 0, slab_target = 0;   // scw_sep_set_streaming (0: defaults)
};
