// mlp.cu -- training and stand-alone inference of the learned-MDF network on
// the tensor cores (tcgen05), plus the C ABI of the trainer object.
//
// A training step over a batch of n samples runs k_mlp_train_tile (one CTA
// per 128 samples: forward, backward and the CTA's partial weight gradients,
// all GEMMs as tcgen05.mma with BF16 operands and FP32 accumulators in tensor
// memory) and k_mlp_adam (sums the partials in a fixed order, so training is
// deterministic, and applies Adam to the FP32 master weights and their BF16
// operand image).  The batches of a call are one chain of launches that are
// set up while their predecessors run; a row list (the shuffled order of an
// epoch) is followed by the tile's own loads, without a shuffled copy.
//
// Loss: mean over samples and outputs of (y - t)^2 on normalised targets; the
// per-sample output gradient 2 (y - t) / 2 and the batch mean follow the
// reference surrogate network (src/ml/simple_nn.cpp:195-198, :236).
#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/softflow_gpu.h"
#include "launch.cuh"
#include "mlp.cuh"

namespace sfg_host {
void set_error(const std::string& msg);
}

namespace sfg {
namespace mlp {

constexpr int HXW = 96;             // width of [H1 | X | 1 | 0]
constexpr int DZW = 2 * N_H;        // width of [dZ2 | dZ1]
constexpr int TRAIN_THREADS = 2 * ROWS;
constexpr int PART_STRIDE = (N_PARAMS + 3) / 4 * 4;  // 16-byte rows of partial gradients
// Words of the status array: failed waits, and the number of the last training
// call whose row list has an entry out of range.
constexpr int ST_TIMEOUT = 0, ST_BAD_ROW = 1, ST_WORDS = 2;

// Shared-memory image of a training tile.  Every operand is stored once and
// read both ways: along its columns by the layers, and transposed (the sample
// index as K, opdesc_t) by the weight-gradient GEMM; W2 and W3 likewise serve
// the forward and the backward pass.
struct __align__(1024) TrainSmem {
    __nv_bfloat16 HX[ROWS * HXW];    // 24 KB: H1 (0..63), X (64..79), ones (80), zeros
    __nv_bfloat16 DZ[ROWS * DZW];    // 32 KB: dZ2 (0..63), dZ1 (64..127)
    __nv_bfloat16 H2[ROWS * N_H];    // 16 KB
    __nv_bfloat16 dY[ROWS * K1];     // 4 KB: columns 0, 1
    __nv_bfloat16 W1[N_H * K1];      // 2 KB
    __nv_bfloat16 W3[N3 * N_H];      // 2 KB
    __nv_bfloat16 W2[N_H * N_H];     // 8 KB
    float2 dYf[ROWS];
    float b2[N_H], b3[N_OUT];
    float in_mean[N_IN], in_inv_std[N_IN], out_mean[N_OUT], out_std[N_OUT];
    float red[ROWS / 32];
    uint64_t bar;
    uint32_t taddr;
    int error;
};

// The row list's entries that a training call uses, looked at before its first
// update: an entry out of range fails the call with the network as it was.
struct RowCheck {
    const long long* rows;
    long long used, n_rows;
    unsigned* bad_call;
    unsigned call;
};

// norm layout: in_mean[8], in_inv_std[8], out_mean[2], out_std[2]
__global__ void k_build_model(const float* __restrict__ p, const float* __restrict__ norm,
                              ModelDev* __restrict__ md, RowCheck rc) {
    bool bad = false;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < rc.used;
         i += (long long)gridDim.x * blockDim.x)
        bad = bad || rc.rows[i] < 0 || rc.rows[i] >= rc.n_rows;
    if (bad) *rc.bad_call = rc.call;   // (all that meet here store the same)
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < N_H * N_H) build_model_elem(md, p, norm, i);
}

__global__ void __launch_bounds__(ROWS)
k_mlp_forward(const ModelDev* __restrict__ md, const float* __restrict__ x, int n,
              float* __restrict__ y, unsigned* __restrict__ status) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    FwdSmem& s = *reinterpret_cast<FwdSmem*>(smem_raw);
    load_model(s, md);
    start_tiles(s, 128);
    uint32_t phase = 0;
    const int ntiles = (n + ROWS - 1) / ROWS;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int i = tile * ROWS + threadIdx.x;
        const bool valid = i < n;
        float f[N_IN];
#pragma unroll
        for (int k = 0; k < N_IN; ++k) f[k] = valid ? x[(size_t)i * N_IN + k] : 0.0f;
        put_input_row(s, f, valid);
        float out[2];
        if (!forward_tile(s, s.taddr, phase, out)) break;
        if (valid) {
            y[(size_t)i * 2 + 0] = out[0] * s.out_std[0] + s.out_mean[0];
            y[(size_t)i * 2 + 1] = out[1] * s.out_std[1] + s.out_mean[1];
        }
    }
    if (finish_tiles(s, phase, 128) && threadIdx.x == 0) status[ST_TIMEOUT] = 1u;
}

// The gradient through a layer's ReLU: the 16 accumulator columns v where the
// activations H (columns h .. h + 15 of row r) are positive, else 0, into
// columns d .. d + 15 of DZ.
__device__ __forceinline__ void put_gated16(__nv_bfloat16* DZ, int d, const __nv_bfloat16* H,
                                            int h, int HW, int r, float* v) {
#pragma unroll
    for (int half = 0; half < 16; half += 8) {
        const uint4 u = *reinterpret_cast<const uint4*>(H + kmaj(r, h + half, HW));
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t bits = (i & 1) ? (w[i >> 1] & 0xffff0000u) : (w[i >> 1] << 16);
            v[half + i] = __uint_as_float(bits) > 0.0f ? v[half + i] : 0.0f;
        }
        put8(DZ, r, d + half, DZW, v + half);
    }
}

// One CTA: samples [128 b, 128 b + 128) of the batch, sample i being row
// rows[i] of the data (row first + i without a row list).  Writes the CTA's
// partial gradient (N_PARAMS floats) and partial squared error.
//
// Bound: one tile's chain of latencies (six rounds of MMAs with their barriers
// and TMEM reads); a batch of 8192 samples is 64 CTAs.  So the weights arrive
// ready-made in the operand layouts (k_mlp_adam keeps the image), no operand
// is transposed through shared memory, warps 4-7 do the layer-3 gradients
// beside the backward rounds of warps 0-3, and the samples are loaded before
// the wait for the previous step.  Batch of 8192, cold caches: 26.0 us with conversion,
// transposed copies and layer 3 at the end, 10.7 us so.
__global__ void __launch_bounds__(TRAIN_THREADS)
k_mlp_train_tile(const ModelDev* md, const float* __restrict__ x,
                 const float* __restrict__ t, const long long* __restrict__ rows, long long first,
                 long long n_rows, int n, float inv_n, float* __restrict__ part,
                 float* __restrict__ part_loss, unsigned* __restrict__ status) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    TrainSmem& s = *reinterpret_cast<TrainSmem*>(smem_raw);
    const int r = threadIdx.x;
    const bool chain = r < ROWS;  // warps 0-3: one sample each
    const int i = blockIdx.x * ROWS + r;
    // The samples are no kernel of the chain's work (the chain's first kernel
    // is launched without overlap): they may be read before the wait.
    bool valid = chain && i < n;
    float f[N_IN] = {}, tr[N_OUT] = {};
    if (valid) {
        const long long row = rows ? rows[first + i] : first + i;
        valid = row >= 0 && row < n_rows;   // (the others fail the call: RowCheck)
        if (valid) {
#pragma unroll
            for (int k = 0; k < N_IN; ++k) f[k] = x[row * N_IN + k];
#pragma unroll
            for (int k = 0; k < N_OUT; ++k) tr[k] = t[row * N_OUT + k];
        }
    }
    chain_begin();
    load_model<TRAIN_THREADS>(s, md);
    // only now: a later step's CTAs must not hold tensor memory that this
    // step's still wait for
    start_tiles(s, 256);
    uint32_t phase = 0;
    const uint32_t tb = s.taddr;
    float* gp = part + (size_t)blockIdx.x * PART_STRIDE;
    bool ok = true;
    if (chain) {
        put_input_cols(s, s.HX, N_H, HXW, f, valid);
        {
            // the ones column (bias gradient of layer 2), then zeros
            float v[8] = {1.0f};
            put8(s.HX, r, 80, HXW, v);
            v[0] = 0.0f;
            put8(s.HX, r, 88, HXW, v);
        }
        float v[16];
        ok = mma_round<true>(s, phase, [&] {
            mma(tb, opdesc(s.HX + kmaj(0, N_H, HXW), HXW, 0), opdesc(s.W1, K1, 0),
                idesc_bf16(ROWS, N_H), 0u);
        });
        if (ok) {
#pragma unroll
            for (int c = 0; c < N_H; c += 16) {
                tmem_ld16(tmem_row(tb, c), v);
                put_relu16(s.HX, r, c, HXW, v, nullptr);
            }
            ok = mma_round<true>(s, phase, [&] {
#pragma unroll
                for (int kk = 0; kk < N_H / 16; ++kk)
                    mma(tb + 64, opdesc(s.HX, HXW, kk), opdesc(s.W2, N_H, kk),
                        idesc_bf16(ROWS, N_H), kk > 0 ? 1u : 0u);
            });
        }
        if (ok) {
#pragma unroll
            for (int c = 0; c < N_H; c += 16) {
                tmem_ld16(tmem_row(tb, 64 + c), v);
                put_relu16(s.H2, r, c, N_H, v, s.b2 + c);
            }
            ok = mma_round<true>(s, phase, [&] {
#pragma unroll
                for (int kk = 0; kk < N_H / 16; ++kk)
                    mma(tb, opdesc(s.H2, N_H, kk), opdesc(s.W3, N_H, kk), idesc_bf16(ROWS, N3),
                        kk > 0 ? 1u : 0u);
            });
        }
        float y[2] = {0.0f, 0.0f};
        if (ok) {
            tmem_ld16(tmem_row(tb, 0), v);
            y[0] = v[0] + s.b3[0];
            y[1] = v[1] + s.b3[1];
        }
        float dy0 = 0.0f, dy1 = 0.0f, se = 0.0f;
        if (valid) {
            const float t0 = (tr[0] - s.out_mean[0]) / s.out_std[0];
            const float t1 = (tr[1] - s.out_mean[1]) / s.out_std[1];
            const float e0 = y[0] - t0, e1 = y[1] - t1;
            se = e0 * e0 + e1 * e1;
            dy0 = e0 * inv_n;
            dy1 = e1 * inv_n;
        }
        s.dYf[r] = make_float2(dy0, dy1);
        {
            float d[8] = {dy0, dy1};
            put8(s.dY, r, 0, K1, d);
            d[0] = d[1] = 0.0f;
            put8(s.dY, r, 8, K1, d);
        }
        // squared error of the CTA
        for (int o = 16; o > 0; o >>= 1) se += __shfl_down_sync(0xffffffffu, se, o);
        if ((r & 31) == 0) s.red[r >> 5] = se;
    }
    __syncthreads();  // dYf, H2 and red are complete
    if (!chain) {
        // layer-3 gradients on the CUDA cores: dW3 = dY^T H2, db3 = sum dY,
        // each one sum over the samples in order
        const int u = r - ROWS;
        if (u < N_H) {
            float a0 = 0.0f, a1 = 0.0f;
#pragma unroll 16
            for (int q = 0; q < ROWS; ++q) {
                const float h = __bfloat162float(s.H2[kmaj(q, u, N_H)]);
                const float2 d = s.dYf[q];
                a0 = fmaf(d.x, h, a0);
                a1 = fmaf(d.y, h, a1);
            }
            gp[P_W3 + u] = a0;
            gp[P_W3 + N_H + u] = a1;
        } else if (u == N_H) {
            float d0 = 0.0f, d1 = 0.0f;
#pragma unroll 16
            for (int q = 0; q < ROWS; ++q) {
                const float2 d = s.dYf[q];
                d0 += d.x;
                d1 += d.y;
            }
            gp[P_B3 + 0] = d0;
            gp[P_B3 + 1] = d1;
        } else if (u == N_H + 32) {
            part_loss[blockIdx.x] = s.red[0] + s.red[1] + s.red[2] + s.red[3];
        }
    } else {
        float v[16];
        // dH2 = dY W3 -> columns [0, 64)
        if (ok)
            ok = mma_round<true>(s, phase, [&] {
                mma(tb, opdesc(s.dY, K1, 0), opdesc_t(s.W3, N_H, 0),
                    idesc_bf16(ROWS, N_H) | B_MN_MAJOR, 0u);
            });
        if (ok) {
#pragma unroll
            for (int c = 0; c < N_H; c += 16) {
                tmem_ld16(tmem_row(tb, c), v);
                put_gated16(s.DZ, c, s.H2, c, N_H, r, v);
            }
            // dH1 = dZ2 W2 -> columns [64, 128)
            ok = mma_round<true>(s, phase, [&] {
#pragma unroll
                for (int kk = 0; kk < N_H / 16; ++kk)
                    mma(tb + 64, opdesc(s.DZ, DZW, kk), opdesc_t(s.W2, N_H, kk),
                        idesc_bf16(ROWS, N_H) | B_MN_MAJOR, kk > 0 ? 1u : 0u);
            });
        }
        if (ok) {
#pragma unroll
            for (int c = 0; c < N_H; c += 16) {
                tmem_ld16(tmem_row(tb, 64 + c), v);
                put_gated16(s.DZ, N_H + c, s.HX, c, HXW, r, v);
            }
            // [dZ2 | dZ1]^T [H1 | X | 1] -> columns [128, 224)
            ok = mma_round<true>(s, phase, [&] {
#pragma unroll
                for (int kk = 0; kk < ROWS / 16; ++kk)
                    mma(tb + 128, opdesc_t(s.DZ, DZW, kk), opdesc_t(s.HX, HXW, kk),
                        idesc_bf16(ROWS, HXW) | A_MN_MAJOR | B_MN_MAJOR, kk > 0 ? 1u : 0u);
            });
        }
        if (ok && r < N_H) {
            float4* g2 = reinterpret_cast<float4*>(gp + P_W2 + r * N_H);
#pragma unroll
            for (int c = 0; c < N_H; c += 16) {
                tmem_ld16(tmem_row(tb, 128 + c), v);
#pragma unroll
                for (int j = 0; j < 16; j += 4)
                    g2[(c + j) / 4] = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
            }
            tmem_ld16(tmem_row(tb, 128 + 80), v);
            gp[P_B2 + r] = v[0];
        } else if (ok) {
            // warps 2 and 3: rows 64..127 are dW1 (columns 64..71) and db1 (72)
            const int o = r - N_H;
            tmem_ld16(tmem_row(tb, 128 + 64), v);
            float4* g1 = reinterpret_cast<float4*>(gp + P_W1 + o * N_IN);
            g1[0] = make_float4(v[0], v[1], v[2], v[3]);
            g1[1] = make_float4(v[4], v[5], v[6], v[7]);
            gp[P_B1 + o] = v[N_IN];
        }
    }
    if (finish_tiles(s, phase, 256) && r == 0) status[ST_TIMEOUT] = 1u;
}

// The parameter's place in the operand image.
__device__ __forceinline__ void put_param(ModelDev* md, int i, float w) {
    const __nv_bfloat16 h = __float2bfloat16_rn(w);
    if (i < P_B1) md->W1[kmaj(i / N_IN, i % N_IN, K1)] = h;
    else if (i < P_W2) md->W1[kmaj(i - P_B1, N_IN, K1)] = h;
    else if (i < P_B2) md->W2[kmaj((i - P_W2) / N_H, (i - P_W2) % N_H, N_H)] = h;
    else if (i < P_W3) md->b2[i - P_B2] = w;
    else if (i < P_B3) md->W3[kmaj((i - P_W3) / N_H, (i - P_W3) % N_H, N_H)] = h;
    else md->b3[i - P_B3] = w;
}

// Sums the CTA partials in CTA order; then Adam (step > 0), which also renews
// the parameter in the operand image, or the plain gradient into g_out
// (step == 0).  The last warp of the grid adds up the loss, also in CTA order.
//
// Bound: the latency of the loads (4866 sums over 64 partials for a batch of
// 8192), so 32 loads are in flight per thread, the threads lie on 77 CTAs, and the
// loss's partials are loaded by 32 lanes: 7.3 us -> 5.5 us (of that the loss alone,
// by one thread, had taken longer than all else).
constexpr int ADAM_THREADS = 64, ADAM_LOADS = 32;
constexpr int ADAM_BLOCKS = (N_PARAMS + ADAM_THREADS - 1) / ADAM_THREADS + 1;
__global__ void __launch_bounds__(ADAM_THREADS)
k_mlp_adam(float* p, float* m, float* v, const float* part, int nparts, int step, float lr,
           float* __restrict__ g_out, const float* part_loss, float loss_scale,
           float* __restrict__ loss_out, ModelDev* __restrict__ md, const unsigned* bad_call,
           unsigned call) {
    chain_begin();
    if (blockIdx.x == gridDim.x - 1) {
        const int lane = threadIdx.x;
        if (lane >= 32 || !loss_out) return;
        float l = 0.0f;
        for (int c0 = 0; c0 < nparts; c0 += 32) {
            const float q = c0 + lane < nparts ? part_loss[c0 + lane] : 0.0f;
            const int cnt = min(32, nparts - c0);
            for (int c = 0; c < cnt; ++c) l += __shfl_sync(0xffffffffu, q, c);
        }
        if (lane == 0) *loss_out = l * loss_scale;
        return;
    }
    const int i = blockIdx.x * ADAM_THREADS + threadIdx.x;
    if (i >= N_PARAMS) return;
    const float m0 = m[i], v0 = v[i], p0 = p[i];
    const bool keep = *bad_call == call;   // the call will fail: nothing is updated
    float g = 0.0f;
    int c = 0;
    for (; c + ADAM_LOADS <= nparts; c += ADAM_LOADS) {
        float q[ADAM_LOADS];
#pragma unroll
        for (int j = 0; j < ADAM_LOADS; ++j) q[j] = part[(size_t)(c + j) * PART_STRIDE + i];
#pragma unroll
        for (int j = 0; j < ADAM_LOADS; ++j) g += q[j];
    }
#pragma unroll 4
    for (; c < nparts; ++c) g += part[(size_t)c * PART_STRIDE + i];
    if (g_out) g_out[i] = g;
    if (step <= 0 || keep) return;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    // the rounding is written out: left to the compiler, which product is fused
    // depends on where the loads stand
    const float mi = fmaf(1.0f - b1, g, b1 * m0);
    const float vi = fmaf((1.0f - b2) * g, g, b2 * v0);
    m[i] = mi;
    v[i] = vi;
    const float mh = mi / (1.0f - powf(b1, (float)step));
    const float vh = vi / (1.0f - powf(b2, (float)step));
    const float w = p0 - lr * mh / (sqrtf(vh) + eps);
    p[i] = w;
    put_param(md, i, w);
}

}  // namespace mlp
}  // namespace sfg

// ============================================================== C ABI

using namespace sfg::mlp;

struct sfg_mlp {
    int device = 0;
    float* d_params = nullptr;
    float* d_m = nullptr;
    float* d_v = nullptr;
    float* d_norm = nullptr;
    sfg::mlp::ModelDev* d_model = nullptr;  // forward's and the step's, built on demand
    sfg::mlp::ModelDev* d_train = nullptr;  // the training steps' own, renewed by each
    float* d_part = nullptr;
    float* d_part_loss = nullptr;
    float* d_loss = nullptr;
    float* d_grad = nullptr;
    unsigned* d_status = nullptr;   // [ST_WORDS]
    unsigned call = 0;              // training and gradient calls so far (never 0 in one)
    int part_cap = 0;
    int step = 0;
    bool model_dirty = true;
};

namespace {

int fail(int code, const std::string& msg) {
    sfg_host::set_error(msg);
    return code;
}

#define MCU(x)                                                                       \
    do {                                                                             \
        cudaError_t e_ = (x);                                                        \
        if (e_ != cudaSuccess)                                                       \
            return fail(SFG_ERR_CUDA, std::string(#x) + ": " + cudaGetErrorString(e_)); \
    } while (0)

int ensure_parts(sfg_mlp* m, int nparts) {
    if (nparts <= m->part_cap) return SFG_OK;
    if (m->d_part) cudaFree(m->d_part);
    if (m->d_part_loss) cudaFree(m->d_part_loss);
    m->d_part = nullptr;
    m->d_part_loss = nullptr;
    MCU(cudaMalloc(&m->d_part, sizeof(float) * (size_t)nparts * PART_STRIDE));
    MCU(cudaMalloc(&m->d_part_loss, sizeof(float) * nparts));
    m->part_cap = nparts;
    return SFG_OK;
}

int check_status(sfg_mlp* m, cudaStream_t st, const char* who, bool training = false) {
    unsigned s[ST_WORDS] = {0};
    MCU(cudaMemcpyAsync(s, m->d_status, sizeof s, cudaMemcpyDeviceToHost, st));
    MCU(cudaStreamSynchronize(st));
    if (s[ST_TIMEOUT])
        return fail(SFG_ERR_CUDA, std::string(who) + ": a tensor-core wait timed out");
    if (training && s[ST_BAD_ROW] == m->call)
        return fail(SFG_ERR_ARG, std::string(who) + ": row index out of range");
    return SFG_OK;
}

int prepare_kernels(int device) {
    static unsigned long long done = 0;  // one bit per device ordinal below 64
    const unsigned long long bit = (device >= 0 && device < 64) ? (1ull << device) : 0ull;
    if (bit && (done & bit)) return SFG_OK;
    MCU(cudaFuncSetAttribute(k_mlp_train_tile, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(TrainSmem)));
    MCU(cudaFuncSetAttribute(k_mlp_forward, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(FwdSmem)));
    done |= bit;
    return SFG_OK;
}

struct Samples {
    const float *x, *t;
    const long long* rows;  // null: consecutive rows
    long long n_rows;
};

// one batch: partial gradients, then the reduction (+ Adam when step > 0).
// `chained`: the stream's previous operation is the batch before it.
int batch_step(sfg_mlp* m, const Samples& d, long long first, int n, int step, float lr,
               float* g_out, float* loss_out, bool chained, cudaStream_t st) {
    const int nparts = (n + ROWS - 1) / ROWS;
    sfg::launch_chain(chained, k_mlp_train_tile, nparts, TRAIN_THREADS, sizeof(TrainSmem), st,
                      m->d_train, d.x, d.t, d.rows, first, d.n_rows, n, 1.0f / (float)n,
                      m->d_part, m->d_part_loss, m->d_status);
    MCU(cudaGetLastError());
    sfg::launch_chain(true, k_mlp_adam, ADAM_BLOCKS, ADAM_THREADS, 0, st, m->d_params, m->d_m,
                      m->d_v, m->d_part, nparts, step, lr, g_out, m->d_part_loss,
                      1.0f / (2.0f * (float)n), loss_out, m->d_train,
                      m->d_status + ST_BAD_ROW, m->call);
    MCU(cudaGetLastError());
    if (step > 0) m->model_dirty = true;
    return SFG_OK;
}

// The training image of the current parameters and normalisation, room for one
// batch's partial gradients, and the check of the first `used` entries of the row
// list (if any) into data of n_rows.
int begin_training(sfg_mlp* m, int batch, const long long* rows, long long used, long long n_rows,
                   cudaStream_t st) {
    int rc = ensure_parts(m, (batch + ROWS - 1) / ROWS);
    if (rc) return rc;
    if (++m->call == 0u) m->call = 1u;
    const RowCheck check{rows, rows ? used : 0, n_rows, m->d_status + ST_BAD_ROW, m->call};
    const long long grid = std::max((long long)(N_H * N_H + 255) / 256,
                                    std::min(256LL, (check.used + 255) / 256));
    k_build_model<<<(unsigned)grid, 256, 0, st>>>(m->d_params, m->d_norm, m->d_train, check);
    MCU(cudaGetLastError());
    return SFG_OK;
}

}  // namespace

extern "C" int sfg_mlp_create(int device, sfg_mlp** out) {
    if (!out) return fail(SFG_ERR_ARG, "sfg_mlp_create: null output");
    *out = nullptr;
    MCU(cudaSetDevice(device));
    int rc = prepare_kernels(device);
    if (rc) return rc;
    sfg_mlp* m = new sfg_mlp();
    m->device = device;
    cudaError_t e = cudaSuccess;
    if (e == cudaSuccess) e = cudaMalloc(&m->d_params, sizeof(float) * N_PARAMS);
    if (e == cudaSuccess) e = cudaMalloc(&m->d_m, sizeof(float) * N_PARAMS);
    if (e == cudaSuccess) e = cudaMalloc(&m->d_v, sizeof(float) * N_PARAMS);
    if (e == cudaSuccess) e = cudaMalloc(&m->d_grad, sizeof(float) * N_PARAMS);
    if (e == cudaSuccess) e = cudaMalloc(&m->d_norm, sizeof(float) * 20);
    if (e == cudaSuccess) e = cudaMalloc(&m->d_model, sizeof(sfg::mlp::ModelDev));
    if (e == cudaSuccess) e = cudaMalloc(&m->d_train, sizeof(sfg::mlp::ModelDev));
    if (e == cudaSuccess) e = cudaMalloc(&m->d_loss, sizeof(float) * 4096);
    if (e == cudaSuccess) e = cudaMalloc(&m->d_status, sizeof(unsigned) * ST_WORDS);
    if (e == cudaSuccess) e = cudaMemset(m->d_params, 0, sizeof(float) * N_PARAMS);
    if (e == cudaSuccess) e = cudaMemset(m->d_m, 0, sizeof(float) * N_PARAMS);
    if (e == cudaSuccess) e = cudaMemset(m->d_v, 0, sizeof(float) * N_PARAMS);
    if (e == cudaSuccess) e = cudaMemset(m->d_status, 0, sizeof(unsigned) * ST_WORDS);
    if (e == cudaSuccess) {
        float norm[20];
        for (int i = 0; i < 20; ++i) norm[i] = (i < 8 || (i >= 16 && i < 18)) ? 0.0f : 1.0f;
        e = cudaMemcpy(m->d_norm, norm, sizeof(norm), cudaMemcpyHostToDevice);
    }
    if (e != cudaSuccess) {
        sfg_mlp_destroy(m);
        return fail(SFG_ERR_CUDA, std::string("sfg_mlp_create: ") + cudaGetErrorString(e));
    }
    *out = m;
    return SFG_OK;
}

extern "C" int sfg_mlp_destroy(sfg_mlp* m) {
    if (!m) return SFG_OK;
    cudaSetDevice(m->device);
    for (void* p : {(void*)m->d_params, (void*)m->d_m, (void*)m->d_v, (void*)m->d_norm,
                    (void*)m->d_model, (void*)m->d_train, (void*)m->d_part, (void*)m->d_part_loss,
                    (void*)m->d_loss, (void*)m->d_grad, (void*)m->d_status})
        if (p) cudaFree(p);
    delete m;
    return SFG_OK;
}

extern "C" int sfg_mlp_set_params(sfg_mlp* m, const float* params) {
    if (!m || !params) return fail(SFG_ERR_ARG, "sfg_mlp_set_params: null argument");
    MCU(cudaSetDevice(m->device));
    MCU(cudaMemcpy(m->d_params, params, sizeof(float) * N_PARAMS, cudaMemcpyHostToDevice));
    MCU(cudaMemset(m->d_m, 0, sizeof(float) * N_PARAMS));
    MCU(cudaMemset(m->d_v, 0, sizeof(float) * N_PARAMS));
    m->step = 0;
    m->model_dirty = true;
    return SFG_OK;
}

extern "C" int sfg_mlp_get_params(sfg_mlp* m, float* params) {
    if (!m || !params) return fail(SFG_ERR_ARG, "sfg_mlp_get_params: null argument");
    MCU(cudaSetDevice(m->device));
    MCU(cudaDeviceSynchronize());
    MCU(cudaMemcpy(params, m->d_params, sizeof(float) * N_PARAMS, cudaMemcpyDeviceToHost));
    return SFG_OK;
}

extern "C" int sfg_mlp_set_normalization(sfg_mlp* m, const float* in_mean, const float* in_std,
                                         const float* out_mean, const float* out_std) {
    if (!m || !in_mean || !in_std || !out_mean || !out_std)
        return fail(SFG_ERR_ARG, "sfg_mlp_set_normalization: null argument");
    float norm[20];
    for (int k = 0; k < 8; ++k) {
        if (!(in_std[k] > 0.0f)) return fail(SFG_ERR_ARG, "sfg_mlp_set_normalization: in_std <= 0");
        norm[k] = in_mean[k];
        norm[8 + k] = 1.0f / in_std[k];
    }
    for (int k = 0; k < 2; ++k) {
        if (!(out_std[k] > 0.0f)) return fail(SFG_ERR_ARG, "sfg_mlp_set_normalization: out_std <= 0");
        norm[16 + k] = out_mean[k];
        norm[18 + k] = out_std[k];
    }
    MCU(cudaSetDevice(m->device));
    MCU(cudaMemcpy(m->d_norm, norm, sizeof(norm), cudaMemcpyHostToDevice));
    m->model_dirty = true;
    return SFG_OK;
}

// Device image of the model in operand layout (built when parameters or
// normalisation changed); used by the forward kernel and the step.
int sfg_mlp_model_device(sfg_mlp* m, const void** model, cudaStream_t st) {
    if (m->model_dirty) {
        k_build_model<<<(N_H * N_H + 255) / 256, 256, 0, st>>>(m->d_params, m->d_norm, m->d_model,
                                                               RowCheck{});
        MCU(cudaGetLastError());
        m->model_dirty = false;
    }
    *model = m->d_model;
    return SFG_OK;
}

extern "C" int sfg_mlp_forward(sfg_mlp* m, const float* d_x, int n, float* d_y, void* stream) {
    if (!m || (n > 0 && (!d_x || !d_y))) return fail(SFG_ERR_ARG, "sfg_mlp_forward: null argument");
    if (n < 0) return fail(SFG_ERR_ARG, "sfg_mlp_forward: negative count");
    if (n == 0) return SFG_OK;
    MCU(cudaSetDevice(m->device));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const void* md = nullptr;
    int rc = sfg_mlp_model_device(m, &md, st);
    if (rc) return rc;
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, m->device);
    const int tiles = (n + ROWS - 1) / ROWS;
    const int grid = tiles < 4 * sms ? tiles : 4 * sms;
    k_mlp_forward<<<grid, ROWS, sizeof(FwdSmem), st>>>(
        static_cast<const sfg::mlp::ModelDev*>(md), d_x, n, d_y, m->d_status);
    MCU(cudaGetLastError());
    return check_status(m, st, "sfg_mlp_forward");
}

extern "C" int sfg_mlp_gradients(sfg_mlp* m, const float* d_x, const float* d_t, int n,
                                 float* grad, float* loss, void* stream) {
    if (!m || !d_x || !d_t || !grad) return fail(SFG_ERR_ARG, "sfg_mlp_gradients: null argument");
    if (n <= 0) return fail(SFG_ERR_ARG, "sfg_mlp_gradients: empty batch");
    MCU(cudaSetDevice(m->device));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int rc = begin_training(m, n, nullptr, 0, n, st);
    if (rc) return rc;
    rc = batch_step(m, {d_x, d_t, nullptr, n}, 0, n, 0, 0.0f, m->d_grad, m->d_loss, false, st);
    if (rc) return rc;
    if ((rc = check_status(m, st, "sfg_mlp_gradients"))) return rc;
    MCU(cudaMemcpy(grad, m->d_grad, sizeof(float) * N_PARAMS, cudaMemcpyDeviceToHost));
    if (loss) MCU(cudaMemcpy(loss, m->d_loss, sizeof(float), cudaMemcpyDeviceToHost));
    return SFG_OK;
}

extern "C" int sfg_mlp_train_rows(sfg_mlp* m, const float* d_x, const float* d_t,
                                  const long long* d_rows, int n, int batch, float lr,
                                  float* losses, void* stream) {
    if (!m || !d_x || !d_t) return fail(SFG_ERR_ARG, "sfg_mlp_train: null argument");
    if (n <= 0 || batch <= 0) return fail(SFG_ERR_ARG, "sfg_mlp_train: empty data or batch");
    MCU(cudaSetDevice(m->device));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int nb = n / batch;
    if (nb < 1) return fail(SFG_ERR_ARG, "sfg_mlp_train: fewer samples than one batch");
    int rc = begin_training(m, batch, d_rows, (long long)nb * batch, n, st);
    if (rc) return rc;
    const int step0 = m->step;
    const Samples d{d_x, d_t, d_rows, n};
    for (int b0 = 0; b0 < nb; b0 += 4096) {
        const int cnt = nb - b0 < 4096 ? nb - b0 : 4096;
        for (int k = 0; k < cnt; ++k) {
            rc = batch_step(m, d, (long long)(b0 + k) * batch, batch, ++m->step, lr, nullptr,
                            m->d_loss + k, k > 0, st);
            if (rc) return rc;
        }
        if (losses) {
            MCU(cudaMemcpyAsync(losses + b0, m->d_loss, sizeof(float) * cnt,
                                cudaMemcpyDeviceToHost, st));
        }
    }
    rc = check_status(m, st, "sfg_mlp_train", true);
    if (rc == SFG_ERR_ARG) m->step = step0;   // (no batch was applied)
    return rc;
}

extern "C" int sfg_mlp_train(sfg_mlp* m, const float* d_x, const float* d_t, int n, int batch,
                             float lr, float* losses, void* stream) {
    return sfg_mlp_train_rows(m, d_x, d_t, nullptr, n, batch, lr, losses, stream);
}

extern "C" int sfg_mlp_step_count(sfg_mlp* m, int* steps) {
    if (!m || !steps) return fail(SFG_ERR_ARG, "sfg_mlp_step_count: null argument");
    *steps = m->step;
    return SFG_OK;
}
