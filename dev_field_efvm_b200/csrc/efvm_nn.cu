// efvm_nn.cu — BF16 tensor-core (tcgen05) kernels of the learned flux correction.
//
// This file holds the tensor-core GEMM tile that the correction network's
// forward and backward kernels are built from, and a stand-alone entry point
// that runs it on caller matrices (used to check the tile against a CPU
// product).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "efvm_internal.h"
#include "efvm_tc.cuh"

namespace efvm {
namespace {

__device__ int g_nn_error;  // set by a kernel whose tensor-core wait ran out

__host__ __device__ constexpr int tmem_cols_for(int n) { return n <= 32 ? 32 : n <= 64 ? 64 : n <= 128 ? 128 : 256; }

// D[M x N] = A[M x K] * B[N x K]^T, row-major BF16 inputs (K contiguous), FP32
// output; one CTA of 128 threads per 128 rows of A.
__global__ void __launch_bounds__(128) nn_gemm_kernel(const __nv_bfloat16* __restrict__ A,
                                                      const __nv_bfloat16* __restrict__ B, float* __restrict__ D,
                                                      int N, int K) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tslot;
    unsigned char* sa = smem;
    unsigned char* sb = smem + 128 * K * 2;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const long long m0 = (long long)blockIdx.x * 128;
    for (int idx = tid; idx < 128 * K; idx += 128) {
        const int r = idx / K, k = idx - r * K;
        *reinterpret_cast<__nv_bfloat16*>(sa + tc::canon_offset(r, k, 128)) = A[(m0 + r) * K + k];
    }
    for (int idx = tid; idx < N * K; idx += 128) {
        const int r = idx / K, k = idx - r * K;
        *reinterpret_cast<__nv_bfloat16*>(sb + tc::canon_offset(r, k, N)) = B[(long long)r * K + k];
    }
    const uint32_t ncols = (uint32_t)tmem_cols_for(N);
    if (warp == 0) tc::tmem_alloc(&tslot, ncols);
    if (tid == 0) tc::mbar_init(&bar, 1);
    tc::fence_smem_to_async();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tslot;
    tc::gemm_issue(tmem, sa, sb, N, K, &bar);
    bool ok = tc::mbar_wait(&bar, 0);
    ok = __syncthreads_and(ok);
    if (!ok) {
        if (tid == 0) atomicExch(&g_nn_error, 1);
        tc::mbar_wait(&bar, 0);  // give the MMA a second bounded chance to retire before TMEM is released
    } else {
        tc::fence_after_sync();
        for (int c0 = 0; c0 < N; c0 += 16) {
            float v[16];
            tc::tmem_ld16(tmem, c0, v);
            float* out = D + (m0 + 32 * warp + lane) * N + c0;
#pragma unroll
            for (int i = 0; i < 16; ++i) out[i] = v[i];
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_free(tmem, ncols);
}


// ===========================================================================
// The correction network.  Per face, the 5 x 5 stencil of primitive variables
// (rho - 1, normal velocity, tangential velocity, p - 1) in the face's own
// frame (x faces as they are; y faces transposed with u and v swapped, so one
// network serves both orientations) feeds
//     h1 = relu(W1 x + b1)   (100 -> 32, K padded to 112)
//     h2 = relu(W2 h1 + b2)  (32 -> 32)
//     y  = W3 h2 + b3        (32 -> 4, N padded to 16)
// and out_scale * y is the correction (rho, m_n, m_t, E) added to that face's
// flux.  Weights are BF16 on the tensor cores, biases and accumulation FP32.
// One CTA of 128 threads handles 128 faces; thread r owns face r of the tile.
// ===========================================================================
namespace nn {

constexpr int IN = 100, K1 = 112, H = 32, NOUT = 4, N3 = 16;
constexpr int P_W1 = 0, P_W2 = P_W1 + H * K1, P_W3 = P_W2 + H * H, P_B1 = P_W3 + NOUT * H, P_B2 = P_B1 + H,
              P_B3 = P_B2 + H, P_COUNT = P_B3 + NOUT;

struct Net {
    const __nv_bfloat16* w1;  // [H][K1], columns >= IN zero
    const __nv_bfloat16* w2;  // [H][H]
    const __nv_bfloat16* w3;  // [N3][H], rows >= NOUT zero
    const float* p;           // FP32 parameters (the biases are read here)
    float out_scale;
    float gamma;
};

// Periodic index for -n <= i < 2n.  Every caller is within 3 cells of the
// grid (the 5x5 stencil) and every entry point
// requires nx, ny >= 5, so one conditional wrap replaces an integer modulo
// (whose division sequence would run per stencil cell).
__device__ __forceinline__ int wrap(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }

// Conserved states [B][4][n][n] (FP64, periodic), as the training batches hold them.
struct PackedStates {
    const double* q;
    int nx, ny;
    __device__ double get(int b, int v, int i, int j) const {
        i = wrap(i, nx);
        j = wrap(j, ny);
        return q[(((long long)b * 4 + v) * ny + j) * nx + i];
    }
};
// One context state buffer (periodic in x and y), read by interior index.
struct PaddedState {
    const double* q;
    long long plane;
    int pitch, nx, ny;
    __device__ double get(int, int v, int i, int j) const {
        i = wrap(i, nx);
        j = wrap(j, ny);
        return q[(long long)v * plane + (long long)(YO + j) * pitch + XO + i];
    }
};

// Shared-memory plans (byte offsets; every operand 128-byte aligned).  Forward:
// the hidden activations overwrite X, which the first product has read by then.
constexpr int X_BYTES = 128 * K1 * 2, H_BYTES = 128 * H * 2, ONE_BYTES = 128 * 8 * 2;
constexpr int W_BYTES = (H * K1 + H * H + N3 * H) * 2;
constexpr int FW_X = 0, FW_H1 = 0, FW_H2 = H_BYTES, FW_W = X_BYTES;
constexpr int SM_FWD = FW_W + W_BYTES;                  // 38.9 KB
// Backward: a column of ones follows H1 and H2 (and stands in X's padding), so
// that the weight gradients' products also form the bias gradients.  dZ1
// overwrites H2 once dW3 has read it.  A transposed operand of M = 128 spans 16
// core-matrix columns (32 KB): X, H1 and H2 each have that much after them,
// and what lies past their own columns only reaches accumulator rows that
// nobody reads.
constexpr int BW_X = 0, BW_H1 = BW_X + X_BYTES, BW_ONE1 = BW_H1 + H_BYTES, BW_H2 = BW_ONE1 + ONE_BYTES,
              BW_ONE2 = BW_H2 + H_BYTES, BW_DZ2 = BW_ONE2 + ONE_BYTES, BW_DY = BW_DZ2 + H_BYTES,
              BW_W = BW_DY + 128 * N3 * 2, BW_DZ1 = BW_H2;
constexpr int SM_BWD = BW_W + W_BYTES;                  // 71.7 KB
static_assert(BW_H2 + 16 * 2048 <= SM_BWD, "transposed operands stay inside the block's shared memory");
// Resident blocks per SM (shared memory and 512 tensor-memory columns: 5 x 32, 3 x 128)
constexpr int FWD_BLOCKS = 5, BWD_BLOCKS = 3;
constexpr uint32_t FWD_COLS = 32, BWD_COLS = 128;
constexpr uint32_t T_D = 0, T_DW1 = 32, T_DW2 = 64, T_DW3 = 96;  // accumulator columns (backward)

struct FaceId {
    int b, orient, i, j;
};
__device__ __forceinline__ FaceId face_of(long long f, int nx, int ny) {
    const long long per = 2LL * nx * ny;
    FaceId id;
    if (f < 0x7fffffffLL && per < 0x7fffffffLL) {  // the same quotients in 32-bit arithmetic
        const unsigned uf = (unsigned)f, up = (unsigned)per, un = (unsigned)nx * (unsigned)ny;
        id.b = (int)(uf / up);
        unsigned rem = uf - (unsigned)id.b * up;
        id.orient = (int)(rem / un);
        rem -= (unsigned)id.orient * un;
        id.j = (int)(rem / (unsigned)nx);
        id.i = (int)(rem - (unsigned)id.j * (unsigned)nx);
        return id;
    }
    id.b = (int)(f / per);
    long long rem = f - (long long)id.b * per;
    id.orient = (int)(rem / ((long long)nx * ny));
    rem -= (long long)id.orient * nx * ny;
    id.j = (int)(rem / nx);
    id.i = (int)(rem - (long long)id.j * nx);
    return id;
}

// Primitive (rho, u, v, p) of a stencil cell.
template <class SV>
__device__ __forceinline__ void prim_at(const SV& sv, int b, int i, int j, float gamma, float (&w)[4]) {
    const double r = sv.get(b, 0, i, j), mx = sv.get(b, 1, i, j), my = sv.get(b, 2, i, j), E = sv.get(b, 3, i, j);
    const double u = mx / r, v = my / r;
    const double p = (gamma - 1.0) * (E - 0.5 * r * (u * u + v * v));
    w[0] = (float)r;
    w[1] = (float)u;
    w[2] = (float)v;
    w[3] = (float)p;
}

// The network's per-cell inputs (rho - 1, u, v, p - 1) in FP32, computed once
// per cell by nn_prims_kernel; each cell feeds 50 face stencils.
struct PrimView {
    const float4* p;
    int nx, ny;
    __device__ float4 get(int b, int i, int j) const {
        i = wrap(i, nx);
        j = wrap(j, ny);
        return p[((long long)b * ny + j) * nx + i];
    }
};

// Programmatic dependent launch, as the step's other kernels (efvm_kernels.cu):
// nothing a predecessor wrote is read before the wait.
__device__ __forceinline__ void pdl_wait_then_release() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class SV>
__global__ void nn_prims_kernel(SV sv, int batch, float gamma, float4* __restrict__ out) {
    pdl_wait_then_release();
    const long long n = (long long)sv.nx * sv.ny, total = (long long)batch * n;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
        const int b = (int)(t / n);
        const long long c = t - (long long)b * n;
        const int j = (int)(c / sv.nx), i = (int)(c - (long long)j * sv.nx);
        float w[4];
        prim_at(sv, b, i, j, gamma, w);
        out[t] = make_float4(w[0] - 1.0f, w[1], w[2], w[3] - 1.0f);
    }
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// The stencil features of face `id`, written as row r of X with one 16-byte
// store per two stencil cells (8 consecutive K in the canonical layout).
// Feature 4q + v is variable v (rho - 1, normal velocity, tangential velocity,
// p - 1) of stencil cell q = (c + 2) * 5 + (a + 3), a the offset along the face
// normal (-3..1), c across.  Feature IN is `one` (a column of ones gives the
// backward pass its bias gradients; the weights of the padding are zero).
__device__ __forceinline__ void gather_face(const PrimView& pv, const FaceId& id, unsigned char* x, int r, float one) {
    // the wrapped offsets of the five cells along and across the normal
    int along[5], across[5];
    const int n_al = id.orient == 0 ? pv.nx : pv.ny, n_ac = id.orient == 0 ? pv.ny : pv.nx;
    const int s_al = id.orient == 0 ? 1 : pv.nx, s_ac = id.orient == 0 ? pv.nx : 1;
    const int p_al = id.orient == 0 ? id.i : id.j, p_ac = id.orient == 0 ? id.j : id.i;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        along[k] = wrap(p_al + k - 3, n_al) * s_al;
        across[k] = wrap(p_ac + k - 2, n_ac) * s_ac;
    }
    const float4* base = pv.p + (long long)id.b * pv.ny * pv.nx;
#pragma unroll
    for (int m = 0; m < K1 / 8; ++m) {
        float f[8];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int q = 2 * m + h;
            if (q < 25) {
                const float4 w = base[across[q / 5] + along[q % 5]];
                f[4 * h + 0] = w.x;
                f[4 * h + 1] = id.orient == 0 ? w.y : w.z;
                f[4 * h + 2] = id.orient == 0 ? w.z : w.y;
                f[4 * h + 3] = w.w;
            } else {
                f[4 * h + 0] = q == 25 ? one : 0.f;
                f[4 * h + 1] = f[4 * h + 2] = f[4 * h + 3] = 0.f;
            }
        }
        *reinterpret_cast<uint4*>(x + tc::canon_offset(r, 8 * m, 128)) =
            make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]),
                       pack_bf16x2(f[6], f[7]));
    }
}

// Weights into shared memory at w (W1, W2, W3), 16 bytes (8 consecutive K of one row) per copy.
constexpr int W2_OFF = H * K1 * 2, W3_OFF = W2_OFF + H * H * 2;
__device__ __forceinline__ void load_weights(const Net& net, unsigned char* w) {
    const uint4* w1 = reinterpret_cast<const uint4*>(net.w1);
    for (int t = threadIdx.x; t < H * K1 / 8; t += blockDim.x) {
        const int o = t / (K1 / 8), g = t - o * (K1 / 8);
        *reinterpret_cast<uint4*>(w + tc::canon_offset(o, 8 * g, H)) = w1[t];
    }
    const uint4* w2 = reinterpret_cast<const uint4*>(net.w2);
    for (int t = threadIdx.x; t < H * H / 8; t += blockDim.x) {
        const int o = t / (H / 8), g = t - o * (H / 8);
        *reinterpret_cast<uint4*>(w + W2_OFF + tc::canon_offset(o, 8 * g, H)) = w2[t];
    }
    const uint4* w3 = reinterpret_cast<const uint4*>(net.w3);
    for (int t = threadIdx.x; t < N3 * H / 8; t += blockDim.x) {
        const int o = t / (H / 8), g = t - o * (H / 8);
        *reinterpret_cast<uint4*>(w + W3_OFF + tc::canon_offset(o, 8 * g, N3)) = w3[t];
    }
}

// Tensor-core state of a block: its tensor memory, the mbarrier and its phase.
struct TC {
    uint64_t* bar;
    uint32_t tmem;
    uint32_t phase;
};

// Shared-memory operands written so far become visible to the tensor core, and
// its accumulators read so far may be overwritten.
__device__ __forceinline__ void publish() {
    tc::fence_smem_to_async();
    tc::fence_before_sync();
    __syncthreads();
}
// Wait (bounded) for the products committed last and make their accumulators
// readable; false if the wait ran out anywhere in the block.
__device__ __forceinline__ bool products_done(TC& t) {
    bool ok = tc::mbar_wait(t.bar, t.phase);
    ok = __syncthreads_and(ok);
    t.phase ^= 1u;
    if (!ok) {
        if (threadIdx.x == 0) atomicExch(&g_nn_error, 1);
        tc::mbar_wait(t.bar, t.phase ^ 1u);  // a second bounded chance to retire before TMEM is released
        return false;
    }
    tc::fence_after_sync();
    return true;
}

// D = A B^T of K-major operands (A 128 rows, B n rows), committed.
__device__ __forceinline__ bool run_gemm(TC& t, const unsigned char* a, const unsigned char* b, int n, int k) {
    publish();
    tc::gemm_issue(t.tmem, a, b, n, k, t.bar);
    return products_done(t);
}

// 32 consecutive FP32 values as a row of 32 BF16 in the canonical layout.
__device__ __forceinline__ void store_row(unsigned char* out, int r, const float (&v)[H]) {
#pragma unroll
    for (int g = 0; g < H / 8; ++g)
        *reinterpret_cast<uint4*>(out + tc::canon_offset(r, 8 * g, 128)) =
            make_uint4(pack_bf16x2(v[8 * g], v[8 * g + 1]), pack_bf16x2(v[8 * g + 2], v[8 * g + 3]),
                       pack_bf16x2(v[8 * g + 4], v[8 * g + 5]), pack_bf16x2(v[8 * g + 6], v[8 * g + 7]));
}
// Accumulator row r (32 columns).
__device__ __forceinline__ void load_row(uint32_t tmem, float (&v)[H]) {
#pragma unroll
    for (int c0 = 0; c0 < H; c0 += 16) {
        float q[16];
        tc::tmem_ld16(tmem, c0, q);
#pragma unroll
        for (int c = 0; c < 16; ++c) v[c0 + c] = q[c];
    }
}
// Row r's accumulator + bias through relu into row r of `out`; bit c of the
// result is set where unit c is active.
__device__ __forceinline__ uint32_t relu_epilogue(uint32_t tmem, const float* bias, unsigned char* out, int r) {
    float v[H];
    load_row(tmem, v);
    uint32_t on = 0;
#pragma unroll
    for (int c = 0; c < H; ++c) {
        v[c] = fmaxf(v[c] + bias[c], 0.f);
        // the activity of the value that is stored, rounded to BF16
        on |= (__bfloat162float(__float2bfloat16_rn(v[c])) > 0.f ? 1u : 0u) << c;
    }
    store_row(out, r, v);
    return on;
}

__device__ __forceinline__ void tile_setup(TC& t, uint64_t* bar, uint32_t* slot, uint32_t cols) {
    if ((threadIdx.x >> 5) == 0) tc::tmem_alloc(slot, cols);
    if (threadIdx.x == 0) tc::mbar_init(bar, 1);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    t.bar = bar;
    t.tmem = *slot;
    t.phase = 0;
}
__device__ __forceinline__ void tile_teardown(const TC& t, uint32_t cols) {
    tc::fence_before_sync();
    __syncthreads();
    if ((threadIdx.x >> 5) == 0) tc::tmem_free(t.tmem, cols);
}

// Forward: the correction of every face, grid frame, corr[((b*2+orient)*4+v)*ny*nx + j*nx + i].
// sensor > 0 (inference): a face whose two cells differ in pressure by more than
// sensor * min(p), or where rho or p is not positive, keeps the plain flux.
//
// Bound by the latency of a tile's chain (gather 25 cells, three products and
// their read-backs), so the blocks are persistent (weights and tensor memory
// set up once) and small enough for five per SM, whose tiles overlap.  One
// 87 KB block per tile, two resident, took 51 us for 262144 faces (2048 tiles);
// this form takes 23.5 us.
__global__ void __launch_bounds__(128) nn_forward_kernel(PrimView pv, Net net, int tiles, float* __restrict__ corr,
                                                         float sensor, unsigned long long* fallbacks) {
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t slot;
    __shared__ float bias[2 * H + NOUT];
    TC t;
    const int r = threadIdx.x;
    load_weights(net, sm + FW_W);
    if (r < 2 * H + NOUT) bias[r] = net.p[P_B1 + r];  // b1, b2, b3 are consecutive
    tile_setup(t, &bar, &slot, FWD_COLS);
    pdl_wait_then_release();
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const FaceId id = face_of((long long)tile * 128 + r, pv.nx, pv.ny);
        gather_face(pv, id, sm + FW_X, r, 0.f);
        if (!run_gemm(t, sm + FW_X, sm + FW_W, H, K1)) break;
        relu_epilogue(t.tmem, bias, sm + FW_H1, r);
        if (!run_gemm(t, sm + FW_H1, sm + FW_W + W2_OFF, H, H)) break;
        relu_epilogue(t.tmem, bias + H, sm + FW_H2, r);
        if (!run_gemm(t, sm + FW_H2, sm + FW_W + W3_OFF, N3, H)) break;
        float v[16];
        tc::tmem_ld16(t.tmem, 0, v);
        float y[4];
#pragma unroll
        for (int o = 0; o < 4; ++o) y[o] = (v[o] + bias[2 * H + o]) * net.out_scale;
        if (sensor > 0.f) {
            const int il = id.orient == 0 ? id.i - 1 : id.i, jl = id.orient == 0 ? id.j : id.j - 1;
            const float4 ql = pv.get(id.b, il, jl), qr = pv.get(id.b, id.i, id.j);
            const float rl = ql.x + 1.0f, rr = qr.x + 1.0f, pl = ql.w + 1.0f, pr = qr.w + 1.0f;
            const bool fire = !(rl > 0.f && rr > 0.f && pl > 0.f && pr > 0.f) ||
                              fabsf(pr - pl) > sensor * fminf(pl, pr);
            if (fire) {
                y[0] = y[1] = y[2] = y[3] = 0.f;
                atomicAdd(fallbacks, 1ull);
            }
        }
        // face frame (rho, m_n, m_t, E) -> grid frame (rho, m_x, m_y, E)
        const float g[4] = {y[0], id.orient == 0 ? y[1] : y[2], id.orient == 0 ? y[2] : y[1], y[3]};
        const long long cell = (long long)id.j * pv.nx + id.i, nn = (long long)pv.nx * pv.ny;
#pragma unroll
        for (int q = 0; q < 4; ++q) corr[((long long)(id.b * 2 + id.orient) * 4 + q) * nn + cell] = g[q];
    }
    tile_teardown(t, FWD_COLS);
}

// The residual loss of a batch: e = R + div(corr) per cell and variable,
// L = sum_v w_v mean(e_v^2).
struct Residual {
    const float* corr;    // the forward pass's corrections, grid frame
    const double* resid;  // R, [batch][4][ny][nx]
    double inv_dx, inv_dy;
    float w[4];
    double inv_cells;     // 1 / (batch ny nx)
    double* loss;
};

// dL/dcorr of one face in the grid frame, from the errors of the two cells it
// divides (+1/dx in the cell before it, -1/dx in its own), and for an x face the
// loss of its own cell, added to `l`.
__device__ __forceinline__ void face_gradient(const Residual& rs, const FaceId& id, int nx, int ny, float (&g)[4],
                                              double& l) {
    const long long n = (long long)nx * ny;
    const int i = id.i, j = id.j;
    const int im = i == 0 ? nx - 1 : i - 1, ip = i == nx - 1 ? 0 : i + 1;
    const int jm = j == 0 ? ny - 1 : j - 1, jp = j == ny - 1 ? 0 : j + 1;
    const bool x = id.orient == 0;
    // the other cell of the face, and the cells after it
    const int oi = x ? im : i, oj = x ? j : jm;
    const int oip = x ? i : ip, ojp = x ? jp : j;
    const int c = j * nx + i, o = oj * nx + oi;
    const double inv = x ? rs.inv_dx : rs.inv_dy;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        const float* cx = rs.corr + ((long long)(id.b * 2 + 0) * 4 + v) * n;  // x face on the left of a cell
        const float* cy = rs.corr + ((long long)(id.b * 2 + 1) * 4 + v) * n;  // y face below it
        const double* r = rs.resid + ((long long)id.b * 4 + v) * n;
        auto err = [&](int cell, int right, int above) {
            return r[cell] + (((double)cx[right] - (double)cx[cell]) * rs.inv_dx +
                              ((double)cy[above] - (double)cy[cell]) * rs.inv_dy);
        };
        const double e = err(c, j * nx + ip, jp * nx + i), eo = err(o, oj * nx + oip, ojp * nx + oi);
        if (x) l += rs.w[v] * e * e;
        g[v] = (float)(2.0 * rs.inv_cells * rs.w[v] * (eo - e) * inv);
    }
}

// Backward: the loss, and its gradient with respect to every parameter summed over
// the block's tiles, into partials[block][P_COUNT].  Each face forms its own dL/dcorr
// (a kernel of its own took 8 us at 131072 cells, and 4 MB out and back).
//
// Per tile four product phases form the chain: X W1^T; H1 W2^T; dZ2 W2 (beside
// dW3 += H2^T dY and dW2 += H1^T dZ2); dW1 += X^T dZ1.  The weight gradients
// are kept as their transposes, features along M, and stay in tensor memory over
// all of a block's tiles; their operands are the forward buffers read MN-major,
// so nothing is stored twice or transposed.  dH2 = dY W3 has K = 4 and runs on
// the FP32 units.  One block per tile with stored transposes (150 KB, one block
// per SM), shuffled column sums for the biases and 39 MB of per-tile partials
// took 235 us and 84 us for their sum at 262144 faces; now 43.5 and 8.9 us, the
// residual's gradient included.
__global__ void __launch_bounds__(128) nn_backward_kernel(PrimView pv, Net net, int tiles, Residual rs,
                                                          float* __restrict__ partials) {
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t slot;
    __shared__ float bias[2 * H];
    __shared__ float4 w3[H];  // column c of W3
    TC t;
    const int r = threadIdx.x;
    load_weights(net, sm + BW_W);
    if (r < 2 * H) bias[r] = net.p[P_B1 + r];
    if (r < H)
        w3[r] = make_float4(__bfloat162float(net.w3[r]), __bfloat162float(net.w3[H + r]),
                            __bfloat162float(net.w3[2 * H + r]), __bfloat162float(net.w3[3 * H + r]));
    {
        const uint4 ones = make_uint4(pack_bf16x2(1.f, 0.f), 0u, 0u, 0u);
        *reinterpret_cast<uint4*>(sm + BW_ONE1 + tc::canon_offset(r, 0, 128)) = ones;
        *reinterpret_cast<uint4*>(sm + BW_ONE2 + tc::canon_offset(r, 0, 128)) = ones;
    }
    tile_setup(t, &bar, &slot, BWD_COLS);
    pdl_wait_then_release();
    const uint32_t idesc_t = tc::idesc_bf16_f32(128, H) | tc::A_MN | tc::B_MN;
    bool ok = true, first = true;
    double l = 0.0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const FaceId id = face_of((long long)tile * 128 + r, pv.nx, pv.ny);
        // output gradient of this face in its own frame, times out_scale, as BF16
        float g[4];
        face_gradient(rs, id, pv.nx, pv.ny, g, l);
        const float dyf[4] = {g[0] * net.out_scale, (id.orient == 0 ? g[1] : g[2]) * net.out_scale,
                              (id.orient == 0 ? g[2] : g[1]) * net.out_scale, g[3] * net.out_scale};
        float dy[4];
#pragma unroll
        for (int o = 0; o < 4; ++o) dy[o] = __bfloat162float(__float2bfloat16_rn(dyf[o]));
        gather_face(pv, id, sm + BW_X, r, 1.f);
        *reinterpret_cast<uint4*>(sm + BW_DY + tc::canon_offset(r, 0, 128)) =
            make_uint4(pack_bf16x2(dy[0], dy[1]), pack_bf16x2(dy[2], dy[3]), 0u, 0u);
        *reinterpret_cast<uint4*>(sm + BW_DY + tc::canon_offset(r, 8, 128)) = make_uint4(0u, 0u, 0u, 0u);
        if (!(ok = run_gemm(t, sm + BW_X, sm + BW_W, H, K1))) break;
        const uint32_t on1 = relu_epilogue(t.tmem + T_D, bias, sm + BW_H1, r);
        if (!(ok = run_gemm(t, sm + BW_H1, sm + BW_W + W2_OFF, H, H))) break;
        const uint32_t on2 = relu_epilogue(t.tmem + T_D, bias + H, sm + BW_H2, r);
        float dz[H];
        // dZ2 = (dY W3) * relu'(h2)
#pragma unroll
        for (int c = 0; c < H; ++c) {
            const float4 w = w3[c];
            const float v = fmaf(dy[3], w.w, fmaf(dy[2], w.z, fmaf(dy[1], w.y, dy[0] * w.x)));
            dz[c] = (on2 >> c) & 1u ? v : 0.f;
        }
        store_row(sm + BW_DZ2, r, dz);
        publish();
        if (threadIdx.x == 0) {
            tc::fence_after_sync();
            // dW3^T += H2^T dY, D = dZ2 W2 (both before the commit: dZ1 overwrites H2), then dW2^T += H1^T dZ2
            tc::mma_steps(t.tmem + T_DW3, sm + BW_H2, 128, 2048, 256, sm + BW_DY, 128, 2048, 256,
                          tc::idesc_bf16_f32(128, N3) | tc::A_MN | tc::B_MN, 8, !first);
            tc::mma_steps(t.tmem + T_D, sm + BW_DZ2, 2048, 128, 4096, sm + BW_W + W2_OFF, 128, 16 * H, 256,
                          tc::idesc_bf16_f32(128, H) | tc::B_MN, H / 16, false);
            tc::mma_commit(t.bar);
            tc::mma_steps(t.tmem + T_DW2, sm + BW_H1, 128, 2048, 256, sm + BW_DZ2, 128, 2048, 256, idesc_t, 8, !first);
        }
        if (!(ok = products_done(t))) break;
        // dZ1 = D * relu'(h1)
        load_row(t.tmem + T_D, dz);
#pragma unroll
        for (int c = 0; c < H; ++c) dz[c] = (on1 >> c) & 1u ? dz[c] : 0.f;
        store_row(sm + BW_DZ1, r, dz);
        publish();
        if (threadIdx.x == 0) {
            tc::fence_after_sync();
            tc::mma_steps(t.tmem + T_DW1, sm + BW_X, 128, 2048, 256, sm + BW_DZ1, 128, 2048, 256, idesc_t, 8, !first);
            tc::mma_commit(t.bar);
        }
        first = false;
        if (!(ok = products_done(t))) break;
    }
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if ((r & 31) == 0 && l != 0.0) atomicAdd(rs.loss, l * rs.inv_cells);
    if (ok) {
        // row k of the transposed gradients is feature k; the row of ones holds the biases
        float* part = partials + (long long)blockIdx.x * P_COUNT;
        float v[H];
        load_row(t.tmem + T_DW1, v);
        if (r < K1)
#pragma unroll
            for (int o = 0; o < H; ++o) part[P_W1 + o * K1 + r] = r < IN ? v[o] : 0.f;
        if (r == IN)
#pragma unroll
            for (int o = 0; o < H; ++o) part[P_B1 + o] = v[o];
        load_row(t.tmem + T_DW2, v);
        if (r < H)
#pragma unroll
            for (int o = 0; o < H; ++o) part[P_W2 + o * H + r] = v[o];
        if (r == H)
#pragma unroll
            for (int o = 0; o < H; ++o) part[P_B2 + o] = v[o];
        float u[16];
        tc::tmem_ld16(t.tmem + T_DW3, 0, u);
        if (r < H)
#pragma unroll
            for (int o = 0; o < NOUT; ++o) part[P_W3 + o * H + r] = u[o];
        if (r == H)
#pragma unroll
            for (int o = 0; o < NOUT; ++o) part[P_B3 + o] = u[o];
    }
    tile_teardown(t, BWD_COLS);
}

// grad[p] = sum over blocks of partials[block][p], in a fixed order: a warp per
// slice of the blocks over 32 parameters, then the slices in order.  The grid's
// first thread also passes the loss on with the tensor-core status beside it,
// so that the host reads both with one copy.  (One thread per parameter over
// 2048 per-tile partials took 84 us: 19 blocks of serial loads; this takes 8.9 us
// for 444.)
constexpr int RED_SLICES = 32;
__global__ void __launch_bounds__(32 * RED_SLICES) nn_reduce_kernel(const float* __restrict__ partials, int blocks,
                                                                    float* __restrict__ grad,
                                                                    float* __restrict__ grad_out, double* loss) {
    __shared__ float sum[RED_SLICES][32];
    pdl_wait_then_release();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int p = blockIdx.x * 32 + lane;
    float s = 0.f;
    if (p < P_COUNT)
#pragma unroll 8
        for (int b = w; b < blocks; b += RED_SLICES) s += partials[(long long)b * P_COUNT + p];
    sum[w][lane] = s;
    __syncthreads();
    if (w == 0 && p < P_COUNT) {
        for (int k = 1; k < RED_SLICES; ++k) s += sum[k][lane];
        grad[p] = s;
        if (grad_out) grad_out[p] = s;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) loss[1] = (double)g_nn_error;
}

// Adam on the FP32 parameters, then the BF16 copies the tensor cores read.
__global__ void nn_adam_kernel(float* __restrict__ p, float* __restrict__ m, float* __restrict__ v,
                               const float* __restrict__ g, float lr, float b1t, float b2t,
                               __nv_bfloat16* w1, __nv_bfloat16* w2, __nv_bfloat16* w3) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= P_COUNT) return;
    const bool pad = q < P_W2 && (q - P_W1) % K1 >= IN;  // W1 columns beyond the 100 inputs stay zero
    if (!pad) {
        const float gq = g[q];
        const float mq = 0.9f * m[q] + 0.1f * gq;
        const float vq = 0.999f * v[q] + 0.001f * gq * gq;
        m[q] = mq;
        v[q] = vq;
        const float mh = mq / (1.f - b1t), vh = vq / (1.f - b2t);
        p[q] -= lr * mh / (sqrtf(vh) + 1e-8f);
    }
    if (q < P_W2) w1[q - P_W1] = __float2bfloat16_rn(pad ? 0.f : p[q]);
    else if (q < P_W3) w2[q - P_W2] = __float2bfloat16_rn(p[q]);
    else if (q < P_B1) w3[q - P_W3] = __float2bfloat16_rn(p[q]);  // rows 0..NOUT-1 of [N3][H]
}

}  // namespace nn
}  // namespace
}  // namespace efvm

using namespace efvm;

// ---- the network object ------------------------------------------------------
struct efvm_nn {
    float *p = nullptr, *m = nullptr, *v = nullptr, *grad = nullptr;
    __nv_bfloat16 *w1 = nullptr, *w2 = nullptr, *w3 = nullptr;
    float out_scale = 1e-3f, gamma = 1.4f;
    int64_t steps = 0;
    float* partials = nullptr;
    size_t partials_cap = 0;
    float* corr = nullptr;
    size_t corr_cap = 0;
    float4* prims = nullptr;
    size_t prims_cap = 0;
    double* loss_d = nullptr;
    std::string err;
};

namespace efvm {
nn::Net nn_net(const efvm_nn* h) {
    nn::Net n;
    n.w1 = h->w1;
    n.w2 = h->w2;
    n.w3 = h->w3;
    n.p = h->p;
    n.out_scale = h->out_scale;
    n.gamma = h->gamma;
    return n;
}

template <typename... KArgs, typename... Args>
static void launch_nn(void (*kernel)(KArgs...), unsigned grid, unsigned block, size_t smem, cudaStream_t s, bool pdl,
                      Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, args...);
}

// One persistent block per resident slot, at most one per tile.
static int nn_blocks(int tiles, int per_sm) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return std::min(tiles, per_sm * sms);
}

static void launch_forward(const nn::PrimView& pv, const efvm_nn* h, int tiles, float* corr, float sensor,
                           unsigned long long* fallbacks, bool pdl, cudaStream_t s) {
    launch_nn(nn::nn_forward_kernel, (unsigned)nn_blocks(tiles, nn::FWD_BLOCKS), 128u, (size_t)nn::SM_FWD, s, pdl, pv,
              nn_net(h), tiles, corr, sensor, fallbacks);
}

// Both launches belong to a captured step: programmatic, like its other kernels
// (the weights do not change while a step runs).
int nn_prims_padded(const efvm_nn* h, const double* q, long long plane, int pitch, int nx, int ny, float4* prims,
                    void* stream) {
    nn::PaddedState sv{q, plane, pitch, nx, ny};
    launch_nn(nn::nn_prims_kernel<nn::PaddedState>, (unsigned)((nx * ny + 255) / 256), 256u, (size_t)0,
              (cudaStream_t)stream, true, sv, 1, h->gamma, prims);
    return 1;
}

int nn_forward_prims(const efvm_nn* h, int nx, int ny, float* corr, float4* prims, float sensor,
                     unsigned long long* fallbacks, void* stream) {
    launch_forward(nn::PrimView{prims, nx, ny}, h, (int)(2LL * nx * ny / 128), corr, sensor, fallbacks, true,
                   (cudaStream_t)stream);
    return 1;
}

int nn_forward_padded(const efvm_nn* h, const double* q, long long plane, int pitch, int nx, int ny, float* corr,
                      float4* prims, float sensor, unsigned long long* fallbacks, void* stream) {
    return nn_prims_padded(h, q, plane, pitch, nx, ny, prims, stream) +
           nn_forward_prims(h, nx, ny, corr, prims, sensor, fallbacks, stream);
}

float nn_gamma(const efvm_nn* h) { return h->gamma; }

int nn_prepare_launches() {
    cudaError_t e = cudaFuncSetAttribute(nn::nn_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, nn::SM_FWD);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(nn::nn_backward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, nn::SM_BWD);
    return e == cudaSuccess ? EFVM_OK : EFVM_ERR_CUDA;
}
}  // namespace efvm

namespace {

int nfail(efvm_nn* h, int code, const std::string& msg) {
    if (h) h->err = msg;
    set_global_error(msg);
    return code;
}

#define NN_TRY(h, call)                                                                                     \
    do {                                                                                                    \
        cudaError_t e_ = (call);                                                                            \
        if (e_ != cudaSuccess) return nfail(h, EFVM_ERR_CUDA, std::string(#call ": ") + cudaGetErrorString(e_)); \
    } while (0)

// splitmix64 and a Box-Muller normal, for the seeded initial weights
uint64_t splitmix(uint64_t& s) {
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
double normal(uint64_t& s) {
    const double u1 = ((splitmix(s) >> 11) + 0.5) * (1.0 / 9007199254740992.0);
    const double u2 = ((splitmix(s) >> 11) + 0.5) * (1.0 / 9007199254740992.0);
    return std::sqrt(-2.0 * std::log(u1)) * std::cos(6.283185307179586 * u2);
}

// Upload FP32 parameters and refresh the BF16 copies (an Adam step with lr = 0
// and a zero gradient leaves p unchanged and rewrites the copies).
int upload_params(efvm_nn* h, const float* host, cudaStream_t s) {
    NN_TRY(h, cudaMemcpyAsync(h->p, host, nn::P_COUNT * sizeof(float), cudaMemcpyHostToDevice, s));
    NN_TRY(h, cudaMemsetAsync(h->grad, 0, nn::P_COUNT * sizeof(float), s));
    nn::nn_adam_kernel<<<(nn::P_COUNT + 255) / 256, 256, 0, s>>>(h->p, h->m, h->v, h->grad, 0.f, 0.5f, 0.5f, h->w1,
                                                                 h->w2, h->w3);
    NN_TRY(h, cudaGetLastError());
    NN_TRY(h, cudaStreamSynchronize(s));
    return EFVM_OK;
}

int check_shape(efvm_nn* h, int batch, int nx, int ny) {
    if (batch < 1 || nx < 5 || ny < 5 || ((long long)nx * ny) % 64)
        return nfail(h, EFVM_ERR_INVALID_ARG, "the network needs batch >= 1, nx, ny >= 5 and nx*ny a multiple of 64");
    return EFVM_OK;
}

int ensure_buffers(efvm_nn* h, int batch, int nx, int ny) {
    const size_t faces = 2ull * batch * nx * ny;
    const size_t blocks = (size_t)nn_blocks((int)(faces / 128), nn::BWD_BLOCKS);
    if (blocks * nn::P_COUNT > h->partials_cap) {
        cudaFree(h->partials);
        h->partials = nullptr;
        h->partials_cap = 0;
        NN_TRY(h, cudaMalloc(&h->partials, blocks * nn::P_COUNT * sizeof(float)));
        h->partials_cap = blocks * nn::P_COUNT;
    }
    if ((size_t)batch * nx * ny > h->prims_cap) {
        cudaFree(h->prims);
        h->prims = nullptr;
        h->prims_cap = 0;
        NN_TRY(h, cudaMalloc(&h->prims, (size_t)batch * nx * ny * sizeof(float4)));
        h->prims_cap = (size_t)batch * nx * ny;
    }
    if (faces * 4 > h->corr_cap) {
        cudaFree(h->corr);
        h->corr = nullptr;
        h->corr_cap = 0;
        NN_TRY(h, cudaMalloc(&h->corr, faces * 4 * sizeof(float)));
        h->corr_cap = faces * 4;
    }
    return EFVM_OK;
}

int tc_status(efvm_nn* h) {
    int err = 0;
    NN_TRY(h, cudaMemcpyFromSymbol(&err, g_nn_error, sizeof(int)));
    if (err) {
        const int zero = 0;
        cudaMemcpyToSymbol(g_nn_error, &zero, sizeof(int));
        return nfail(h, EFVM_ERR_TIMEOUT, "a tensor-core completion wait ran out");
    }
    return EFVM_OK;
}

}  // namespace

extern "C" {

int efvm_nn_param_count(void) { return nn::P_COUNT; }

int efvm_nn_create(float out_scale, float gamma, uint64_t seed, efvm_nn** out) {
    if (!out || !(out_scale > 0.f) || !(gamma > 1.f)) return nfail(nullptr, EFVM_ERR_INVALID_ARG, "efvm_nn_create: invalid argument");
    *out = nullptr;
    efvm_nn* h = new efvm_nn();
    h->out_scale = out_scale;
    h->gamma = gamma;
    auto bad = [&](int code) {
        efvm_nn_destroy(h);
        return code;
    };
    const size_t pb = nn::P_COUNT * sizeof(float);
    if (cudaMalloc(&h->p, pb) || cudaMalloc(&h->m, pb) || cudaMalloc(&h->v, pb) || cudaMalloc(&h->grad, pb) ||
        cudaMalloc(&h->w1, nn::H * nn::K1 * 2) || cudaMalloc(&h->w2, nn::H * nn::H * 2) ||
        cudaMalloc(&h->w3, nn::N3 * nn::H * 2) || cudaMalloc(&h->loss_d, 2 * sizeof(double)))
        return bad(nfail(nullptr, EFVM_ERR_OOM, "efvm_nn_create: cudaMalloc"));
    cudaMemset(h->m, 0, pb);
    cudaMemset(h->v, 0, pb);
    cudaMemset(h->w3, 0, nn::N3 * nn::H * 2);  // rows >= NOUT stay zero
    if (nn_prepare_launches()) return bad(nfail(nullptr, EFVM_ERR_CUDA, "efvm_nn_create: kernel attributes"));
    // He-normal hidden layers, a small output layer (the initial correction is near zero), zero biases
    std::vector<float> p(nn::P_COUNT, 0.f);
    uint64_t s = seed;
    for (int o = 0; o < nn::H; ++o)
        for (int k = 0; k < nn::IN; ++k) p[nn::P_W1 + o * nn::K1 + k] = (float)(normal(s) * std::sqrt(2.0 / nn::IN));
    for (int q = 0; q < nn::H * nn::H; ++q) p[nn::P_W2 + q] = (float)(normal(s) * std::sqrt(2.0 / nn::H));
    for (int q = 0; q < nn::NOUT * nn::H; ++q) p[nn::P_W3 + q] = (float)(normal(s) * 0.01);
    const int rc = upload_params(h, p.data(), 0);
    if (rc) return bad(rc);
    *out = h;
    return EFVM_OK;
}

int efvm_nn_destroy(efvm_nn* h) {
    if (!h) return EFVM_OK;
    cudaFree(h->p);
    cudaFree(h->m);
    cudaFree(h->v);
    cudaFree(h->grad);
    cudaFree(h->w1);
    cudaFree(h->w2);
    cudaFree(h->w3);
    cudaFree(h->partials);
    cudaFree(h->corr);
    cudaFree(h->prims);
    cudaFree(h->loss_d);
    delete h;
    return EFVM_OK;
}

int efvm_nn_get_params(efvm_nn* h, float* host) {
    if (!h || !host) return nfail(h, EFVM_ERR_INVALID_ARG, "null argument");
    NN_TRY(h, cudaMemcpy(host, h->p, nn::P_COUNT * sizeof(float), cudaMemcpyDeviceToHost));
    return EFVM_OK;
}

int efvm_nn_set_params(efvm_nn* h, const float* host) {
    if (!h || !host) return nfail(h, EFVM_ERR_INVALID_ARG, "null argument");
    return upload_params(h, host, 0);
}

int efvm_nn_get_scale(efvm_nn* h, float* out_scale) {
    if (!h || !out_scale) return nfail(h, EFVM_ERR_INVALID_ARG, "null argument");
    *out_scale = h->out_scale;
    return EFVM_OK;
}

int efvm_nn_forward(efvm_nn* h, const double* states, int32_t batch, int32_t nx, int32_t ny, float* corr,
                    void* stream) {
    if (!h || !states || !corr) return nfail(h, EFVM_ERR_INVALID_ARG, "null argument");
    int rc = check_shape(h, batch, nx, ny);
    if (rc) return rc;
    rc = ensure_buffers(h, batch, nx, ny);
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    nn::PackedStates sv{states, nx, ny};
    const long long cells = (long long)batch * nx * ny;
    nn::nn_prims_kernel<nn::PackedStates><<<(unsigned)((cells + 255) / 256), 256, 0, s>>>(sv, batch, h->gamma, h->prims);
    const int tiles = (int)(2LL * batch * nx * ny / 128);
    launch_forward(nn::PrimView{h->prims, nx, ny}, h, tiles, corr, 0.f, nullptr, false, s);
    NN_TRY(h, cudaGetLastError());
    NN_TRY(h, cudaStreamSynchronize(s));
    return tc_status(h);
}

int efvm_nn_loss_grad(efvm_nn* h, const double* states, const double* resid, int32_t batch, int32_t nx, int32_t ny,
                      double dx, double dy, const float w[4], float* grad_out, double* loss, void* stream) {
    if (!h || !states || !resid || !w) return nfail(h, EFVM_ERR_INVALID_ARG, "null argument");
    int rc = check_shape(h, batch, nx, ny);
    if (rc) return rc;
    rc = ensure_buffers(h, batch, nx, ny);
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    nn::PackedStates sv{states, nx, ny};
    const long long cells = (long long)batch * nx * ny;
    const int tiles = (int)(2 * cells / 128);
    NN_TRY(h, cudaMemsetAsync(h->loss_d, 0, sizeof(double), s));
    nn::nn_prims_kernel<nn::PackedStates><<<(unsigned)((cells + 255) / 256), 256, 0, s>>>(sv, batch, h->gamma, h->prims);
    const nn::PrimView pv{h->prims, nx, ny};
    // The chain is launched programmatically: each kernel sets up (weights, tensor
    // memory) while its predecessor drains.
    launch_forward(pv, h, tiles, h->corr, 0.f, nullptr, true, s);
    const int blocks = nn_blocks(tiles, nn::BWD_BLOCKS);
    const nn::Residual rs{h->corr, resid, 1.0 / dx, 1.0 / dy, {w[0], w[1], w[2], w[3]}, 1.0 / (double)cells, h->loss_d};
    launch_nn(nn::nn_backward_kernel, (unsigned)blocks, 128u, (size_t)nn::SM_BWD, s, true, pv, nn_net(h), tiles, rs,
              h->partials);
    launch_nn(nn::nn_reduce_kernel, (unsigned)((nn::P_COUNT + 31) / 32), 32u * nn::RED_SLICES, (size_t)0, s, true,
              (const float*)h->partials, blocks, h->grad, grad_out, h->loss_d);
    NN_TRY(h, cudaGetLastError());
    double out[2] = {0.0, 0.0};  // the loss and the tensor-core status
    NN_TRY(h, cudaMemcpyAsync(out, h->loss_d, sizeof(out), cudaMemcpyDeviceToHost, s));
    NN_TRY(h, cudaStreamSynchronize(s));
    if (loss) *loss = out[0];
    return out[1] != 0.0 ? tc_status(h) : EFVM_OK;
}

int efvm_nn_adam(efvm_nn* h, float lr, void* stream) {
    if (!h) return nfail(h, EFVM_ERR_INVALID_ARG, "null argument");
    cudaStream_t s = (cudaStream_t)stream;
    h->steps += 1;
    const float b1t = (float)std::pow(0.9, (double)h->steps), b2t = (float)std::pow(0.999, (double)h->steps);
    nn::nn_adam_kernel<<<(nn::P_COUNT + 255) / 256, 256, 0, s>>>(h->p, h->m, h->v, h->grad, lr, b1t, b2t, h->w1, h->w2,
                                                                 h->w3);
    NN_TRY(h, cudaGetLastError());
    return EFVM_OK;
}

}  // extern "C"


extern "C" int efvm_nn_gemm_bf16(const uint16_t* a, const uint16_t* b, float* d, int32_t m, int32_t n, int32_t k,
                                 void* stream) {
    if (!a || !b || !d) {
        set_global_error("efvm_nn_gemm_bf16: null argument");
        return EFVM_ERR_INVALID_ARG;
    }
    if (m <= 0 || m % 128 || n < 16 || n > 256 || n % 16 || k < 16 || k > 256 || k % 16) {
        set_global_error("efvm_nn_gemm_bf16: need m a multiple of 128, n and k multiples of 16 in [16, 256]");
        return EFVM_ERR_INVALID_ARG;
    }
    cudaStream_t s = (cudaStream_t)stream;
    const int zero = 0;
    cudaError_t e = cudaMemcpyToSymbolAsync(g_nn_error, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, s);
    // The operands need (128 + n) * k * 2 bytes; the launch takes 200 KB so that
    // every descriptor stride stays inside the CTA's shared memory whatever the
    // operand shape.
    const size_t smem = 200 * 1024;
    if (e == cudaSuccess) e = cudaFuncSetAttribute(nn_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) {
        set_global_error(std::string("efvm_nn_gemm_bf16: ") + cudaGetErrorString(e));
        return EFVM_ERR_CUDA;
    }
    nn_gemm_kernel<<<m / 128, 128, smem, s>>>(reinterpret_cast<const __nv_bfloat16*>(a),
                                              reinterpret_cast<const __nv_bfloat16*>(b), d, n, k);
    int err = 0;
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyFromSymbolAsync(&err, g_nn_error, sizeof(int), 0, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        set_global_error(std::string("efvm_nn_gemm_bf16: ") + cudaGetErrorString(e));
        return EFVM_ERR_CUDA;
    }
    if (err) {
        set_global_error("efvm_nn_gemm_bf16: a tensor-core completion wait ran out");
        return EFVM_ERR_TIMEOUT;
    }
    return EFVM_OK;
}
