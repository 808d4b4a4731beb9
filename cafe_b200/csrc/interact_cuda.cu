// interact_cuda.cu -- the dot interaction of DLRM (dlrm_s_pytorch.py:779-812, `interact_features`, "dot") as one
// kernel per direction.  The reference concatenates the dense vector and the F pooled embedding vectors of a sample
// into T [(F+1), D], forms Z = T T^t with a batched matrix product, picks the entries below the diagonal (or on and
// below it with arch_interaction_itself) through two index lists and concatenates them behind the dense vector:
// four launches, a [B, F+1, F+1] intermediate and a gather per direction.  Here a block takes one sample: the F+1
// vectors are staged in shared memory once, every thread computes a few of the dot products and writes them to their
// place in the output row; the backward forms the symmetric weight matrix of the sample from the incoming gradient
// and multiplies it back onto the staged vectors.  27 x 27 x 128 multiply-adds per sample: no tensor cores needed.
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/cafe_b200.h"
#include "cafe_internal.h"

#define CAFE_INTERACT_MAX_VECS 64   // F + 1
#define CAFE_INTERACT_THREADS 128
#define CAFE_SMS 148

// pair number p of (i, j), j < i + off (off = 1: the diagonal counts), in the reference's order: i ascending, j ascending
__device__ __forceinline__ int cafe_pair_index(int i, int j, int off) { return i * (i - 1 + 2 * off) / 2 + j; }

// x [B, D] (dense vector; may be null: no dense vector, F vectors only), emb: vector f of sample b at
// emb + b * sample_stride + f * field_stride, out [B, out_stride] = { x (if given) | pairs }
__global__ void __launch_bounds__(CAFE_INTERACT_THREADS)
k_interact_forward(const float* __restrict__ x, const float* __restrict__ emb, int64_t field_stride, int64_t sample_stride, int F,
                   int D, int off, float* __restrict__ out, int64_t out_stride) {
    extern __shared__ float sh[];
    const int nv = F + (x ? 1 : 0);
    const int ld = D + 1;   // row pitch: two rows never start in the same bank
    float* T = sh;
    const int64_t b = blockIdx.x;
    for (int e = threadIdx.x; e < nv * D; e += blockDim.x) {
        const int v = e / D, d = e - v * D;
        float val;
        if (x && v == 0) val = x[b * D + d];
        else val = emb[b * sample_stride + (int64_t)(v - (x ? 1 : 0)) * field_stride + d];
        T[v * ld + d] = val;
    }
    __syncthreads();
    float* o = out + b * out_stride;
    const int lead = x ? D : 0;
    for (int d = threadIdx.x; d < lead; d += blockDim.x) o[d] = T[d];
    const int npairs = cafe_pair_index(nv, 0, off);
    for (int p = threadIdx.x; p < npairs; p += blockDim.x) {
        // (i, j) of pair p: the largest i whose first pair number is <= p
        int i = off ? 0 : 1;
        while (cafe_pair_index(i + 1, 0, off) <= p) ++i;
        const int j = p - cafe_pair_index(i, 0, off);
        const float* a = T + i * ld;
        const float* c = T + j * ld;
        float s = 0.f;
        for (int d = 0; d < D; ++d) s += a[d] * c[d];
        o[lead + p] = s;
    }
}

// grad_out [B, out_stride] -> grad_x [B, D] (if x was given), grad_emb (same addressing as emb)
__global__ void __launch_bounds__(CAFE_INTERACT_THREADS)
k_interact_backward(const float* __restrict__ x, const float* __restrict__ emb, int64_t field_stride, int64_t sample_stride, int F,
                    int D, int off, const float* __restrict__ grad_out, int64_t out_stride, float* __restrict__ grad_x,
                    float* __restrict__ grad_emb, int64_t gfield_stride, int64_t gsample_stride) {
    extern __shared__ float sh[];
    const int nv = F + (x ? 1 : 0);
    const int ld = D + 1;
    float* T = sh;                       // [nv][ld]
    float* G = sh + nv * ld;             // [nv][nv]: d(loss)/d(T_i . T_j), symmetric; the diagonal doubled
    const int64_t b = blockIdx.x;
    for (int e = threadIdx.x; e < nv * D; e += blockDim.x) {
        const int v = e / D, d = e - v * D;
        float val;
        if (x && v == 0) val = x[b * D + d];
        else val = emb[b * sample_stride + (int64_t)(v - (x ? 1 : 0)) * field_stride + d];
        T[v * ld + d] = val;
    }
    const float* g = grad_out + b * out_stride;
    const int lead = x ? D : 0;
    for (int e = threadIdx.x; e < nv * nv; e += blockDim.x) {
        const int i = e / nv, j = e - i * nv;
        float w = 0.f;
        if (j < i) w = g[lead + cafe_pair_index(i, j, off)];
        else if (j > i) w = g[lead + cafe_pair_index(j, i, off)];
        else if (off) w = 2.0f * g[lead + cafe_pair_index(i, i, off)];
        G[e] = w;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nv * D; e += blockDim.x) {
        const int i = e / D, d = e - i * D;
        float s = 0.f;
        for (int j = 0; j < nv; ++j) s += G[i * nv + j] * T[j * ld + d];
        if (x && i == 0) grad_x[b * D + d] = s + g[d];
        else grad_emb[b * gsample_stride + (int64_t)(i - (x ? 1 : 0)) * gfield_stride + d] = s;
    }
}

// ---- vectors of 16-byte pieces --------------------------------------------------------------------------------------
// Rows of a multiple of four floats on 16-byte boundaries (every embedding dimension in use) take these kernels; the two
// above remain for all other dimensions and addresses.  Those read one float per load and per multiply-add from shared
// memory and are bound by that.
//
// What the path has to move per sample is its vectors (27 x 128: 13.8 KB in, and out again in the backward), so the work
// between must hide behind that.  A block walks over groups of samples: while it works on one group, the next one's
// vectors are on their way into the other half of the stage (cp.async, 16 bytes each), so every SM has tens of KB in
// flight whatever its warps do.
#define CAFE_IT_EDGE 7          // vectors per tile edge: 27 vectors (26 fields and the dense one) are four blocks with one row spare
#define CAFE_IT_THREADS 256     // most threads of a block

__device__ __forceinline__ void cafe_cp16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cafe_cp4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cafe_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cafe_cp_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

struct CafeInteract {
    const float *x, *emb;
    int64_t field_stride, sample_stride;
    int B, F, D, off, nv, npairs, width;   // width: floats of an output row
    int per_group, lane_shift;             // samples per group; log2 of the lanes that share a vector (>= D / 4)
    int blocks_of_rows;                    // ceil(nv / CAFE_IT_EDGE)
};

// the vectors of samples [b0, b0 + ns), one every `pitch` floats
template <int DD>
__device__ __forceinline__ void cafe_interact_stage(const CafeInteract& P, int64_t b0, int ns, float* T, const int pitch) {
    const int D = DD ? DD : P.D;
    const int q = (threadIdx.x & ((1 << P.lane_shift) - 1)) * 4, step = blockDim.x >> P.lane_shift;
    if (q >= D) return;
    const int lead = P.x ? 1 : 0;
    int s = 0, v = threadIdx.x >> P.lane_shift;
    for (int r = v; r < ns * P.nv; r += step, v += step) {
        while (v >= P.nv) { v -= P.nv; ++s; }
        const int64_t b = b0 + s;
        const float* src = v < lead ? P.x + b * D : P.emb + b * P.sample_stride + (int64_t)(v - lead) * P.field_stride;
        cafe_cp16(T + r * pitch + q, src + q);
    }
}

// Forward.  The pairs of a sample are tiles of 7 x 7 vectors on and below the diagonal.  KL neighbouring lanes share a
// tile and take every KL-th 16-byte piece of its vectors, four pieces each: 14 loads from shared memory feed 196
// multiply-adds.  The lanes' partial sums are added in a halving exchange that leaves 8 / KL rows of the tile with every lane;
// the kernel is bound by instruction issue (67 % of the slots, the multiply-adds 30 % of the pipe), and with fewer pieces per
// lane the exchange is as long as the sums.  65 536 samples of 27 vectors: D 64 254 us (525 a sample per block, a float per load;
// 285 with eight lanes a tile), D 32 149 (339; 199), D 16 98 (250; 127); 29 000 of D 128 193 us (419) = 2.4 TB/s.  Double
// multiply-adds (f32x2) halve the instructions but take 166 registers and were no faster at D 64, slower at D 128.
// The vectors lie at a pitch that puts the pieces which the tiles of a load phase (eight lanes) read, 7 vectors apart, into
// different banks.
template <int DD, int KL> __host__ __device__ constexpr int cafe_interact_pitch(int D) { return KL == 1 ? D + 4 : KL == 2 ? D + 8 : KL == 4 ? D + 16 : D; }
template <int DD, int KL>
__global__ void __launch_bounds__(CAFE_IT_THREADS, 2) k_interact_forward_tiled(const CafeInteract P, float* __restrict__ out, int64_t out_stride) {
    extern __shared__ __align__(16) float sh[];
    constexpr int E = CAFE_IT_EDGE, N = 8 * E;
    const int D = DD ? DD : P.D, pitch = cafe_interact_pitch<DD, KL>(D);
    const int group = P.per_group * P.nv * pitch;
    float* Z = sh + 2 * group + (E - 1) * pitch;   // (tiles read up to E - 1 vectors past the last one)
    const int tiles = P.blocks_of_rows * (P.blocks_of_rows + 1) / 2;
    const int slots = blockDim.x / KL, slot = threadIdx.x / KL, kl = threadIdx.x % KL;
    const int lead = P.x ? D : 0;
    const int64_t step = (int64_t)gridDim.x * P.per_group;
    int64_t b0 = (int64_t)blockIdx.x * P.per_group;
    cafe_interact_stage<DD>(P, b0, (int)min((int64_t)P.per_group, P.B - b0), sh, pitch);
    cafe_cp_commit();
    for (int half = 0; b0 < P.B; b0 += step, half ^= 1) {
        const int ns = (int)min((int64_t)P.per_group, P.B - b0);
        const float* T = sh + half * group;
        cafe_cp_wait();
        __syncthreads();   // this group has arrived; everyone is done with the other half and with Z
        if (b0 + step < P.B) cafe_interact_stage<DD>(P, b0 + step, (int)min((int64_t)P.per_group, P.B - b0 - step), sh + (half ^ 1) * group, pitch);
        cafe_cp_commit();
        for (int t0 = 0; t0 < ns * tiles; t0 += slots) {
            const int t = min(t0 + slot, ns * tiles - 1);   // (spare lanes repeat the last tile and write nothing)
            const int s = t / tiles, tile = t - s * tiles;
            int bi = 0;
            while ((bi + 1) * (bi + 2) / 2 <= tile) ++bi;
            const int bj = tile - bi * (bi + 1) / 2;
            const float* A = T + (s * P.nv + bi * E) * pitch;
            const float* C = T + (s * P.nv + bj * E) * pitch;
            float acc[N];
#pragma unroll
            for (int i = 0; i < N; ++i) acc[i] = 0.f;
#pragma unroll 1
            for (int q = kl * 4; q < D; q += KL * 4) {
                float4 a[E];
#pragma unroll
                for (int r = 0; r < E; ++r) a[r] = *reinterpret_cast<const float4*>(A + r * pitch + q);
#pragma unroll
                for (int c = 0; c < E; ++c) {
                    const float4 w = *reinterpret_cast<const float4*>(C + c * pitch + q);
#pragma unroll
                    for (int r = 0; r < E; ++r) {
                        float v = acc[r * E + c];
                        v += a[r].x * w.x; v += a[r].y * w.y; v += a[r].z * w.z; v += a[r].w * w.w;
                        acc[r * E + c] = v;
                    }
                }
            }
#pragma unroll
            for (int m = KL / 2, n = N / 2; m > 0; m >>= 1, n >>= 1) {
                const bool up = (kl & m) != 0;
#pragma unroll
                for (int i = 0; i < N / 2; ++i) {
                    if (i < n) {
                        const float send = up ? acc[i] : acc[i + n], keep = up ? acc[i + n] : acc[i];
                        acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
                    }
                }
            }
            constexpr int RL = 8 / KL;   // rows left with this lane
            if (t0 + slot < ns * tiles) {
#pragma unroll
                for (int h = 0; h < RL; ++h) {
                    const int r = kl * RL + h, i = bi * E + r;
                    if (r < E && i < P.nv) {
                        float* z = Z + s * P.npairs + cafe_pair_index(i, 0, P.off) + bj * E;
                        const int n = i + P.off - bj * E;   // columns of the row that count
#pragma unroll
                        for (int c = 0; c < E; ++c) if (c < n) z[c] = acc[h * E + c];
                    }
                }
            }
        }
        __syncthreads();
        for (int s = 0; s < ns; ++s) {
            float* o = out + (b0 + s) * out_stride;
            for (int e = threadIdx.x; e < P.width; e += blockDim.x) o[e] = e < lead ? T[s * P.nv * pitch + e] : Z[s * P.npairs + e - lead];
        }
    }
}

// Backward.  The incoming row of a sample is spread into its symmetric weight matrix, rows padded to eight columns per
// block of seven; a thread makes one 16-byte piece of seven gradient vectors, so that one piece of a vector (its lanes
// read consecutive pieces) and two broadcast pieces of weights feed 28 multiply-adds.  Vectors are added in ascending order.
// Bound by instruction issue too (75 %).  65 536 samples of 27 vectors: D 64 280 us (1052 with one output per thread and turn),
// D 32 176 (591), D 16 141 (371); 29 000 of D 128 227 us (893) = 3.8 TB/s.
template <int DD>
__global__ void __launch_bounds__(CAFE_IT_THREADS, 2) k_interact_backward_tiled(const CafeInteract P, const float* __restrict__ grad_out,
                                                                             int64_t out_stride, float* __restrict__ grad_x,
                                                                             float* __restrict__ grad_emb, int64_t gfield_stride,
                                                                             int64_t gsample_stride) {
    extern __shared__ __align__(16) float sh[];
    constexpr int E = CAFE_IT_EDGE;
    const int D = DD ? DD : P.D;
    const int pitch = P.blocks_of_rows * 8 + 4;
    const int group = P.per_group * P.nv * D;
    const int gsize = P.per_group * P.nv * pitch;
    float* G = sh + 2 * group;
    uint32_t* place = reinterpret_cast<uint32_t*>(G + gsize);   // per pair: its two places in the matrix
    float* raw = reinterpret_cast<float*>(place + P.npairs);    // incoming rows, two halves
    const int rows = P.per_group * P.width;
    const int lead = P.x ? D : 0;
    const int64_t step = (int64_t)gridDim.x * P.per_group;
    int64_t b0 = (int64_t)blockIdx.x * P.per_group;
    auto fetch = [&](int64_t b, int half) {
        const int ns = (int)min((int64_t)P.per_group, P.B - b);
        cafe_interact_stage<DD>(P, b, ns, sh + half * group, D);
        for (int s = 0; s < ns; ++s)
            for (int e = threadIdx.x; e < P.width; e += blockDim.x)
                cafe_cp4(raw + half * rows + s * P.width + e, grad_out + (b + s) * out_stride + e);
    };
    fetch(b0, 0);
    cafe_cp_commit();
    for (int e = threadIdx.x; e < gsize; e += blockDim.x) G[e] = 0.f;
    for (int e = threadIdx.x; e < P.nv * P.nv; e += blockDim.x) {
        const int i = e / P.nv, j = e - i * P.nv;
        if (j < i + P.off) {
            const int ri = i / E, rj = j / E;
            place[cafe_pair_index(i, j, P.off)] = (uint32_t)(i * pitch + rj * 8 + j - rj * E) | (uint32_t)(j * pitch + ri * 8 + i - ri * E) << 16;
        }
    }
    const int q = (threadIdx.x & ((1 << P.lane_shift) - 1)) * 4;
    const int units = blockDim.x >> P.lane_shift;
    for (int half = 0; b0 < P.B; b0 += step, half ^= 1) {
        const int ns = (int)min((int64_t)P.per_group, P.B - b0);
        const float* T = sh + half * group;
        const float* in = raw + half * rows;
        cafe_cp_wait();
        __syncthreads();   // this group has arrived; everyone is done with the other half and with G
        if (b0 + step < P.B) fetch(b0 + step, half ^ 1);
        cafe_cp_commit();
        for (int s = 0; s < ns; ++s)
            for (int p = threadIdx.x; p < P.npairs; p += blockDim.x) {
                const uint32_t at = place[p], a = at & 0xffffu, c = at >> 16;
                const float w = in[s * P.width + lead + p];
                float* g = G + s * P.nv * pitch;
                if (a == c) g[a] = 2.0f * w;
                else { g[a] = w; g[c] = w; }
            }
        __syncthreads();
        for (int u = threadIdx.x >> P.lane_shift; u < ns * P.blocks_of_rows; u += units) {
            if (q >= D) break;
            const int s = u / P.blocks_of_rows, rb = u - s * P.blocks_of_rows;
            const float* t = T + s * P.nv * D + q;
            const float* g = G + s * P.nv * pitch + rb * 8;
            float4 acc[E];
#pragma unroll
            for (int r = 0; r < E; ++r) acc[r] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 3
            for (int j = 0; j < P.nv; ++j) {
                const float4 v = *reinterpret_cast<const float4*>(t + j * D);
                const float4 g0 = *reinterpret_cast<const float4*>(g + j * pitch), g1 = *reinterpret_cast<const float4*>(g + j * pitch + 4);
                const float w[E] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z};
#pragma unroll
                for (int r = 0; r < E; ++r) { acc[r].x += w[r] * v.x; acc[r].y += w[r] * v.y; acc[r].z += w[r] * v.z; acc[r].w += w[r] * v.w; }
            }
            const int64_t b = b0 + s;
#pragma unroll
            for (int r = 0; r < E; ++r) {
                const int i = rb * E + r;
                if (i >= P.nv) break;
                if (lead && i == 0) {
                    const float* d = in + s * P.width + q;
                    *reinterpret_cast<float4*>(grad_x + b * D + q) = make_float4(acc[r].x + d[0], acc[r].y + d[1], acc[r].z + d[2], acc[r].w + d[3]);
                } else {
                    __stcs(reinterpret_cast<float4*>(grad_emb + b * gsample_stride + (int64_t)(i - (lead ? 1 : 0)) * gfield_stride + q), acc[r]);
                }
            }
        }
    }
}

static bool interact_pieces_ok(const void* p, int64_t fs, int64_t ss) { return ((uintptr_t)p & 15) == 0 && fs % 4 == 0 && ss % 4 == 0; }

static void interact_plan(CafeInteract* P, const float* x, const float* emb, int64_t fs, int64_t ss, int B, int F, int D, int itself) {
    P->x = x; P->emb = emb; P->field_stride = fs; P->sample_stride = ss; P->B = B; P->F = F; P->D = D; P->off = itself;
    P->nv = F + (x ? 1 : 0);
    P->npairs = P->nv * (P->nv - 1 + 2 * itself) / 2;
    P->width = (x ? D : 0) + P->npairs;
    P->blocks_of_rows = (P->nv + CAFE_IT_EDGE - 1) / CAFE_IT_EDGE;
    P->lane_shift = 0;
    while ((4 << P->lane_shift) < D) ++P->lane_shift;
}
// Threads and samples per group for `lanes` threads of work and `bytes` of shared memory per sample: about `want` threads a
// block, but no more samples than leave every SM `resident` blocks to work on, and room for them.
static int interact_group(CafeInteract* P, int lanes, size_t bytes, int want, int resident) {
    int s = want / lanes;
    const int room = (int)(224 * 1024 / resident / bytes);
    if (s > room) s = room;
    const int fair = (P->B + CAFE_SMS * resident - 1) / (CAFE_SMS * resident);
    s = s < 1 ? 1 : (s > fair ? fair : s);
    P->per_group = s;
    const int threads = (s * lanes + 31) & ~31;
    return threads > CAFE_IT_THREADS ? CAFE_IT_THREADS : threads;
}
// as many blocks as are resident at once: `sm_threads` threads of these kernels' registers and 227 KB of shared memory an SM
template <typename K>
static cudaError_t interact_grid(K kernel, const CafeInteract& P, int threads, int sm_threads, size_t smem, unsigned* grid) {
    if (smem > 48 * 1024) {
        // (the limit belongs to the kernel, not to the launch, and threads share it: always the same value, the largest a block
        // can have, or one thread's smaller call would lower it between another's setting and its launch)
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e != cudaSuccess) return e;
    }
    const int by_threads = sm_threads / threads, by_memory = (int)((227 * 1024) / (smem + 1024));
    const int64_t resident = by_threads < by_memory ? by_threads : by_memory;
    const int64_t groups = ((int64_t)P.B + P.per_group - 1) / P.per_group, most = CAFE_SMS * (resident > 0 ? resident : 1);
    *grid = (unsigned)(groups < most ? groups : most);
    return cudaSuccess;
}
#define INTERACT_DISPATCH(D, ...)                                   \
    switch (D) {                                                    \
        case 16: { constexpr int DD = 16; __VA_ARGS__; } break;     \
        case 32: { constexpr int DD = 32; __VA_ARGS__; } break;     \
        case 64: { constexpr int DD = 64; __VA_ARGS__; } break;     \
        case 128: { constexpr int DD = 128; __VA_ARGS__; } break;   \
        default: { constexpr int DD = 0; __VA_ARGS__; } break;      \
    }

extern "C" {

static int interact_args_ok(const float* emb, int B, int F, int D, int itself, int64_t fs, int64_t ss) {
    if (B < 0 || F < 1 || F + 1 > CAFE_INTERACT_MAX_VECS || D < 1 || D > CAFE_MAX_DIM || (itself != 0 && itself != 1)) return 0;
    if (B > 0 && (!emb || fs < D || ss < D)) return 0;
    return 1;
}

int cafe_dot_interaction_forward(const float* x_dev, const float* emb_dev, int64_t field_stride, int64_t sample_stride, int B,
                                 int F, int D, int itself, float* out_dev, int64_t out_stride, void* stream) {
    if (!interact_args_ok(emb_dev, B, F, D, itself, field_stride, sample_stride)) return CAFE_ERR_ARG;
    const int nv = F + (x_dev ? 1 : 0);
    const int npairs = nv * (nv - 1 + 2 * itself) / 2;
    if (B == 0) return CAFE_OK;
    if (!out_dev || out_stride < (x_dev ? D : 0) + npairs) return CAFE_ERR_ARG;
    const size_t smem = sizeof(float) * (size_t)nv * (D + 1);
    if (smem > 48 * 1024) return CAFE_ERR_UNSUPPORTED;
    if (D % 4 == 0 && interact_pieces_ok(emb_dev, field_stride, sample_stride) && interact_pieces_ok(x_dev, 0, 0)) {
        CafeInteract P;
        interact_plan(&P, x_dev, emb_dev, field_stride, sample_stride, B, F, D, itself);
        const int tiles = P.blocks_of_rows * (P.blocks_of_rows + 1) / 2;
        cudaError_t e = cudaSuccess;
        INTERACT_DISPATCH(D, {
            constexpr int KL = DD == 16 ? 1 : DD == 32 ? 2 : DD == 64 ? 4 : 8;
            const int pitch = cafe_interact_pitch<DD, KL>(D);
            const int threads = interact_group(&P, tiles * KL, sizeof(float) * (2 * (size_t)nv * pitch + npairs), KL == 8 ? 240 : 128, 3);
            const size_t sm = sizeof(float) * ((size_t)(2 * P.per_group * nv + CAFE_IT_EDGE - 1) * pitch + (size_t)P.per_group * npairs);
            unsigned grid = 1;
            e = interact_grid(k_interact_forward_tiled<DD, KL>, P, threads, 512, sm, &grid);
            if (e == cudaSuccess) k_interact_forward_tiled<DD, KL><<<grid, threads, sm, (cudaStream_t)stream>>>(P, out_dev, out_stride);
        });
        if (e == cudaSuccess) e = cudaGetLastError();
        if (e != cudaSuccess) { cafe_internal_set_error(cudaGetErrorString(e)); return CAFE_ERR_CUDA; }
        return CAFE_OK;
    }
    k_interact_forward<<<B, CAFE_INTERACT_THREADS, smem, (cudaStream_t)stream>>>(x_dev, emb_dev, field_stride, sample_stride, F, D,
                                                                                itself, out_dev, out_stride);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { cafe_internal_set_error(cudaGetErrorString(e)); return CAFE_ERR_CUDA; }
    return CAFE_OK;
}

int cafe_dot_interaction_backward(const float* x_dev, const float* emb_dev, int64_t field_stride, int64_t sample_stride, int B,
                                  int F, int D, int itself, const float* grad_out_dev, int64_t out_stride, float* grad_x_dev,
                                  float* grad_emb_dev, int64_t gfield_stride, int64_t gsample_stride, void* stream) {
    if (!interact_args_ok(emb_dev, B, F, D, itself, field_stride, sample_stride)) return CAFE_ERR_ARG;
    if (B == 0) return CAFE_OK;
    if (!grad_out_dev || !grad_emb_dev || (x_dev && !grad_x_dev) || gfield_stride < D || gsample_stride < D) return CAFE_ERR_ARG;
    const int nv = F + (x_dev ? 1 : 0);
    const size_t smem = sizeof(float) * ((size_t)nv * (D + 1) + (size_t)nv * nv);
    if (smem > 48 * 1024) return CAFE_ERR_UNSUPPORTED;
    if (D % 4 == 0 && interact_pieces_ok(emb_dev, field_stride, sample_stride) && interact_pieces_ok(x_dev, 0, 0) &&
        interact_pieces_ok(grad_emb_dev, gfield_stride, gsample_stride) && interact_pieces_ok(grad_x_dev, 0, 0)) {
        CafeInteract P;
        interact_plan(&P, x_dev, emb_dev, field_stride, sample_stride, B, F, D, itself);
        const int threads = interact_group(&P, P.blocks_of_rows << P.lane_shift,
                                           sizeof(float) * (size_t)(2 * (nv * D + P.width) + nv * (P.blocks_of_rows * 8 + 4)), 128, 4);
        const size_t sm = sizeof(float) * ((size_t)P.per_group * (2 * (nv * D + P.width) + nv * (P.blocks_of_rows * 8 + 4)) + P.npairs);
        unsigned grid = 1;
        cudaError_t e = cudaSuccess;
        INTERACT_DISPATCH(D, {
            e = interact_grid(k_interact_backward_tiled<DD>, P, threads, 640, sm, &grid);
            if (e == cudaSuccess)
                k_interact_backward_tiled<DD><<<grid, threads, sm, (cudaStream_t)stream>>>(P, grad_out_dev, out_stride, grad_x_dev,
                                                                                          grad_emb_dev, gfield_stride, gsample_stride);
        });
        if (e == cudaSuccess) e = cudaGetLastError();
        if (e != cudaSuccess) { cafe_internal_set_error(cudaGetErrorString(e)); return CAFE_ERR_CUDA; }
        return CAFE_OK;
    }
    k_interact_backward<<<B, CAFE_INTERACT_THREADS, smem, (cudaStream_t)stream>>>(x_dev, emb_dev, field_stride, sample_stride, F, D,
                                                                                 itself, grad_out_dev, out_stride, grad_x_dev,
                                                                                 grad_emb_dev, gfield_stride, gsample_stride);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { cafe_internal_set_error(cudaGetErrorString(e)); return CAFE_ERR_CUDA; }
    return CAFE_OK;
}

}  // extern "C"
