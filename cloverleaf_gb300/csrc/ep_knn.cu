// ep_knn.cu -- node embeddings from feature embeddings and exact cosine
// top-k on the GPU (the evaluation side of the path).
//
//   ep_embed_features  NodeEmbedder.embed_feature_set (src/lib.rs:2092-2124)
//                      with AvgAggregator / WeightedAggregator
//                      (src/algos/aggregator.rs:17-120): warp per node.
//   ep_align           NeighborhoodAligner.align (src/algos/alignment.rs,
//                      src/lib.rs:3040-3110): warp per node, hubs by slices.
//   ep_knn_cosine      NodeEmbeddings.nearest_neighbor for many queries at
//                      once (src/embeddings.rs:149-173, cosine distance):
//                      rows normalised to BF16, then a tcgen05 GEMM (FP32
//                      accumulation in tensor memory) fused with a per-query
//                      top-k that never leaves registers.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/ep_gb300.h"
#include "ep_device.cuh"
#include "ep_hostmem.h"

namespace ep {
namespace {

thread_local std::string g_knn_err;
thread_local float g_knn_ms = 0.f;     // CUDA-event time of the last top-k or alignment kernel

int knn_fail(int code, const char* msg) {
    g_knn_err = msg;
    return code;
}
int knn_cuda_fail(cudaError_t e, const char* what) {
    cudaGetLastError();
    g_knn_err = std::string(what) + ": " + cudaGetErrorString(e);
    return e == cudaErrorMemoryAllocation ? EP_ERR_OOM : EP_ERR_CUDA;
}

#define KCK(call, what)                                 \
    do {                                                \
        cudaError_t e_ = (call);                        \
        if (e_ != cudaSuccess) return knn_cuda_fail(e_, what); \
    } while (0)

struct DevMem {
    void* p = nullptr;
    ~DevMem() { if (p) cudaFree(p); }
    cudaError_t alloc(size_t n) { return cudaMalloc(&p, n ? n : 16); }
};

// One device allocation cut into 256-byte-aligned pieces: a call allocates
// and frees once (each cudaMalloc / cudaFree pair of some MB costs 50-200 us).
struct Arena {
    DevMem mem;
    size_t used = 0;
    size_t reserve(size_t n) { const size_t at = used; used += (n + 255) & ~(size_t)255; return at; }
    template <typename X> X* at(size_t o) const { return reinterpret_cast<X*>(static_cast<char*>(mem.p) + o); }
};

// Counts whether any id is out of range.
__global__ void __launch_bounds__(256) k_check_ids(const uint32_t* __restrict__ ids, uint64_t n, uint64_t bound,
                                                   uint32_t* __restrict__ bad) {
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
    bool out = false;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) out = out || ids[i] >= bound;
    if (out) *bad = 1u;
}

// Copies the ids to the device and reports whether all are below bound; the
// kernels that follow index with the copy.  Few ids are checked by the host,
// in less time than the answer takes to come back (35 us).
constexpr uint64_t HOST_IDS = 1u << 17;
cudaError_t upload_ids(uint32_t* dst, const uint32_t* src, uint64_t n, uint64_t bound, uint32_t* d_bad, cudaStream_t s,
                       bool* ok) {
    *ok = true;
    if (!n) return cudaSuccess;
    if (n <= HOST_IDS) {
        *ok = all_below(src, n, bound);
        return *ok ? cudaMemcpyAsync(dst, src, n * 4, cudaMemcpyHostToDevice, s) : cudaSuccess;
    }
    cudaError_t e = cudaMemsetAsync(d_bad, 0, 4, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(dst, src, n * 4, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return e;
    k_check_ids<<<(unsigned)std::min<uint64_t>((n + 255) / 256, 152 * 8), 256, 0, s>>>(dst, n, bound, d_bad);
    uint32_t bad = 0;
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(&bad, d_bad, 4, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    *ok = !bad;
    return e;
}

cudaError_t upload(void* dst, const void* src, size_t bytes, cudaStream_t s) {
    return bytes ? cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s) : cudaSuccess;
}

// Bytes of a result array whose pages the host may touch: none of memory that
// is the device's (the copy to it fails, as it should).
size_t host_bytes(const void* out, size_t bytes) {
    cudaPointerAttributes pa{};
    const bool dev = cudaPointerGetAttributes(&pa, out) == cudaSuccess && pa.type == cudaMemoryTypeDevice;
    cudaGetLastError();
    return dev ? 0 : bytes;
}

// A result into the caller's array, each slab once its pages are resident.
cudaError_t download(char* out, const void* d_out, size_t bytes, ResultPages& pages, cudaStream_t s) {
    cudaError_t e = cudaSuccess;
    for (size_t at = 0; at < bytes && e == cudaSuccess; at += ResultPages::SLAB) {
        pages.wait(at / ResultPages::SLAB);
        e = cudaMemcpyAsync(out + at, static_cast<const char*>(d_out) + at, std::min(bytes - at, ResultPages::SLAB),
                            cudaMemcpyDeviceToHost, s);
    }
    return e == cudaSuccess ? cudaStreamSynchronize(s) : e;
}

// ---------------------------------------------------------------------------
// Weighted sums of rows, one warp per node (k_rows):
//   ROWS_MEAN / ROWS_WEIGHTED (node embeddings): out[v] = sum_f w_f E[f] /
//     sum_f w_f over v's features in CSR order, f32 as the reference (w_f * e
//     rounded, then added; the weights summed in f32); nodes without features
//     get zeros.
//   ROWS_ALIGN (NeighborhoodAligner.align, src/algos/alignment.rs:25-75):
//     out[v] = (1 - a) * sum_j p_j E[u_j] + a * E[v] over the first
//     min(deg, kmax) edges in CSR order, p_j the edge probability recovered
//     from the CDF weights (w_0, w_j - w_{j-1}), a = alpha, or min(1, 1 /
//     ln(deg + 1)) when alpha < 0; every product rounded, then added, per
//     element in edge order.
// A lane owns NV groups of 4 consecutive elements (V4; dims a multiple of 4
// and a 16-byte-aligned result) or NV elements 32 apart.  Ids and
// coefficients come 32 at a time across the lanes; U rows are in flight.
// Bound by the row reads from L2 (ROWS_ALIGN, 200,000 nodes, 4M edges x 128:
// 2 GB).
// The longest rows, whose sums are one long chain, are left to the first
// HUB_CTAS CTAs of the grid: a CTA per hub and slice of 32 elements, whose
// warps load and weigh HUB_TILE rows at a time into shared memory while one
// warp adds up the tile before, in edge order.  (4.1 ms before, all of it the
// 10,000-edge hub's chain with one row in flight.)
// ---------------------------------------------------------------------------
enum RowsMode : int { ROWS_MEAN = 0, ROWS_WEIGHTED = 1, ROWS_ALIGN = 2 };
constexpr unsigned HUB_CTAS = 152;
constexpr uint32_t HUB_TILE = 128;

// Which rows are hubs.  The warps of all rows run at once, each as long as its
// row; the HUB_CTAS CTAs share all hubs' slices.  So the hubs are the rows
// above the smallest length T = HUB_ROWS x 2^b at which the hubs' slices
// together are in proportion to T:
//   edges(rows above T) x slices <= T x share,
// with a share four times as large above 128 elements, where a warp has half
// the rows in flight and each is twice as long.  A graph whose rows are all
// long has no hubs.  Kernel time in us with every row above 256 a hub / by
// this rule / without hubs: 4,000 nodes of 1,000 edges x 128 1,300 / 210 /
// 211; 20,000 of 400 x 128 3,300 / 287 / 289; 300 of 3,000 x 128 245 / 259 /
// 256; one of 10,000 among 100,000 133 / 138 / 978; 200,000 nodes of a power
// law with a 6,000-edge hub x 128 618 / 544 / 1,089 and x 256 1,102 / 1,042 /
// 2,823, with a 44,000-edge hub x 128 843 / 649 / 6,628.
constexpr uint32_t HUB_ROWS = 256;
constexpr int HUB_CLASSES = 25;              // the last: more than 2^32 edges
__host__ __device__ constexpr uint64_t hub_share(uint32_t d) { return d <= 128 ? 4640u : 4u * 4640u; }

struct Hubs {
    unsigned long long edges[HUB_CLASSES];   // class b: edges of the rows of (HUB_ROWS << b, HUB_ROWS << (b + 1)]
    unsigned long long above;                // T
    uint32_t n;                              // hubs
};

struct RowsParams {
    uint64_t n;                  // nodes
    const uint64_t* ptr;         // CSR offsets
    const uint32_t* ids;         // feature ids / neighbours
    const float* w;              // feature weights / CDF weights
    uint32_t d;
    const float* table;
    float alpha;
    uint64_t kmax;
    uint32_t* hubs;              // nodes of the hubs
    Hubs* hub;
    float* out;
};

__device__ __forceinline__ float align_keep(const RowsParams& p, uint64_t deg) {
    return p.alpha >= 0.f ? p.alpha : fminf(__fdiv_rn(1.f, logf(__fadd_rn((float)deg, 1.f))), 1.f);
}

__device__ __forceinline__ float edge_p(const RowsParams& p, uint64_t b, uint64_t j) {
    return j ? __fsub_rn(p.w[b + j], p.w[b + j - 1]) : p.w[b];
}

__device__ void hub_rows(const RowsParams& p) {
    __shared__ float tile[2][HUB_TILE][32];
    constexpr uint32_t PW = HUB_TILE / 8;                // rows of a tile per warp
    const int lane = threadIdx.x & 31;
    const uint32_t w = threadIdx.x >> 5;
    const uint32_t slices = (p.d + 31) / 32;
    const uint64_t n = (uint64_t)p.hub->n * slices;
    for (uint64_t it = blockIdx.x; it < n; it += HUB_CTAS) {
        const uint64_t v = p.hubs[it / slices];
        const uint32_t k = (uint32_t)(it % slices) * 32u + lane;
        const uint32_t kl = k < p.d ? k : p.d - 1;       // lanes past the row read its last element
        const uint64_t b = p.ptr[v], deg = p.ptr[v + 1] - b;
        const uint64_t m = deg < p.kmax ? deg : p.kmax;
        float x[PW], pj = 0.f;
        // this warp's rows of the tile at edge t0, into registers
        auto load = [&](uint64_t t0) {
            const uint64_t j = t0 + w * PW + lane;
            uint32_t id = 0;
            pj = 0.f;
            if ((uint32_t)lane < PW && j < m) {
                id = p.ids[b + j];
                pj = edge_p(p, b, j);
            }
#pragma unroll
            for (uint32_t t = 0; t < PW; ++t) {
                const uint32_t u = __shfl_sync(FULL, id, (int)t);
                if (t0 + w * PW + t < m) x[t] = p.table[(uint64_t)u * p.d + kl];
            }
        };
        auto store = [&](uint64_t t0, uint32_t buf) {
#pragma unroll
            for (uint32_t t = 0; t < PW; ++t) {
                const float q = __shfl_sync(FULL, pj, (int)t);
                if (t0 + w * PW + t < m) tile[buf][w * PW + t][lane] = __fmul_rn(q, x[t]);
            }
        };
        float acc = 0.f;
        uint32_t buf = 0;
        load(0);
        store(0, 0);
        __syncthreads();
        for (uint64_t t0 = 0; t0 < m; t0 += HUB_TILE, buf ^= 1u) {
            const bool more = t0 + HUB_TILE < m;
            if (more) load(t0 + HUB_TILE);               // in flight while the tile is summed
            if (w == 0) {
                const uint32_t cnt = (uint32_t)min((uint64_t)HUB_TILE, m - t0);
                if (cnt == HUB_TILE) {
#pragma unroll 16
                    for (uint32_t t = 0; t < HUB_TILE; ++t) acc = __fadd_rn(acc, tile[buf][t][lane]);
                } else {
                    for (uint32_t t = 0; t < cnt; ++t) acc = __fadd_rn(acc, tile[buf][t][lane]);
                }
            }
            if (more) store(t0 + HUB_TILE, buf ^ 1u);
            __syncthreads();
        }
        const float a = align_keep(p, deg), c = __fsub_rn(1.f, a);
        if (w == 0 && k < p.d) p.out[v * p.d + k] = __fadd_rn(__fmul_rn(acc, c), __fmul_rn(p.table[v * p.d + k], a));
    }
}

template <int NV, bool V4, int MODE>
__global__ void __launch_bounds__(256) k_rows(const RowsParams p) {
    unsigned block = blockIdx.x;
    if constexpr (MODE == ROWS_ALIGN) {
        if (block < HUB_CTAS) {
            hub_rows(p);
            return;
        }
        block -= HUB_CTAS;
    }
    constexpr int E = V4 ? 4 : 1;
    constexpr int U = NV * E >= 16 ? 2 : (NV * E >= 8 ? 4 : 8);     // rows in flight
    const int lane = threadIdx.x & 31;
    const uint64_t v = ((uint64_t)block * blockDim.x + threadIdx.x) >> 5;
    if (v >= p.n) return;
    const uint32_t d = p.d;
    const uint64_t b = p.ptr[v], deg = p.ptr[v + 1] - b;
    const uint64_t m = MODE == ROWS_ALIGN && p.kmax < deg ? p.kmax : deg;
    if (MODE == ROWS_ALIGN && m > p.hub->above) return;
    float acc[NV][E];
#pragma unroll
    for (int i = 0; i < NV; ++i)
#pragma unroll
        for (int e = 0; e < E; ++e) acc[i][e] = 0.f;
    uint32_t at[NV];
    bool on[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        at[i] = (uint32_t)(lane + 32 * i) * E;
        on[i] = at[i] < d;
        if (!on[i]) at[i] = 0;         // read, and not stored
    }
    auto load = [&](uint64_t row, float (&x)[NV][E]) {
        const float* r = p.table + row * d;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            if constexpr (V4) {
                const float4 q = *reinterpret_cast<const float4*>(r + at[i]);
                x[i][0] = q.x; x[i][1] = q.y; x[i][2] = q.z; x[i][3] = q.w;
            } else {
                x[i][0] = r[at[i]];
            }
        }
    };
    float wsum = 0.f;
    for (uint64_t j0 = 0; j0 < m; j0 += 32) {
        const uint32_t cnt = (uint32_t)min((uint64_t)32, m - j0);
        uint32_t id = 0;
        float cf = 1.f;
        if ((uint32_t)lane < cnt) {
            id = p.ids[b + j0 + lane];
            if (MODE == ROWS_WEIGHTED) cf = p.w[id];
            if (MODE == ROWS_ALIGN) cf = edge_p(p, b, j0 + lane);
        }
        for (uint32_t t0 = 0; t0 < cnt; t0 += U) {
            float x[U][NV][E];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint32_t row = __shfl_sync(FULL, id, (int)(t0 + u) & 31);
                if (t0 + u < cnt) load(row, x[u]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const float c = __shfl_sync(FULL, cf, (int)(t0 + u) & 31);
                if (t0 + u < cnt) {
                    if (MODE != ROWS_ALIGN) wsum += c;
#pragma unroll
                    for (int i = 0; i < NV; ++i)
#pragma unroll
                        for (int e = 0; e < E; ++e)
                            acc[i][e] = __fadd_rn(acc[i][e], MODE == ROWS_MEAN ? x[u][i][e] : __fmul_rn(c, x[u][i][e]));
                }
            }
        }
    }
    float own[NV][E];
    float a = 0.f, c = 0.f;
    if constexpr (MODE == ROWS_ALIGN) {
        a = align_keep(p, deg);
        c = __fsub_rn(1.f, a);
        load(v, own);
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        float o[E];
#pragma unroll
        for (int e = 0; e < E; ++e) {
            if constexpr (MODE == ROWS_ALIGN) o[e] = __fadd_rn(__fmul_rn(acc[i][e], c), __fmul_rn(own[i][e], a));
            else o[e] = m ? acc[i][e] / wsum : 0.f;
        }
        if (on[i]) {
            float* to = p.out + v * d + at[i];
            if constexpr (V4) *reinterpret_cast<float4*>(to) = make_float4(o[0], o[1], o[2], o[3]);
            else *to = o[0];
        }
    }
}

// The edges of each class of long rows (Hubs::edges, zeroed before).
__global__ void __launch_bounds__(256) k_hub_edges(const RowsParams p) {
    __shared__ unsigned long long sum[HUB_CLASSES];
    __shared__ uint32_t any;
    if (threadIdx.x == 0) any = 0;
    if (threadIdx.x < HUB_CLASSES) sum[threadIdx.x] = 0;
    __syncthreads();
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < p.n; v += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t m = min(p.ptr[v + 1] - p.ptr[v], p.kmax);
        if (m <= HUB_ROWS) continue;
        const int b = 63 - __clzll((long long)((m - 1) / HUB_ROWS));
        atomicAdd(&sum[min(b, HUB_CLASSES - 1)], (unsigned long long)m);
        any = 1;
    }
    __syncthreads();
    if (any && threadIdx.x < HUB_CLASSES && sum[threadIdx.x]) atomicAdd(&p.hub->edges[threadIdx.x], sum[threadIdx.x]);
}

// The hubs, in any order, and the length they exceed.
__global__ void __launch_bounds__(256) k_find_hubs(const RowsParams p) {
    __shared__ uint64_t above;
    if (threadIdx.x == 0) {
        const uint64_t slices = (p.d + 31) / 32;
        uint64_t left = 0;                   // edges of the rows above T
        for (int b = 0; b < HUB_CLASSES; ++b) left += p.hub->edges[b];
        uint64_t t = HUB_ROWS;
        for (int b = 0; b < HUB_CLASSES && left * slices > hub_share(p.d) * t; ++b, t *= 2) left -= p.hub->edges[b];
        above = left ? t : ~0ull;
        if (blockIdx.x == 0) p.hub->above = above;
    }
    __syncthreads();
    if (above == ~0ull) return;
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < p.n; v += (uint64_t)gridDim.x * blockDim.x)
        if (min(p.ptr[v + 1] - p.ptr[v], p.kmax) > above) p.hubs[atomicAdd(&p.hub->n, 1u)] = (uint32_t)v;
}

template <int MODE>
cudaError_t launch_rows(const RowsParams& p, cudaStream_t s) {
    const unsigned blocks = (unsigned)((p.n + 7) / 8) + (MODE == ROWS_ALIGN ? HUB_CTAS : 0u);
    const uint32_t d = p.d;
    if (d % 4 == 0) {            // rows of 16-byte multiples (table and result are arena pieces)
        if (d <= 128) k_rows<1, true, MODE><<<blocks, 256, 0, s>>>(p);
        else if (d <= 256) k_rows<2, true, MODE><<<blocks, 256, 0, s>>>(p);
        else k_rows<4, true, MODE><<<blocks, 256, 0, s>>>(p);
    } else {
        if (d <= 32) k_rows<1, false, MODE><<<blocks, 256, 0, s>>>(p);
        else if (d <= 64) k_rows<2, false, MODE><<<blocks, 256, 0, s>>>(p);
        else if (d <= 128) k_rows<4, false, MODE><<<blocks, 256, 0, s>>>(p);
        else if (d <= 256) k_rows<8, false, MODE><<<blocks, 256, 0, s>>>(p);
        else k_rows<16, false, MODE><<<blocks, 256, 0, s>>>(p);
    }
    return cudaGetLastError();
}

// Rows scaled to unit L2 norm (zero rows stay zero), rounded to BF16 and
// written straight into the tile image the tensor core reads (see below):
// tiles of 2^tlog rows; per tile, per 64-element K block, 8-row atoms of
// 1024 B in which the 16-byte chunk c of row r sits at chunk c ^ (r % 8).
// Rows from n up to the tile boundary are written as zeros.
__device__ __forceinline__ uint64_t swz_offset(uint64_t row, uint32_t k, uint32_t nkb, uint32_t tlog) {
    const uint64_t tile = row >> tlog;
    const uint32_t r = (uint32_t)row & ((1u << tlog) - 1u), kb = k >> 6, c = (k & 63u) >> 3, e = k & 7u;
    const uint64_t kb_bytes = (uint64_t)128u << tlog;
    return tile * nkb * kb_bytes + kb * kb_bytes + (r >> 3) * 1024u + (r & 7u) * 128u + ((c ^ (r & 7u)) << 4) + e * 2u;
}

// Rows r0 up to n_tiled (x starts at row r0), a warp per row; a row's values
// are loaded once, all of them in flight (dims <= 256: up to 8 per lane).
__global__ void __launch_bounds__(256) k_norm_swz(uint64_t r0, uint64_t n, uint64_t n_tiled, uint32_t d, uint32_t dpad,
                                                  uint32_t tlog, const float* __restrict__ x,
                                                  unsigned char* __restrict__ y) {
    const int lane = threadIdx.x & 31;
    const uint64_t r = r0 + (((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (r >= n_tiled) return;
    const bool in = r < n;
    float t[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t k = (uint32_t)(lane + 32 * i);
        t[i] = in && k < d ? x[(r - r0) * d + k] : 0.f;
    }
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i)
        if ((uint32_t)(lane + 32 * i) < d) ss += t[i] * t[i];
    ss = warp_sum<float>(ss);
    const float inv = ss > 0.f ? 1.f / sqrtf(ss) : 0.f;
    const uint32_t nkb = dpad / 64;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t k = (uint32_t)(lane + 32 * i);
        if (k < dpad) {
            const float v = (in && k < d) ? t[i] * inv : 0.f;
            *reinterpret_cast<__nv_bfloat16*>(y + swz_offset(r, k, nkb, tlog)) = __float2bfloat16_rn(v);
        }
    }
}

// ---------------------------------------------------------------------------
// Cosine top-k: one CTA per 128 queries, warp-specialised.
//
// Copy warp: copies the query tile (M = 128 rows, all of K) once, then
// streams the database through KNN_STAGES shared-memory stages, one stage
// per 64-element K block of a 256-row tile, with cp.async.bulk from the tile
// images (completion counted in bytes on mbarriers).  A stage is refilled
// once the MMAs that read it have completed.
// MMA warp: per database tile, once its accumulator is free, lane 0 issues
// 4 MMAs per K block (M = 128, N = 256, K = 16; BF16 x BF16 -> FP32) into one
// of two 256-column accumulators in tensor memory, frees each stage through
// a commit, and signals the finished tile through another.  Both loops run
// warp-uniform; the MMA descriptors are built once and advanced by adds.
// Epilogue warps: warp w reads TMEM lane quarter w % 4 (lane = query row)
// and the column slice w / 4 of each tile, 32 columns per load, then
// releases the accumulator.  Each thread keeps a sorted top-KMAX of its
// columns in registers and admits a value only above its k-th best so far,
// skipping blocks of 16 or 32 values whose maximum cannot enter; the slices'
// lists are merged per query at the end.  Operands sit in shared memory as K-major,
// 128-byte-swizzled tiles.
// The database may be split (blockIdx.y, tiles_per tiles each, from tile t0
// on): every split's slice lists go to `part` and k_merge_topk joins them.
// All waits are bounded; a timeout sets an abort flag that ends every role's
// loop, the copies and MMAs still in flight are waited for, and the error
// word is set.
// ---------------------------------------------------------------------------
constexpr int KNN_BM = 128, KNN_BN = 256, KNN_STAGES = 4, KNN_ACC = 2;
constexpr uint32_t KNN_A_KB = KNN_BM * 128u, KNN_B_KB = KNN_BN * 128u;   // bytes per 64-element K block
constexpr uint32_t KNN_TMEM_COLS = KNN_BN * KNN_ACC;                     // 512: all of tensor memory
constexpr uint32_t KNN_WAIT_LIMIT = 1u << 22;    // mbarrier polls (32 ns sleeps) before giving up
enum : uint32_t { KNN_ERR_TIMEOUT = 1u };

// This warp's TMEM lane quarter, columns taddr .. taddr + N - 1 (one 32-bit
// value per column) into r, and the largest of the thread's N values in mx:
// the reducing TMEM load of sm_103a, so that a block's skip test costs no
// instructions.  The caller waits for the load.
__device__ __forceinline__ void tmem_ld_max(uint32_t taddr, uint32_t (&r)[32], float& mx) {
    asm volatile(
        "tcgen05.ld.red.sync.aligned.32x32b.x32.max.f32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, %32, [%33];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]),
          "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]),
          "=r"(r[30]), "=r"(r[31]), "=f"(mx)
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_max(uint32_t taddr, uint32_t (&r)[16], float& mx) {
    asm volatile(
        "tcgen05.ld.red.sync.aligned.32x32b.x16.max.f32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
        "%16, [%17];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=f"(mx)
        : "r"(taddr)
        : "memory");
}

// Epilogue shape per list length, within the register file: 16 warps (4
// column slices of 64, loaded 16 columns at a time) for KMAX <= 16; 8 warps
// (2 slices of 128, 32 at a time) for KMAX 32.
template <int KMAX>
struct KnnRoles {
    static constexpr int EPI = KMAX <= 16 ? 16 : 8;
    static constexpr int BW = KMAX <= 16 ? 16 : 32;    // columns per TMEM load and per skip test
    static constexpr int SLICES = EPI / 4, CW = KNN_BN / SLICES, BLOCKS = CW / BW;
    static constexpr int COPY = EPI, MMA = EPI + 1, THREADS = 32 * (EPI + 2);
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// K-major, 128-byte swizzle, version 1; SBO = 1024 B between 8-row atoms.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3fffu);          // start address
    d |= (uint64_t)1u << 16;                           // leading byte offset (unused when swizzled)
    d |= (uint64_t)(1024u >> 4) << 32;                 // stride byte offset
    d |= (uint64_t)1u << 46;                           // descriptor version
    d |= (uint64_t)2u << 61;                           // 128-byte swizzle
    return d;
}

// kind::f16 instruction descriptor: BF16 A and B (K-major), FP32 D, M x N.
__host__ __device__ constexpr uint32_t umma_idesc(uint32_t M, uint32_t N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((N >> 3) << 17) | ((M >> 4) << 24);
}

__device__ __forceinline__ void mbar_init(uint64_t* m, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(m)), "r"(count) : "memory");
}

// Polls the mbarrier for the completion of the phase with the given parity:
// at most KNN_WAIT_LIMIT polls, 32 ns apart, and none once *abort is set.
// Returns 1 when the phase completed.
__device__ __forceinline__ uint32_t mbar_wait(uint64_t* mbar, uint32_t parity, volatile uint32_t* abort) {
    uint32_t done = 0;
    for (uint32_t it = 0; it < KNN_WAIT_LIMIT; ++it) {
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
            : "=r"(done)
            : "r"(smem_u32(mbar)), "r"(parity)
            : "memory");
        if (done || *abort) break;
        __nanosleep(32);
    }
    return done;
}

__device__ __forceinline__ void mbar_arrive(uint64_t* mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(mbar)) : "memory");
}

// One thread: `pieces` bulk copies of `bytes` each, from src + i * src_stride
// to dst + i * bytes, all counted on mbar.
__device__ __forceinline__ void bulk_load(unsigned char* dst, const unsigned char* src, uint32_t pieces,
                                          uint32_t bytes, uint64_t src_stride, uint64_t* mbar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(mbar)), "r"(pieces * bytes)
                 : "memory");
    for (uint32_t i = 0; i < pieces; ++i)
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         smem_u32(dst + i * bytes)),
                     "l"(src + i * src_stride), "r"(bytes), "r"(smem_u32(mbar))
                     : "memory");
}

// The 4 MMAs of one K block (K = 64) into the accumulator at tmem_d.  Every
// lane of the (converged) MMA warp runs this; the instructions are predicated
// on `leader`, so one thread issues them.  ad / bd: descriptors of the
// block; a K step of 16 elements moves the start address by 32 B.
__device__ __forceinline__ void issue_kblock_mma(uint64_t ad, uint64_t bd, uint32_t tmem_d, bool first,
                                                 uint32_t leader) {
    constexpr uint32_t idesc = umma_idesc(KNN_BM, KNN_BN);
#pragma unroll
    for (uint32_t s = 0; s < 4; ++s) {
        const uint32_t acc = (!first || s) ? 1u : 0u;
        asm volatile(
            "{\n .reg .pred p, l;\n setp.ne.b32 p, %4, 0;\n setp.ne.b32 l, %5, 0;\n"
            " @l tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem_d),
            "l"(ad + s * 2u), "l"(bd + s * 2u), "r"(idesc), "r"(acc), "r"(leader)
            : "memory");
    }
}

// Arrives on mbar once every MMA this thread issued so far has completed.
__device__ __forceinline__ void mma_commit(uint64_t* mbar, uint32_t leader) {
    asm volatile(
        "{\n .reg .pred l;\n setp.ne.b32 l, %1, 0;\n"
        " @l tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(smem_u32(mbar)),
        "r"(leader)
        : "memory");
}

template <int KMAX>
__device__ __forceinline__ void topk_push(float (&vals)[KMAX], uint32_t (&ids)[KMAX], float v, uint32_t id) {
    vals[KMAX - 1] = v;
    ids[KMAX - 1] = id;
#pragma unroll
    for (int i = KMAX - 1; i >= 1; --i) {
        if (vals[i] > vals[i - 1]) {
            const float tv = vals[i];
            vals[i] = vals[i - 1];
            vals[i - 1] = tv;
            const uint32_t ti = ids[i];
            ids[i] = ids[i - 1];
            ids[i - 1] = ti;
        }
    }
}

// k-th largest of a list sorted in descending order (k in [1, KMAX]): the
// minimum of its first k entries, written so that the registers are never
// indexed at run time
template <int KMAX>
__device__ __forceinline__ float kth_value(const float (&vals)[KMAX], uint32_t k) {
    float t = vals[0];
#pragma unroll
    for (int i = 1; i < KMAX; ++i) t = fminf(t, (uint32_t)i < k ? vals[i] : INFINITY);
    return t;
}

template <int KMAX>
__global__ void __launch_bounds__(KnnRoles<KMAX>::THREADS, 1)
    k_cos_topk(const unsigned char* __restrict__ Q, uint64_t nq, const unsigned char* __restrict__ Dall, uint64_t ndb,
               uint32_t dpad, const uint64_t* __restrict__ qself, uint32_t k, uint32_t* __restrict__ idx_out,
               float* __restrict__ sim_out, uint32_t* __restrict__ err, uint32_t t0, uint32_t t1, uint32_t tiles_per,
               uint32_t split0, uint2* __restrict__ part) {
    using R = KnnRoles<KMAX>;
    extern __shared__ unsigned char knn_smem_raw[];
    __shared__ uint64_t bar_a, bar_full[KNN_STAGES], bar_empty[KNN_STAGES], bar_acc_full[KNN_ACC],
        bar_acc_free[KNN_ACC];
    __shared__ uint64_t s_loaded, s_landed, s_issued;    // stages copied / seen landed / stages whose MMAs issued
    __shared__ uint32_t tmem_slot, s_a_landed;
    __shared__ volatile uint32_t abort_flag;
    unsigned char* smem = (unsigned char*)(((uintptr_t)knn_smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t nkb = dpad / 64;
    const uint32_t a_bytes = nkb * KNN_A_KB;
    unsigned char* sA = smem;
    auto sB = [&](uint32_t st) { return smem + a_bytes + st * KNN_B_KB; };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t first = t0 + blockIdx.y * tiles_per;              // this split's tiles [first, last)
    const uint32_t last = min(t1, first + tiles_per);
    const uint64_t ntiles = first < last ? last - first : 0, nstages = ntiles * nkb;
    const unsigned char* D = Dall + (uint64_t)first * nkb * KNN_B_KB;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(KNN_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x == 0) {
        abort_flag = 0;
        s_loaded = s_landed = s_issued = 0;
        s_a_landed = 0;
        mbar_init(&bar_a, 1);
        for (int i = 0; i < KNN_STAGES; ++i) {
            mbar_init(&bar_full[i], 1);
            mbar_init(&bar_empty[i], 1);
        }
        for (int i = 0; i < KNN_ACC; ++i) {
            mbar_init(&bar_acc_full[i], 1);
            mbar_init(&bar_acc_free[i], R::EPI);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;

    // per-thread top-k (epilogue warps)
    float vals[KMAX];
    uint32_t ids[KMAX];
#pragma unroll
    for (int i = 0; i < KMAX; ++i) { vals[i] = -INFINITY; ids[i] = 0xffffffffu; }
    const int quarter = warp & 3, slice = warp >> 2;
    const uint32_t qrow = 32u * quarter + lane;                 // TMEM lane = accumulator row = query
    const uint64_t myq = (uint64_t)blockIdx.x * KNN_BM + qrow;
    // column ids fit 32 bits (the host keeps n_db below 2^32 - 1); ~0 = no row to skip
    const uint32_t self = (warp < R::EPI && qself && myq < nq && qself[myq] < ndb) ? (uint32_t)qself[myq] : ~0u;
    const uint32_t ndb32 = (uint32_t)ndb;

    if (warp == R::COPY) {
        // ---- copies ----
        uint64_t loaded = 0;
        if (ntiles) {
            if (lane == 0) bulk_load(sA, Q + (uint64_t)blockIdx.x * a_bytes, nkb, KNN_A_KB, KNN_A_KB, &bar_a);
            for (uint64_t sg = 0; sg < nstages; ++sg) {
                const uint32_t st = (uint32_t)(sg % KNN_STAGES), use = (uint32_t)(sg / KNN_STAGES);
                // the stage is free once the MMAs of its previous K block completed
                if (sg >= (uint64_t)KNN_STAGES &&
                    !__all_sync(0xffffffffu, mbar_wait(&bar_empty[st], (use - 1u) & 1u, &abort_flag))) {
                    abort_flag = 1;
                    break;
                }
                if (lane == 0) bulk_load(sB(st), D + sg * KNN_B_KB, 2, KNN_B_KB / 2, KNN_B_KB / 2, &bar_full[st]);
                loaded = sg + 1;
            }
        }
        if (lane == 0) s_loaded = loaded;
    } else if (warp == R::MMA) {
        // ---- MMA issue ----
        uint64_t landed = 0, issued = 0;
        uint32_t a_ok = 0;
        if (ntiles) {
            const uint64_t ad0 = umma_desc(smem_u32(sA)), bd0 = umma_desc(smem_u32(sB(0)));
            bool ok = a_ok = __all_sync(0xffffffffu, mbar_wait(&bar_a, 0, &abort_flag));
            uint64_t sg = 0;
            for (uint64_t j = 0; ok && j < ntiles; ++j) {
                const uint32_t acc = (uint32_t)(j % KNN_ACC), ause = (uint32_t)(j / KNN_ACC);
                if (j >= (uint64_t)KNN_ACC &&
                    !__all_sync(0xffffffffu, mbar_wait(&bar_acc_free[acc], (ause - 1u) & 1u, &abort_flag))) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (uint32_t kb = 0; kb < nkb; ++kb, ++sg) {
                    const uint32_t st = (uint32_t)(sg % KNN_STAGES), use = (uint32_t)(sg / KNN_STAGES);
                    if (!__all_sync(0xffffffffu, mbar_wait(&bar_full[st], use & 1u, &abort_flag))) {
                        ok = false;
                        break;
                    }
                    landed = sg + 1;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    issue_kblock_mma(ad0 + kb * (KNN_A_KB >> 4), bd0 + st * (KNN_B_KB >> 4), tmem + acc * KNN_BN,
                                     kb == 0, lane == 0);
                    mma_commit(&bar_empty[st], lane == 0);
                    issued = sg + 1;
                }
                if (!ok) break;
                mma_commit(&bar_acc_full[acc], lane == 0);
            }
            if (!ok) abort_flag = 1;
        }
        if (lane == 0) {
            s_landed = landed;
            s_issued = issued;
            s_a_landed = a_ok;
        }
    } else {
        // ---- epilogue ----
        float thr = -INFINITY;                     // k-th best so far
        for (uint64_t j = 0; j < ntiles; ++j) {
            const uint32_t acc = (uint32_t)(j % KNN_ACC), ause = (uint32_t)(j / KNN_ACC);
            // warp-uniform decision: the loads below are .sync.aligned
            if (!__all_sync(0xffffffffu, mbar_wait(&bar_acc_full[acc], ause & 1u, &abort_flag))) {
                abort_flag = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // Blocks are software-pipelined where registers allow (16-column
            // blocks): block bl+1's TMEM load is in flight while block bl is
            // scanned, with two register sets alternating.  32-column blocks
            // (k > 16) load and wait one block at a time.
            constexpr int NB = R::BW <= 16 ? 2 : 1;
            uint32_t r[NB][R::BW];
            float bmax[NB];
            const uint32_t tl = tmem + acc * KNN_BN + (uint32_t)(slice * R::CW) + ((uint32_t)(32 * quarter) << 16);
            if constexpr (NB == 2) {
                __syncwarp();
                tmem_ld_max(tl, r[0], bmax[0]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            }
            // (unrolled only when pipelined: four copies of the 32-entry
            // insertion path would not fit the instruction cache)
            constexpr int UNR = NB == 2 ? R::BLOCKS : 1;
#pragma unroll UNR
            for (int bl = 0; bl < R::BLOCKS; ++bl) {
                const int cb = NB == 2 ? (bl & 1) : 0;
                __syncwarp();
                if constexpr (NB == 1) {
                    tmem_ld_max(tl + (uint32_t)(bl * R::BW), r[0], bmax[0]);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                }
                if (NB == 2 && bl + 1 < R::BLOCKS) {
                    tmem_ld_max(tl + (uint32_t)((bl + 1) * R::BW), r[(cb ^ 1) % NB], bmax[(cb ^ 1) % NB]);
                } else if (bl + 1 == R::BLOCKS) {
                    // release the accumulator: this warp's values are all in registers
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bar_acc_free[acc]);
                }
                // the block's largest similarity first: most blocks cannot enter
                if (bmax[cb] > thr) {
                    unsigned cand = 0;
#pragma unroll
                    for (int t = 0; t < R::BW; ++t) cand |= (__uint_as_float(r[cb][t]) > thr ? 1u : 0u) << t;
                    const uint32_t col0 = (first + (uint32_t)j) * KNN_BN + (uint32_t)(slice * R::CW + bl * R::BW);
                    while (cand) {
                        const int t = __ffs(cand) - 1;
                        cand &= cand - 1;
                        float v = __uint_as_float(r[cb][0]);
#pragma unroll
                        for (int u = 1; u < R::BW; ++u) v = t == u ? __uint_as_float(r[cb][u]) : v;
                        const uint32_t col = col0 + (uint32_t)t;
                        if (v > thr && col < ndb32 && col != self) {
                            topk_push<KMAX>(vals, ids, v, col);
                            thr = kth_value<KMAX>(vals, k);
                        }
                    }
                }
                if (NB == 2 && bl + 1 < R::BLOCKS) {
                    __syncwarp();
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                }
            }
        }
    }
    __syncthreads();
    const bool aborted = abort_flag != 0;
    if (aborted) {
        if (threadIdx.x == 0) atomicOr(err, KNN_ERR_TIMEOUT);
        if (warp == R::MMA && lane == 0 && ntiles) {
            // last bounded waits for the copies and MMAs that may still be in flight
            volatile uint32_t never = 0;
            if (!s_a_landed) mbar_wait(&bar_a, 0, &never);
            for (uint64_t sg = s_landed; sg < s_loaded; ++sg)
                mbar_wait(&bar_full[sg % KNN_STAGES], (uint32_t)((sg / KNN_STAGES) & 1), &never);
            if (s_issued) {     // a commit covers every earlier MMA
                const uint64_t sg = s_issued - 1;
                mbar_wait(&bar_empty[sg % KNN_STAGES], (uint32_t)((sg / KNN_STAGES) & 1), &never);
            }
        }
    } else if (part) {
        // the first k entries of every slice's list, for k_merge_topk
        if (warp < R::EPI && myq < nq) {
            uint2* to = part + (((uint64_t)(split0 + blockIdx.y) * nq + myq) * R::SLICES + slice) * k;
#pragma unroll
            for (int i = 0; i < KMAX; ++i)
                if ((uint32_t)i < k) to[i] = make_uint2(__float_as_uint(vals[i]), ids[i]);
        }
    } else {
        // merge the slices' sorted lists per query (the stages are free now)
        float* pv = reinterpret_cast<float*>(smem);                         // [SLICES][128][KMAX]
        uint32_t* pi = reinterpret_cast<uint32_t*>(smem + (size_t)R::SLICES * KNN_BM * KMAX * 4);
        if (warp < R::EPI) {
            const size_t base = ((size_t)slice * KNN_BM + qrow) * KMAX;
#pragma unroll
            for (int i = 0; i < KMAX; ++i) { pv[base + i] = vals[i]; pi[base + i] = ids[i]; }
        }
        __syncthreads();
        if (warp < 4 && myq < nq) {
            float thr = kth_value<KMAX>(vals, k);
            for (int sl = 1; sl < R::SLICES; ++sl) {
                const size_t b2 = ((size_t)sl * KNN_BM + qrow) * KMAX;
                for (uint32_t i = 0; i < k; ++i) {
                    const float v = pv[b2 + i];
                    if (!(v > thr)) break;     // sorted: the rest cannot enter
                    topk_push<KMAX>(vals, ids, v, pi[b2 + i]);
                    thr = kth_value<KMAX>(vals, k);
                }
            }
#pragma unroll
            for (int i = 0; i < KMAX; ++i) {
                if ((uint32_t)i < k) {
                    idx_out[myq * k + i] = ids[i];
                    sim_out[myq * k + i] = vals[i];
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(KNN_TMEM_COLS)
                     : "memory");
    }
}

// Joins the sorted lists of one query (splits x slices lists of k entries),
// a warp per query: k rounds of picking the best head.  Among equal
// similarities the lower slice comes first, then the lower row: the order in
// which one CTA over the whole database admits them (its slice lists keep
// row order, and are joined slice by slice).
__global__ void __launch_bounds__(128) k_merge_topk(const uint2* __restrict__ part, uint64_t nq, uint32_t splits,
                                                    uint32_t slices, uint32_t k, uint32_t* __restrict__ idx_out,
                                                    float* __restrict__ sim_out) {
    extern __shared__ uint8_t merge_pos[];               // [warps][lists]: entries taken of each list
    const int lane = threadIdx.x & 31;
    const uint64_t q = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (q >= nq) return;
    const uint32_t lists = splits * slices;
    uint8_t* pos = merge_pos + (size_t)(threadIdx.x >> 5) * lists;
    for (uint32_t l = lane; l < lists; l += 32) pos[l] = 0;
    for (uint32_t r = 0; r < k; ++r) {
        float bv = -INFINITY;
        uint32_t bid = 0xffffffffu, bsl = 0xffffffffu, bl = 0xffffffffu;
        auto better = [&](float v, uint32_t sl, uint32_t id) {
            return v > bv || (v == bv && v > -INFINITY && (sl < bsl || (sl == bsl && id < bid)));
        };
        for (uint32_t l = lane; l < lists; l += 32) {
            const uint32_t i = pos[l], sl = l % slices;
            if (i >= k) continue;
            const uint2 e = part[(((uint64_t)(l / slices)) * nq + q) * slices * k + (uint64_t)sl * k + i];
            if (better(__uint_as_float(e.x), sl, e.y)) { bv = __uint_as_float(e.x); bid = e.y; bsl = sl; bl = l; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float v = __shfl_xor_sync(FULL, bv, o);
            const uint32_t id = __shfl_xor_sync(FULL, bid, o), sl = __shfl_xor_sync(FULL, bsl, o), l = __shfl_xor_sync(FULL, bl, o);
            if (better(v, sl, id)) { bv = v; bid = id; bsl = sl; bl = l; }
        }
        if (bl != 0xffffffffu && (uint32_t)lane == (bl & 31u)) ++pos[bl];
        if (lane == 0) {
            idx_out[q * k + r] = bid;
            sim_out[q * k + r] = bv;
        }
    }
}

// One launch of k_cos_topk over database tiles [t0, t1) in `splits` splits;
// part null: the whole database, straight to the results.
struct KnnArgs {
    const unsigned char *Q, *D;
    uint64_t nq, ndb;
    uint32_t dpad;
    const uint64_t* qself;
    uint32_t k;
    uint32_t* idx;
    float* sim;
    uint32_t* err;
    uint2* part;
};

template <int KMAX>
cudaError_t knn_launch(const KnnArgs& a, uint32_t t0, uint32_t t1, uint32_t splits, uint32_t split0, cudaStream_t s) {
    // query tile + KNN_STAGES K-block stages (reused at the end for the slices' lists)
    const size_t tiles = (size_t)(a.dpad / 64) * KNN_A_KB + (size_t)KNN_STAGES * KNN_B_KB;
    const size_t lists = (size_t)KnnRoles<KMAX>::SLICES * KNN_BM * KMAX * 8;
    const size_t smem = std::max(tiles, lists) + 1024;
    const cudaError_t e = cudaFuncSetAttribute(k_cos_topk<KMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const dim3 grid((unsigned)((a.nq + KNN_BM - 1) / KNN_BM), splits);
    const uint32_t per = (t1 - t0 + splits - 1) / splits;
    k_cos_topk<KMAX><<<grid, KnnRoles<KMAX>::THREADS, smem, s>>>(a.Q, a.nq, a.D, a.ndb, a.dpad, a.qself, a.k, a.idx, a.sim,
                                                                a.err, t0, t1, per, split0, a.part);
    return cudaGetLastError();
}

// compile-time selection by k: the shortest list that holds it (insertion and
// the k-th-value scan cost O(KMAX))
cudaError_t knn_launch_k(const KnnArgs& a, uint32_t t0, uint32_t t1, uint32_t splits, uint32_t split0, cudaStream_t s) {
    return a.k <= 8    ? knn_launch<8>(a, t0, t1, splits, split0, s)
           : a.k <= 12 ? knn_launch<12>(a, t0, t1, splits, split0, s)
           : a.k <= 16 ? knn_launch<16>(a, t0, t1, splits, split0, s)
                       : knn_launch<32>(a, t0, t1, splits, split0, s);
}

}  // namespace
}  // namespace ep

using namespace ep;

// The result of a call that checks its ids on the way to the device: one that
// got no device or no memory is refused for a bad id all the same.
static int refused(int rc, const uint32_t* ids, uint64_t n, uint64_t bound, const char* msg) {
    if (rc == EP_OK || rc == EP_ERR_INVALID_ARG || all_below(ids, n, bound)) return rc;
    return knn_fail(EP_ERR_INVALID_ARG, msg);
}

static int embed_run(int device, uint64_t n_nodes, const uint64_t* fptr, const uint32_t* fids,
                     const float* fweight, uint32_t n_feat, uint32_t dims, const float* table, float* out) {
    const uint64_t nf = fptr[n_nodes];
    KCK(cudaSetDevice(device), "select device");
    if (!n_nodes) return EP_OK;
    cudaStream_t s;
    KCK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "stream");
    struct SG { cudaStream_t s; ~SG() { cudaStreamDestroy(s); } } sg{s};
    Arena ar;
    const size_t out_bytes = (size_t)n_nodes * dims * 4;
    const size_t o_bad = ar.reserve(4), o_ptr = ar.reserve((n_nodes + 1) * 8), o_ids = ar.reserve(nf * 4),
                 o_tab = ar.reserve((size_t)n_feat * dims * 4), o_w = ar.reserve(fweight ? (size_t)n_feat * 4 : 0),
                 o_out = ar.reserve(out_bytes);
    KCK(ar.mem.alloc(ar.used), "alloc");
    bool ok = true;
    KCK(upload_ids(ar.at<uint32_t>(o_ids), fids, nf, n_feat, ar.at<uint32_t>(o_bad), s, &ok), "upload");
    if (!ok) return knn_fail(EP_ERR_INVALID_ARG, "feature id out of range");
    ResultPages pages(out, host_bytes(out, out_bytes));
    KCK(upload(ar.at<void>(o_ptr), fptr, (n_nodes + 1) * 8, s), "upload");
    KCK(upload(ar.at<void>(o_tab), table, (size_t)n_feat * dims * 4, s), "upload");
    if (fweight) KCK(upload(ar.at<void>(o_w), fweight, (size_t)n_feat * 4, s), "upload");
    RowsParams p{};
    p.n = n_nodes;
    p.ptr = ar.at<uint64_t>(o_ptr);
    p.ids = ar.at<uint32_t>(o_ids);
    p.w = ar.at<float>(o_w);
    p.d = dims;
    p.table = ar.at<float>(o_tab);
    p.out = ar.at<float>(o_out);
    KCK((fweight ? launch_rows<ROWS_WEIGHTED>(p, s) : launch_rows<ROWS_MEAN>(p, s)), "embed launch");
    KCK(download((char*)out, p.out, out_bytes, pages, s), "embed");
    return EP_OK;
}

extern "C" int ep_embed_features(int device, uint64_t n_nodes, const uint64_t* fptr, const uint32_t* fids,
                                 const float* fweight, uint32_t n_feat, uint32_t dims, const float* table,
                                 float* out) {
    if (!fptr || !out || (n_nodes && !table && n_feat) || dims == 0 || dims > 512)
        return knn_fail(EP_ERR_INVALID_ARG, "invalid arguments (dims must be in [1, 512])");
    if (!monotone(fptr, n_nodes)) return knn_fail(EP_ERR_INVALID_ARG, "fptr is not monotone");
    if (!n_nodes && !all_below(fids, fptr[0], n_feat))      // no node reads them, but they are the caller's
        return knn_fail(EP_ERR_INVALID_ARG, "feature id out of range");
    return refused(embed_run(device, n_nodes, fptr, fids, fweight, n_feat, dims, table, out), fids, fptr[n_nodes], n_feat,
                   "feature id out of range");
}

static int align_run(int device, uint64_t n_nodes, const uint64_t* row_ptr, const uint32_t* cols,
                     const float* w_cdf, uint32_t dims, const float* emb, float alpha, uint64_t max_neighbors, float* out) {
    const uint64_t ne = row_ptr[n_nodes];
    KCK(cudaSetDevice(device), "select device");
    if (!n_nodes) return EP_OK;
    cudaStream_t s;
    KCK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "stream");
    struct SG { cudaStream_t s; ~SG() { cudaStreamDestroy(s); } } sg{s};
    Arena ar;
    const size_t out_bytes = (size_t)n_nodes * dims * 4;
    const size_t o_bad = ar.reserve(4), o_nh = ar.reserve(sizeof(Hubs)), o_rp = ar.reserve((n_nodes + 1) * 8), o_cols = ar.reserve(ne * 4),
                 o_cdf = ar.reserve(ne * 4), o_emb = ar.reserve(out_bytes),
                 o_hubs = ar.reserve((ne / (HUB_ROWS + 1) + 1) * 4), o_out = ar.reserve(out_bytes);
    KCK(ar.mem.alloc(ar.used), "alloc");
    bool ok = true;
    KCK(upload_ids(ar.at<uint32_t>(o_cols), cols, ne, n_nodes, ar.at<uint32_t>(o_bad), s, &ok), "upload");
    if (!ok) return knn_fail(EP_ERR_INVALID_ARG, "column id out of range");
    ResultPages pages(out, host_bytes(out, out_bytes));
    KCK(upload(ar.at<void>(o_rp), row_ptr, (n_nodes + 1) * 8, s), "upload");
    KCK(upload(ar.at<void>(o_cdf), w_cdf, ne * 4, s), "upload");
    KCK(upload(ar.at<void>(o_emb), emb, out_bytes, s), "upload");
    RowsParams p{};
    p.n = n_nodes;
    p.ptr = ar.at<uint64_t>(o_rp);
    p.ids = ar.at<uint32_t>(o_cols);
    p.w = ar.at<float>(o_cdf);
    p.d = dims;
    p.table = ar.at<float>(o_emb);
    p.alpha = alpha;
    p.kmax = max_neighbors ? max_neighbors : ~0ull;
    p.hubs = ar.at<uint32_t>(o_hubs);
    p.hub = ar.at<Hubs>(o_nh);
    p.out = ar.at<float>(o_out);
    cudaEvent_t e0, e1;
    KCK(cudaEventCreate(&e0), "events");
    KCK(cudaEventCreate(&e1), "events");
    struct EG { cudaEvent_t a, b; ~EG() { cudaEventDestroy(a); cudaEventDestroy(b); } } eg{e0, e1};
    KCK(cudaMemsetAsync(p.hub, 0, sizeof(Hubs), s), "clear");
    cudaEventRecord(e0, s);
    const unsigned scan = (unsigned)std::min<uint64_t>((n_nodes + 255) / 256, 152 * 8);
    k_hub_edges<<<scan, 256, 0, s>>>(p);
    k_find_hubs<<<scan, 256, 0, s>>>(p);
    KCK(launch_rows<ROWS_ALIGN>(p, s), "align launch");
    cudaEventRecord(e1, s);
    KCK(download((char*)out, p.out, out_bytes, pages, s), "align");
    cudaEventElapsedTime(&g_knn_ms, e0, e1);
    return EP_OK;
}

extern "C" int ep_align(int device, uint64_t n_nodes, const uint64_t* row_ptr, const uint32_t* cols,
                        const float* w_cdf, uint32_t dims, const float* emb, float alpha, uint64_t max_neighbors,
                        float* out) {
    if (!row_ptr || (n_nodes && (!emb || !out)) || dims == 0 || dims > 512)
        return knn_fail(EP_ERR_INVALID_ARG, "invalid arguments (dims must be in [1, 512])");
    if (alpha > 1.f || alpha != alpha) return knn_fail(EP_ERR_INVALID_ARG, "alpha must be <= 1 (negative: adaptive)");
    const uint64_t ne = row_ptr[n_nodes];
    if (ne && (!cols || !w_cdf)) return knn_fail(EP_ERR_INVALID_ARG, "null edge arrays");
    if (!monotone(row_ptr, n_nodes)) return knn_fail(EP_ERR_INVALID_ARG, "row_ptr is not monotone");
    if (!n_nodes && ne) return knn_fail(EP_ERR_INVALID_ARG, "column id out of range");
    return refused(align_run(device, n_nodes, row_ptr, cols, w_cdf, dims, emb, alpha, max_neighbors, out), cols, ne, n_nodes,
                   "column id out of range");
}

extern "C" int ep_knn_cosine(int device, uint64_t n_db, uint32_t dims, const float* db, uint64_t n_q,
                             const float* q, const uint64_t* q_self, uint32_t k, uint32_t* idx_out, float* sim_out) {
    if (dims == 0 || dims > 256) return knn_fail(EP_ERR_INVALID_ARG, "dims must be in [1, 256]");
    if (k == 0 || k > 32) return knn_fail(EP_ERR_INVALID_ARG, "k must be in [1, 32]");
    if (n_db >= 0xffffffffull) return knn_fail(EP_ERR_INVALID_ARG, "n_db must be below 2^32 - 1");
    if ((n_db && !db) || (n_q && (!q || !idx_out || !sim_out)))
        return knn_fail(EP_ERR_INVALID_ARG, "null array");
    if (q_self)
        for (uint64_t i = 0; i < n_q; ++i)
            if (q_self[i] != ~0ull && q_self[i] >= n_db) return knn_fail(EP_ERR_INVALID_ARG, "q_self out of range");
    KCK(cudaSetDevice(device), "select device");
    if (!n_q) return EP_OK;
    const uint32_t dpad = (dims + 63) / 64 * 64;
    const uint64_t q_tile_bytes = (uint64_t)(dpad / 64) * 128 * KNN_BM, db_tile_bytes = (uint64_t)(dpad / 64) * 128 * KNN_BN;
    const uint64_t db_tiles = (n_db + KNN_BN - 1) / KNN_BN, q_tiles = (n_q + KNN_BM - 1) / KNN_BM;
    // Plan.  One CTA per 128 queries over the whole database fills the chip
    // from about 128 query tiles on; fewer tiles split the database, so that
    // tiles x splits come near the 152 SMs, and take it in chunks of about
    // 32 MB, each searched while the next one is uploaded and normalised.
    // 8,192 x 262,144 x 256, top 10 (64 CTAs, 1.89 ms of search, after a 1.5 ms
    // upload): the call 4.25 -> 2.7 ms; 739 x 48,046 x 48, top 20: 1.31 -> 0.54.
    // Two splits fit the SMs up to 76 tiles; the call in ms, one / two: 76 tiles
    // x 262,144 x 256 4.11 / 2.71, 77 tiles (two waves) 4.12 / 4.43; x 100,000 x
    // 64 1.13 / 0.95 and 1.12 / 1.35.  (Chunks without a split: 3.77 and 1.13
    // at 77 tiles.)
    const uint64_t db_bytes = n_db * dims * 4;
    uint32_t chunks = 1, splits = 1;                   // splits per chunk
    if (q_tiles <= 76 && db_tiles >= 8) {
        splits = (uint32_t)std::min<uint64_t>(152 / q_tiles, db_tiles / 4);
        chunks = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>({16, db_bytes >> 25, db_tiles / (4ull * splits)}));
    }
    const bool split = splits * chunks > 1;
    const uint32_t slices = k <= 16 ? KnnRoles<16>::SLICES : KnnRoles<32>::SLICES;
    cudaStream_t s, up;
    KCK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "stream");
    struct SG { cudaStream_t s; ~SG() { cudaStreamDestroy(s); } } sg{s};
    KCK(cudaStreamCreateWithFlags(&up, cudaStreamNonBlocking), "stream");
    SG ug{up};
    struct EV {
        cudaEvent_t e = nullptr;
        ~EV() { if (e) cudaEventDestroy(e); }
    };
    // one timed stretch for each chunk's search, the last one with the join of the splits
    std::vector<EV> ready(chunks), t_from(chunks), t_to(chunks);
    for (uint32_t c = 0; c < chunks; ++c) {
        KCK(cudaEventCreateWithFlags(&ready[c].e, cudaEventDisableTiming), "events");
        KCK(cudaEventCreate(&t_from[c].e), "events");
        KCK(cudaEventCreate(&t_to[c].e), "events");
    }
    Arena ar;
    const uint64_t chunk_tiles = (db_tiles + chunks - 1) / chunks, chunk_rows = chunk_tiles * KNN_BN;
    const size_t o_err = ar.reserve(4), o_raw = ar.reserve(std::min(n_db, chunk_rows) * dims * 4), o_qraw = ar.reserve(n_q * dims * 4),
                 o_D = ar.reserve(std::max<uint64_t>(db_tiles, 1) * db_tile_bytes), o_Q = ar.reserve(q_tiles * q_tile_bytes),
                 o_idx = ar.reserve(n_q * k * 4), o_sim = ar.reserve(n_q * k * 4), o_self = ar.reserve(q_self ? n_q * 8 : 0),
                 o_part = ar.reserve(split ? (uint64_t)chunks * splits * n_q * slices * k * 8 : 0);
    KCK(ar.mem.alloc(ar.used), "alloc");
    KCK(cudaMemsetAsync(ar.at<void>(o_err), 0, 4, s), "clear");
    KCK(upload(ar.at<void>(o_self), q_self, q_self ? n_q * 8 : 0, s), "upload");
    KCK(upload(ar.at<void>(o_qraw), q, n_q * dims * 4, s), "upload");
    k_norm_swz<<<(unsigned)((q_tiles * KNN_BM * 32 + 255) / 256), 256, 0, s>>>(0, n_q, q_tiles * KNN_BM, dims, dpad, 7,
                                                                              ar.at<float>(o_qraw),
                                                                              ar.at<unsigned char>(o_Q));
    KCK(cudaGetLastError(), "normalise");
    KnnArgs a{ar.at<unsigned char>(o_Q), ar.at<unsigned char>(o_D), n_q, n_db, dpad,
              q_self ? ar.at<uint64_t>(o_self) : nullptr, k, ar.at<uint32_t>(o_idx), ar.at<float>(o_sim),
              ar.at<uint32_t>(o_err), split ? ar.at<uint2>(o_part) : nullptr};
    for (uint32_t c = 0; c < chunks; ++c) {
        const uint64_t tile0 = std::min<uint64_t>(db_tiles, c * chunk_tiles), tile1 = std::min(db_tiles, tile0 + chunk_tiles);
        const uint64_t row0 = std::min<uint64_t>(n_db, c * chunk_rows), row1 = std::min(n_db, row0 + chunk_rows);
        KCK(upload(ar.at<float>(o_raw), db + row0 * dims, (row1 - row0) * dims * 4, up), "upload");   // after the chunk before
        if (tile1 > tile0)
            k_norm_swz<<<(unsigned)((tile1 - tile0) * KNN_BN * 32 / 256), 256, 0, up>>>(
                tile0 * KNN_BN, n_db, tile1 * KNN_BN, dims, dpad, 8, ar.at<float>(o_raw), ar.at<unsigned char>(o_D));
        KCK(cudaGetLastError(), "normalise");
        cudaEventRecord(ready[c].e, up);
        cudaStreamWaitEvent(s, ready[c].e, 0);
        cudaEventRecord(t_from[c].e, s);
        KCK(knn_launch_k(a, (uint32_t)tile0, (uint32_t)tile1, splits, c * splits, s), "knn launch");
        if (c + 1 < chunks) cudaEventRecord(t_to[c].e, s);
    }
    if (split) {
        const uint32_t lists = chunks * splits * slices;
        k_merge_topk<<<(unsigned)((n_q + 3) / 4), 128, 4 * (size_t)lists, s>>>(a.part, n_q, chunks * splits, slices, k, a.idx,
                                                                             a.sim);
        KCK(cudaGetLastError(), "knn merge");
    }
    cudaEventRecord(t_to[chunks - 1].e, s);
    uint32_t herr = 0;
    ResultPages pi(idx_out, host_bytes(idx_out, n_q * k * 4)), ps(sim_out, host_bytes(sim_out, n_q * k * 4));
    KCK(download((char*)idx_out, a.idx, n_q * k * 4, pi, s), "download");
    KCK(download((char*)sim_out, a.sim, n_q * k * 4, ps, s), "download");
    KCK(cudaMemcpyAsync(&herr, ar.at<void>(o_err), 4, cudaMemcpyDeviceToHost, s), "download");
    KCK(cudaStreamSynchronize(s), "knn");
    g_knn_ms = 0.f;
    for (uint32_t c = 0; c < chunks; ++c) {
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, t_from[c].e, t_to[c].e) == cudaSuccess) g_knn_ms += ms;
    }
    if (herr) return knn_fail(EP_ERR_DEVICE, "tensor-core wait timed out");
    return EP_OK;
}

extern "C" const char* ep_knn_last_error(void) { return g_knn_err.c_str(); }

extern "C" float ep_knn_last_kernel_ms(void) { return g_knn_ms; }
