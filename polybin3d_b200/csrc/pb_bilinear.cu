// Bilinear maps: out[o](x) = sum_t [o_t == o] c_t G[i_t](x) G[j_t](x).
//
// The gradient of a weighted sum of triplet sums, sum_t gamma_t sum_x G_a G_b G_c, with
// respect to map G_o is the map sum over the triplets' legs of gamma_t times the product of
// the other two maps; gathering all legs that end on the same output into one real-space
// map leaves one forward transform per output instead of one per (pair of maps).
//
// A block stages a tile of 32 BL_V voxels of every input map in shared memory as
// [map][voxel]; its warps take the outputs round-robin, lane l owning tile voxels l, l+32,
// ..., l+32(BL_V-1) (a warp reads one map at 32 consecutive voxels: one wavefront).  An
// output's terms are sorted by (i, j): per i-group a lane accumulates s = sum_j c G_j, then
// acc += G_i s.  Term records are read by the whole warp at once (a broadcast load) and stay
// in L1 across tiles; four blocks per SM keep enough warps in flight to cover their latency.
#include <algorithm>
#include <cstring>
#include <tuple>
#include <vector>
#include "pb_common.cuh"

namespace pb {

constexpr int BL_THREADS = 256;
constexpr int BL_MAXG = 128;      // input maps
constexpr int BL_MAXOUT = 4096;   // outputs

// term record: code = j | i << 8 | (first term of an i-group) << 16, the coefficient in
// FP32 and FP64
struct BlTerm {
    uint32_t code;
    float cf;
    double c;
};

template <typename T>
__device__ __forceinline__ T term_coef(const BlTerm &r);
template <>
__device__ __forceinline__ float term_coef<float>(const BlTerm &r) { return r.cf; }
template <>
__device__ __forceinline__ double term_coef<double>(const BlTerm &r) { return r.c; }

// BL_V voxels per lane (8 in FP32, 4 in FP64: the same registers), tile = 32 BL_V voxels
template <typename T, int BL_V>
__global__ void __launch_bounds__(BL_THREADS, 4) bilinear_kernel(const T *G, int n_g, int64_t n_vox,
                                                                 const int32_t *offs, const BlTerm *rec, int n_out,
                                                                 T *out) {
    extern __shared__ __align__(16) unsigned char bl_smem[];
    constexpr int BL_TILE = 32 * BL_V;
    T *sg = reinterpret_cast<T *>(bl_smem);  // [map][BL_TILE]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = BL_THREADS >> 5;
    for (int64_t v0 = (int64_t)blockIdx.x * BL_TILE; v0 < n_vox; v0 += (int64_t)gridDim.x * BL_TILE) {
        __syncthreads();
        for (int e = threadIdx.x; e < n_g * BL_TILE; e += BL_THREADS) {
            const int m = e / BL_TILE, v = e - m * BL_TILE;
            sg[e] = (v0 + v < n_vox) ? G[(int64_t)m * n_vox + v0 + v] : (T)0;
        }
        __syncthreads();
        for (int o = warp; o < n_out; o += nw) {
            T acc[BL_V], s[BL_V], gi[BL_V];
#pragma unroll
            for (int u = 0; u < BL_V; ++u) acc[u] = s[u] = gi[u] = (T)0;
            const int r1 = offs[o + 1];
            for (int r = offs[o]; r < r1; ++r) {
                const BlTerm t = rec[r];
                if (t.code & (1u << 16)) {
#pragma unroll
                    for (int u = 0; u < BL_V; ++u) {
                        acc[u] += gi[u] * s[u];
                        s[u] = (T)0;
                    }
                    const T *gr = sg + ((t.code >> 8) & 0xFF) * BL_TILE + lane;
#pragma unroll
                    for (int u = 0; u < BL_V; ++u) gi[u] = gr[32 * u];
                }
                const T c = term_coef<T>(t);
                const T *gr = sg + (t.code & 0xFF) * BL_TILE + lane;
#pragma unroll
                for (int u = 0; u < BL_V; ++u) s[u] += c * gr[32 * u];
            }
#pragma unroll
            for (int u = 0; u < BL_V; ++u) {
                acc[u] += gi[u] * s[u];
                const int64_t x = v0 + lane + 32 * u;
                if (x < n_vox) out[(int64_t)o * n_vox + x] = acc[u];
            }
        }
    }
}

// ------------------------------------------------------------------------------------
// The same maps with four outputs per pass over the terms.  One output at a time costs one
// shared-memory load per FMA, which bounds it.  A block of four outputs shares its (i, j) pairs: a
// warp loads G_j once, 16 bytes per lane, and feeds the four outputs' sums s_o = sum_j c_oij G_j
// with four coefficients that come with the record, then acc_o += G_i s_o per i.  Outputs next to each
// other in (multipole, bin) order hold mostly the same pairs: 2752 terms of 16 bins, l = 0, 2 make 912
// records, 75 % of their coefficients non-zero.  Records go through shared memory 32 at a time: with 200
// KB of maps per SM there is little L1 left, and a record that misses it costs the warp an L2
// round trip (2850 us).  A zero coefficient stands for a term that is not there: harmless for finite values, so a tile
// that holds a NaN or an infinity (one FMA per staged value finds it) takes its records one by one, each into the outputs
// that its code names, and such a value reaches only the outputs that use its map.  Measured on a B200, those terms of 32 maps on 192^3: FP32 1980 us against
// 3170 us one output at a time, FP64 3960 against 8500 us; 66 % of
// the issue slots and 55 % of the shared-memory wavefronts (FP32).  Packed FP32 pairs (fma.rn.f32x2) were slower, 2460 us.
// ------------------------------------------------------------------------------------
constexpr int BB_OUT = 4;

// one (i, j) of a block of outputs: code as BlTerm's with the outputs that have the term in bits 17 - 20, the
// coefficients in FP32 and FP64 (0: no such term)
struct BbTerm {
    uint32_t code, pad[3];
    float cf[BB_OUT];
    double c[BB_OUT];
};
template <typename T> __device__ __forceinline__ T bb_coef(const BbTerm &r, int k);
template <> __device__ __forceinline__ float bb_coef<float>(const BbTerm &r, int k) { return r.cf[k]; }
template <> __device__ __forceinline__ double bb_coef<double>(const BbTerm &r, int k) { return r.c[k]; }

template <typename T> struct alignas(16) BbPack {
    static constexpr int N = 16 / sizeof(T);
    T v[N];
};
template <typename T> struct alignas(16) BbCoef {
    T v[BB_OUT];
};
constexpr int BB_P = 2;      // 16-byte packs per lane (1: 2340 us for the case above, more loads per sum)
constexpr int BB_OCC = 2;    // blocks per SM: 122 registers; three blocks spill (3350 us)
// A lane owns BB_P x 16 bytes of consecutive voxels in a span of 32 lanes; a tile holds n_span such spans of every map.  The
// units (span, block of outputs) go to the warps as they come free: blocks differ several times
// in their number of records.
template <typename T>
__global__ void __launch_bounds__(BL_THREADS, BB_OCC) bilinear_block_kernel(const T *G, int n_g, int64_t n_vox,
                                                                       const int32_t *offs, const BbTerm *rec, int n_out,
                                                                       int n_span, int vec, T *out) {
    extern __shared__ __align__(16) unsigned char bb_smem[];
    __shared__ int next;
    __shared__ uint32_t scode[BL_THREADS / 32][32];
    __shared__ BbCoef<T> scoef[BL_THREADS / 32][32];
    using Pack = BbPack<T>;
    constexpr int N = Pack::N, V = N * BB_P, SPAN = 32 * V;
    const int tile = SPAN * n_span;
    T *sg = reinterpret_cast<T *>(bb_smem);  // [map][tile]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = BL_THREADS >> 5;
    const int n_blk = (n_out + BB_OUT - 1) / BB_OUT;
    for (int64_t v0 = (int64_t)blockIdx.x * tile; v0 < n_vox; v0 += (int64_t)gridDim.x * tile) {
        const bool whole = vec && v0 + tile <= n_vox;   // rows 16-byte aligned and inside the map
        __syncthreads();
        if (threadIdx.x == 0) next = nw;
        T odd[N];   // 0, or NaN once a value is not finite
#pragma unroll
        for (int u = 0; u < N; ++u) odd[u] = (T)0;
        for (int m = warp; m < n_g; m += nw) {
            const T *src = G + (int64_t)m * n_vox + v0;
            T *dst = sg + m * tile;
            if (whole) {
#pragma unroll 4
                for (int e = lane * N; e < tile; e += 32 * N) {
                    const Pack g = *reinterpret_cast<const Pack *>(src + e);
                    *reinterpret_cast<Pack *>(dst + e) = g;
#pragma unroll
                    for (int u = 0; u < N; ++u) odd[u] += (T)0 * g.v[u];
                }
            } else {
                for (int e = lane; e < tile; e += 32) {
                    const T g = v0 + e < n_vox ? src[e] : (T)0;
                    dst[e] = g;
                    odd[0] += (T)0 * g;
                }
            }
        }
#pragma unroll
        for (int u = 1; u < N; ++u) odd[0] += odd[u];
        const bool finite = !__syncthreads_or(odd[0] != (T)0);
        int unit = warp;
        while (unit < n_span * n_blk) {
            const int blk = n_blk - 1 - unit / n_span, at = (unit % n_span) * SPAN + lane * N;
            T acc[BB_OUT][V], s[BB_OUT][V], gi[V];
#pragma unroll
            for (int u = 0; u < V; ++u) {
                gi[u] = (T)0;
#pragma unroll
                for (int k = 0; k < BB_OUT; ++k) acc[k][u] = s[k][u] = (T)0;
            }
            auto close = [&]() {
#pragma unroll
                for (int k = 0; k < BB_OUT; ++k)
#pragma unroll
                    for (int u = 0; u < V; ++u) {
                        acc[k][u] += gi[u] * s[k][u];
                        s[k][u] = (T)0;
                    }
            };
            if (!finite) {
                unsigned group = 0;   // outputs with a term of the current i
                auto close_used = [&]() {
#pragma unroll
                    for (int k = 0; k < BB_OUT; ++k)
                        if (group >> k & 1u) {
#pragma unroll
                            for (int u = 0; u < V; ++u) {
                                acc[k][u] += gi[u] * s[k][u];
                                s[k][u] = (T)0;
                            }
                        }
                    group = 0;
                };
#pragma unroll 1
                for (int q = offs[blk]; q < offs[blk + 1]; ++q) {
                    const BbTerm &t = rec[q];
                    const uint32_t now = t.code, used = now >> 17;
                    if (now & (1u << 16)) {
                        close_used();
#pragma unroll
                        for (int p = 0; p < BB_P; ++p)
#pragma unroll
                            for (int u = 0; u < N; ++u) gi[p * N + u] = sg[((now >> 8) & 0xFF) * tile + at + p * 32 * N + u];
                    }
                    group |= used;
#pragma unroll
                    for (int p = 0; p < BB_P; ++p)
#pragma unroll
                        for (int u = 0; u < N; ++u) {
                            const T g = sg[(now & 0xFF) * tile + at + p * 32 * N + u];
#pragma unroll
                            for (int k = 0; k < BB_OUT; ++k)
                                if (used >> k & 1u) s[k][p * N + u] += bb_coef<T>(t, k) * g;
                        }
                }
                close_used();
            } else {
            // 32 records at a time: lane i fetches record i of the next 32 while the warp works on these
            const int r1 = offs[blk + 1];
            int r = offs[blk];
            uint32_t code = 0;
            T c[BB_OUT];
            auto fetch = [&](int at_r) {
                const BbTerm &t = rec[at_r < r1 ? at_r : r1 - 1];
                code = t.code;
#pragma unroll
                for (int k = 0; k < BB_OUT; ++k) c[k] = bb_coef<T>(t, k);
            };
            if (r < r1) fetch(r + lane);
            for (; r < r1; r += 32) {
                const int n = r1 - r < 32 ? r1 - r : 32;
                __syncwarp();
                scode[warp][lane] = code;
#pragma unroll
                for (int k = 0; k < BB_OUT; ++k) scoef[warp][lane].v[k] = c[k];
                __syncwarp();
                if (r + 32 < r1) fetch(r + 32 + lane);
#pragma unroll 2
                for (int q = 0; q < n; ++q) {
                    const uint32_t now = scode[warp][q];
                    const BbCoef<T> cq = scoef[warp][q];
                    if (now & (1u << 16)) {
                        close();
#pragma unroll
                        for (int p = 0; p < BB_P; ++p) {
                            const Pack g = *reinterpret_cast<const Pack *>(sg + ((now >> 8) & 0xFF) * tile + at + p * 32 * N);
#pragma unroll
                            for (int u = 0; u < N; ++u) gi[p * N + u] = g.v[u];
                        }
                    }
#pragma unroll
                    for (int p = 0; p < BB_P; ++p) {
                        const Pack g = *reinterpret_cast<const Pack *>(sg + (now & 0xFF) * tile + at + p * 32 * N);
#pragma unroll
                        for (int k = 0; k < BB_OUT; ++k)
#pragma unroll
                            for (int u = 0; u < N; ++u) s[k][p * N + u] += cq.v[k] * g.v[u];
                    }
                }
            }
            close();
            }
#pragma unroll
            for (int k = 0; k < BB_OUT; ++k) {
                const int o = blk * BB_OUT + k;
                if (o >= n_out) break;
#pragma unroll
                for (int p = 0; p < BB_P; ++p) {
                    const int64_t x = v0 + at + p * 32 * N;
                    T *dst = out + (int64_t)o * n_vox + x;
                    if (whole) {
                        Pack w;
#pragma unroll
                        for (int u = 0; u < N; ++u) w.v[u] = acc[k][p * N + u];
                        *reinterpret_cast<Pack *>(dst) = w;
                    } else {
#pragma unroll
                        for (int u = 0; u < N; ++u)
                            if (x + u < n_vox) dst[u] = acc[k][p * N + u];
                    }
                }
            }
            if (lane == 0) unit = atomicAdd(&next, 1);
            unit = __shfl_sync(0xFFFFFFFFu, unit, 0);
        }
    }
}

template <typename T>
static int launch_blocks(const void *G, int n_g, int64_t n_vox, const int32_t *offs, const BbTerm *rec, int n_out,
                         void *out, cudaStream_t s) {
    const int span = 32 * BB_P * BbPack<T>::N, row = span * (int)sizeof(T) * n_g;
    const int fixed = BL_THREADS * (4 + (int)sizeof(BbCoef<T>));   // the warps' records
    const int vec = (n_vox * (int64_t)sizeof(T)) % 16 == 0 && (((uintptr_t)G | (uintptr_t)out) & 15) == 0;
    // BB_OCC blocks per SM (227 KB, 1 KB of it taken per block); one span of 128 maps is 128 KB, one block
    int n_span = std::min(8, ((227 * 1024 / BB_OCC - 2048) - fixed) / row);
    // and no more than leave every SM its blocks (13,824 voxels, 16 bins, l = 0, 2: 42 us with tiles as large as fit, now
    // 20 us; 4 bins 10 and 4.5 us)
    n_span = std::max(1, (int)std::min<int64_t>(n_span, (n_vox + span - 1) / span / ((int64_t)num_sms() * BB_OCC)));
    const int tile = span * n_span;
    const size_t smem = (size_t)row * n_span;
    const int blocks = (int)std::min<int64_t>((n_vox + tile - 1) / tile, (int64_t)num_sms() * BB_OCC * 16);
    PB_CUDA(cudaFuncSetAttribute(bilinear_block_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    bilinear_block_kernel<T><<<blocks, BL_THREADS, smem, s>>>((const T *)G, n_g, n_vox, offs, rec, n_out, n_span, vec,
                                                              (T *)out);
    PB_LAUNCH_CHECK("pb_bilinear_block_maps");
    return PB_OK;
}

}  // namespace pb

using namespace pb;

// table: int32 offsets[n_out + 1] (padded to 16 bytes), then the term records of output 0,
// 1, ... each sorted by (i, j) with i <= j and duplicates merged.  An output without terms
// has an empty range and is written as zeros.
extern "C" int pb_bilinear_plan(int n_g, int n_out, const int32_t *o, const int32_t *i, const int32_t *j,
                                const double *c, int n_terms, void *table, size_t *table_bytes, int32_t *n_table) {
    if (!table_bytes || !n_table || (n_terms > 0 && (!o || !i || !j || !c)))
        return fail(PB_ERR_INVALID, "pb_bilinear_plan: NULL argument");
    if (n_g < 1 || n_g > BL_MAXG || n_out < 1 || n_out > BL_MAXOUT)
        return fail(PB_ERR_INVALID, "pb_bilinear_plan: need 1..128 maps and 1..4096 outputs");
    std::vector<std::tuple<int, int, int, double>> t;
    t.reserve(n_terms);
    for (int k = 0; k < n_terms; ++k) {
        if (o[k] < 0 || o[k] >= n_out || i[k] < 0 || i[k] >= n_g || j[k] < 0 || j[k] >= n_g)
            return fail(PB_ERR_INVALID, "pb_bilinear_plan: term index out of range");
        t.emplace_back(o[k], std::min(i[k], j[k]), std::max(i[k], j[k]), c[k]);
    }
    std::sort(t.begin(), t.end(), [](const auto &a, const auto &b) {
        return std::make_tuple(std::get<0>(a), std::get<1>(a), std::get<2>(a)) <
               std::make_tuple(std::get<0>(b), std::get<1>(b), std::get<2>(b));
    });
    std::vector<std::tuple<int, int, int, double>> u;
    for (auto &e : t) {
        if (!u.empty() && std::get<0>(u.back()) == std::get<0>(e) && std::get<1>(u.back()) == std::get<1>(e) &&
            std::get<2>(u.back()) == std::get<2>(e))
            std::get<3>(u.back()) += std::get<3>(e);
        else
            u.push_back(e);
    }
    const int n = (int)u.size();
    const size_t head = ((size_t)(n_out + 1) * 4 + 15) / 16 * 16;
    *table_bytes = head + (size_t)n * sizeof(BlTerm);
    *n_table = n;
    if (!table) return PB_OK;
    int32_t *offs = (int32_t *)table;
    BlTerm *rec = (BlTerm *)((char *)table + head);
    int k = 0;
    for (int q = 0; q < n_out; ++q) {
        offs[q] = k;
        int prev_i = -1;
        while (k < n && std::get<0>(u[k]) == q) {
            const int i_k = std::get<1>(u[k]), j_k = std::get<2>(u[k]);
            rec[k].code = (uint32_t)j_k | ((uint32_t)i_k << 8) | ((uint32_t)(i_k != prev_i) << 16);
            rec[k].cf = (float)std::get<3>(u[k]);
            rec[k].c = std::get<3>(u[k]);
            prev_i = i_k;
            ++k;
        }
    }
    offs[n_out] = k;
    return PB_OK;
}

extern "C" int pb_bilinear_maps(int precision, int64_t n_vox, const void *G, int n_g, const void *table, int n_table,
                                int n_out, void *out, void *stream) {
    if (!G || !table || !out) return fail(PB_ERR_INVALID, "pb_bilinear_maps: NULL argument");
    if (n_vox < 1 || n_g < 1 || n_g > BL_MAXG) return fail(PB_ERR_INVALID, "pb_bilinear_maps: need 1..128 maps");
    if (n_out < 1 || n_out > BL_MAXOUT || n_table < 0)
        return fail(PB_ERR_INVALID, "pb_bilinear_maps: bad output or term count");
    if (((uintptr_t)table & 15) != 0) return fail(PB_ERR_INVALID, "pb_bilinear_maps: table must be 16-byte aligned");
    const bool f64 = precision == PB_F64;
    const int tile = f64 ? 32 * 4 : 32 * 8;
    const size_t smem = (size_t)n_g * tile * (f64 ? 8 : 4);
    const size_t head = ((size_t)(n_out + 1) * 4 + 15) / 16 * 16;
    const int32_t *offs = (const int32_t *)table;
    const BlTerm *rec = (const BlTerm *)((const char *)table + head);
    const int64_t tiles = (n_vox + tile - 1) / tile;
    const int blocks = (int)std::min<int64_t>(tiles, (int64_t)num_sms() * 4 * 8);
    cudaStream_t s = as_stream(stream);
    if (precision == PB_F32) {
        PB_CUDA(cudaFuncSetAttribute(bilinear_kernel<float, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        bilinear_kernel<float, 8><<<blocks, BL_THREADS, smem, s>>>((const float *)G, n_g, n_vox, offs, rec, n_out,
                                                                   (float *)out);
    } else if (precision == PB_F64) {
        PB_CUDA(cudaFuncSetAttribute(bilinear_kernel<double, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        bilinear_kernel<double, 4><<<blocks, BL_THREADS, smem, s>>>((const double *)G, n_g, n_vox, offs, rec, n_out,
                                                                    (double *)out);
    } else {
        return fail(PB_ERR_INVALID, "pb_bilinear_maps: bad precision");
    }
    PB_LAUNCH_CHECK("pb_bilinear_maps");
    return PB_OK;
}

// table: int32 offsets[ceil(n_out / 4) + 1] (padded to 16 bytes), then the records of block 0, 1, ... sorted by
// (i, j) with i <= j; slot[t] (optional, n_terms): index of term t's coefficient, 4 record + output % 4.
// Duplicate terms share a slot and add up.
extern "C" int pb_bilinear_block_plan(int n_g, int n_out, const int32_t *o, const int32_t *i, const int32_t *j,
                                      const double *c, int n_terms, void *table, size_t *table_bytes, int32_t *n_table,
                                      int32_t *slot) {
    if (!table_bytes || !n_table || (n_terms > 0 && (!o || !i || !j || !c)))
        return fail(PB_ERR_INVALID, "pb_bilinear_block_plan: NULL argument");
    if (n_g < 1 || n_g > BL_MAXG || n_out < 1 || n_out > BL_MAXOUT)
        return fail(PB_ERR_INVALID, "pb_bilinear_block_plan: need 1..128 maps and 1..4096 outputs");
    std::vector<std::pair<uint32_t, int>> t(n_terms);  // (block, i, j) and the term
    for (int k = 0; k < n_terms; ++k) {
        if (o[k] < 0 || o[k] >= n_out || i[k] < 0 || i[k] >= n_g || j[k] < 0 || j[k] >= n_g)
            return fail(PB_ERR_INVALID, "pb_bilinear_block_plan: term index out of range");
        const uint32_t a = std::min(i[k], j[k]), b = std::max(i[k], j[k]);
        t[k] = {(uint32_t)(o[k] / BB_OUT) << 16 | a << 8 | b, k};
    }
    std::sort(t.begin(), t.end());
    int n = 0;
    for (int k = 0; k < n_terms; ++k) n += k == 0 || t[k].first != t[k - 1].first;
    const int n_blk = (n_out + BB_OUT - 1) / BB_OUT;
    const size_t head = ((size_t)(n_blk + 1) * 4 + 15) / 16 * 16;
    const size_t need = head + (size_t)n * sizeof(BbTerm);
    *n_table = n;
    if (!table) {
        *table_bytes = need;
        return PB_OK;
    }
    if (*table_bytes < need) return fail(PB_ERR_INVALID, "pb_bilinear_block_plan: table buffer too small");
    *table_bytes = need;
    memset(table, 0, need);
    int32_t *offs = (int32_t *)table;
    BbTerm *rec = (BbTerm *)((char *)table + head);
    int r = -1;
    for (int k = 0; k < n_terms; ++k) {
        const uint32_t key = t[k].first;
        if (k == 0 || key != t[k - 1].first) {
            ++r;
            const bool first = k == 0 || (key >> 8) != (t[k - 1].first >> 8);
            rec[r].code = (key & 0xFFFF) | (first ? 1u << 16 : 0u);
            ++offs[(key >> 16) + 1];
        }
        const int q = o[t[k].second] % BB_OUT;
        rec[r].code |= 1u << (17 + q);
        rec[r].c[q] += c[t[k].second];
        if (slot) slot[t[k].second] = BB_OUT * r + q;
    }
    for (int k = 0; k < n; ++k)
        for (int q = 0; q < BB_OUT; ++q) rec[k].cf[q] = (float)rec[k].c[q];
    for (int b = 0; b < n_blk; ++b) offs[b + 1] += offs[b];
    return PB_OK;
}

extern "C" int pb_bilinear_block_maps(int precision, int64_t n_vox, const void *G, int n_g, const void *table,
                                      int n_table, int n_out, void *out, void *stream) {
    if (!G || !table || !out) return fail(PB_ERR_INVALID, "pb_bilinear_block_maps: NULL argument");
    if (n_vox < 1 || n_g < 1 || n_g > BL_MAXG) return fail(PB_ERR_INVALID, "pb_bilinear_block_maps: need 1..128 maps");
    if (n_out < 1 || n_out > BL_MAXOUT || n_table < 0)
        return fail(PB_ERR_INVALID, "pb_bilinear_block_maps: bad output or term count");
    if (((uintptr_t)table & 15) != 0) return fail(PB_ERR_INVALID, "pb_bilinear_block_maps: table must be 16-byte aligned");
    if (precision != PB_F32 && precision != PB_F64) return fail(PB_ERR_INVALID, "pb_bilinear_block_maps: bad precision");
    const size_t head = ((size_t)((n_out + BB_OUT - 1) / BB_OUT + 1) * 4 + 15) / 16 * 16;
    const int32_t *offs = (const int32_t *)table;
    const BbTerm *rec = (const BbTerm *)((const char *)table + head);
    return precision == PB_F64 ? launch_blocks<double>(G, n_g, n_vox, offs, rec, n_out, out, as_stream(stream))
                               : launch_blocks<float>(G, n_g, n_vox, offs, rec, n_out, out, as_stream(stream));
}
