// CUDA-core kernels for the three stages of the block, templated on the storage type.
//
// T = float is the fp32 path (IEEE fp32 FMA throughout, no TF32, expf-based sigmoid): it has to
// meet a 1e-5 relative tolerance against the fp32 reference, which rules the tensor cores out.
// T = __nv_bfloat16 uses the same layouts and the same bf16 rounding points as the tensor-core
// kernels (x_n, a, b, tri, tri_n, out) with fp32 arithmetic in between; it serves channel widths
// the tensor-core kernels do not cover and is the stage-by-stage cross-check for them.
//
// All three read/write the channel-major operand planes through PlaneView, which implements the
// chunked addressing of trimul_planes, so they work on gathered multi-GPU operands unchanged.
//
// What bounds them: FP32 FMA issue (148 SMs x 128 lanes, 74 TFLOP/s at 1.965 GHz).  So each stage is a
// register-tiled matrix product: 256 threads, both operands K-major in shared memory as [k][position] and
// [k][column].  A thread owns TM positions x 8 columns in stage 1 (four of a projection, four of its gate), TM x TM outputs in
// the contraction and TM positions x 4 columns in stage 3 (of the gate, then of the projection): one K step at TM = 8
// costs four 16-byte shared-memory reads per 64 FMAs in stages 1 and 2, three per 32 in stage 3, which is why that
// stage's load/store pipe is the busiest.  Eight lanes of a warp walk positions and four walk columns, so a
// position fragment of a warp is one 128-byte wavefront.  Every output is still ONE fma chain over ascending k: the rounding of the products
// is what a plain dot product gives; the FMAs are the packed two-lane form.
// Measured (fp32, B = 1, N = 256, c = 128; before: one output channel per thread, 8 positions, weights read
// from global memory with a stride of c): stage 1 2215 -> 302 us, contraction 646 -> 143, stage 3 1206 -> 193,
// the block 4080 -> 618; N = 32: 102 -> 39 us.  Counters of the three kernels now: FMA pipe 41-52 %, the
// load/store data pipe 53-68 % (weight and position fragments, and the turns to [k][..]).
#pragma once

#include "ptx_sm100.cuh"

namespace trimul {

struct PlaneView {
    void* base;
    long long rows, cols, pitch, plane_stride, chunk_stride, row_chunk, col_chunk;
    // p: plane, r: row, q: column; rows and columns fit 32 bits, and a chunk is no longer than its extent
    __device__ __forceinline__ long long offset(long long p, int r, int q) const {
        if (row_chunk >= rows && col_chunk >= cols) return p * plane_stride + r * pitch + q;
        const unsigned rc = (unsigned)row_chunk, cc = (unsigned)col_chunk;
        const unsigned chunk = (unsigned)r / rc + (unsigned)q / cc;   // at most one of the two is non-zero
        return chunk * chunk_stride + p * plane_stride + ((unsigned)r % rc) * pitch + ((unsigned)q % cc);
    }
    // four consecutive columns starting at a multiple of four are adjacent and 4-element aligned in memory
    __device__ __forceinline__ bool quads() const { return col_chunk >= cols || (col_chunk & 3) == 0; }
};

template <typename T> __device__ __forceinline__ float load_f(const T* p);
template <> __device__ __forceinline__ float load_f<float>(const float* p) { return *p; }
template <> __device__ __forceinline__ float load_f<__nv_bfloat16>(const __nv_bfloat16* p) {
    return __bfloat162float(*p);
}
// four consecutive elements at a 4-element aligned address
__device__ __forceinline__ float4 load_f4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load_f4(const __nv_bfloat16* p) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    return make_float4(bf16_lo(v.x), bf16_hi(v.x), bf16_lo(v.y), bf16_hi(v.y));
}
__device__ __forceinline__ void store_f4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void store_f4(__nv_bfloat16* p, float4 v) {
    *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
}
template <typename T> __device__ __forceinline__ T store_t(float v);
template <> __device__ __forceinline__ float store_t<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 store_t<__nv_bfloat16>(float v) {
    return __float2bfloat16_rn(v);
}
// value as it would be after a round trip through storage type T
template <typename T> __device__ __forceinline__ float round_t(float v);
template <> __device__ __forceinline__ float round_t<float>(float v) { return v; }
template <> __device__ __forceinline__ float round_t<__nv_bfloat16>(float v) {
    return __bfloat162float(__float2bfloat16_rn(v));
}

__device__ __forceinline__ float sigmoid_ref(float x) { return 1.0f / (1.0f + expf(-x)); }

constexpr int kPlainThreads = 256;
constexpr int kPlainMaxC = 256;
constexpr int kPlainKC = 32;            // K slice of the weights in shared memory (two slices, double-buffered)
constexpr int kPlainCh = 64;            // output channels per block (two columns each: proj and gate, or gate and out)

// positions per block and row pitch (floats) of its [k][position] tile; the pitch is 4 mod 32, so that eight
// lanes storing 16 bytes to consecutive k hit all 32 banks
template <int TM> struct PlainTile {
    static constexpr int kPos = 16 * TM;
    static constexpr int kPitch = kPos + 4;
};
constexpr int kPlainWPitch = 2 * kPlainCh + 4;
template <int TM> constexpr int plain_tm1_smem(int c) {
    return ((c > kPlainCh ? c : kPlainCh) * PlainTile<TM>::kPitch + 2 * kPlainKC * kPlainWPitch) * 4;
}
template <int TM> constexpr int plain_tm2_smem(int c, int h) {
    return ((c > h ? c : h) * PlainTile<TM>::kPitch + 2 * kPlainKC * (kPlainCh + 4)) * 4;
}

// a thread's place in the 16 x 16 arrangement: tx walks positions, ty columns
__device__ __forceinline__ void plain_thread_xy(int& tx, int& ty) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    tx = (warp & 1) * 8 + (lane & 7);
    ty = (warp >> 1) * 4 + (lane >> 3);
}
// index inside the tile of a thread's i-th position
template <int TM> __device__ __forceinline__ int plain_pos(int tx, int i) {
    return TM == 8 ? (i >> 2) * 64 + tx * 4 + (i & 3) : tx * TM + i;
}
// a thread's positions of one K row, as fp32 pairs
template <int TM> __device__ __forceinline__ void plain_frag(f32x2 (&x)[TM / 2], const float* row, int tx) {
    if constexpr (TM >= 4) {
#pragma unroll
        for (int v = 0; v < TM / 4; ++v) {
            const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(row + v * 64 + tx * 4);
            x[2 * v] = t.x; x[2 * v + 1] = t.y;
        }
    } else {
        x[0] = *reinterpret_cast<const f32x2*>(row + tx * 2);
    }
}
// acc[i][j] += x pair i * w[j], both lanes
template <int TM, int NJ>
__device__ __forceinline__ void plain_fma4(f32x2 (&acc)[TM / 2][NJ], int j0, const f32x2 (&x)[TM / 2], const float4 w) {
    const f32x2 w2[4] = {f2_pack(w.x, w.x), f2_pack(w.y, w.y), f2_pack(w.z, w.z), f2_pack(w.w, w.w)};
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < TM / 2; ++i) acc[i][j0 + j] = f2_fma(w2[j], x[i], acc[i][j0 + j]);
}
template <int TM, int NJ> __device__ __forceinline__ float plain_acc(const f32x2 (&acc)[TM / 2][NJ], int i, int j) {
    float lo, hi;
    f2_unpack(acc[i / 2][j], lo, hi);
    return (i & 1) ? hi : lo;
}

// LayerNorm of a tile of positions, from global memory into xs[channel][position].  A warp takes four positions
// at a time: coalesced reads along the channels, the sums by shuffles, and the four normalised values
// of a channel stored as 16 bytes.  NC = ceil of c / 32 this instance is for (4 or 8); src(first, x) fills the
// addresses of four consecutive positions' channels, null past the end.
template <typename T, int TM, int NC, typename Src>
__device__ __forceinline__ void plain_layernorm_tile_n(float* xs, int c, const float* gamma, const float* beta, float eps,
                                                     Src src) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int g = warp; g < PlainTile<TM>::kPos / 4; g += kPlainThreads / 32) {
        float v[4][NC];
        const T* rows[4];
        src(4 * g, rows);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const T* x = rows[q];
#pragma unroll
            for (int i = 0; i < NC; ++i)
                v[q][i] = (x != nullptr && lane + 32 * i < c) ? load_f<T>(x + lane + 32 * i) : 0.f;
        }
        float mean[4], rstd[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            float s = 0.f;
#pragma unroll
            for (int i = 0; i < NC; ++i) s += v[q][i];
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            mean[q] = s / (float)c;
            float t = 0.f;
#pragma unroll
            for (int i = 0; i < NC; ++i)
                if (lane + 32 * i < c) {
                    const float d = v[q][i] - mean[q];
                    t = fmaf(d, d, t);
                }
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            rstd[q] = 1.0f / sqrtf(t / (float)c + eps);
        }
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            const int ch = lane + 32 * i;
            if (ch < c) {
                const float ga = gamma[ch], be = beta[ch];
                float y[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) y[q] = round_t<T>((v[q][i] - mean[q]) * rstd[q] * ga + be);
                *reinterpret_cast<float4*>(xs + ch * PlainTile<TM>::kPitch + 4 * g) = make_float4(y[0], y[1], y[2], y[3]);
            }
        }
    }
}

template <typename T, int TM, typename Src>
__device__ __forceinline__ void plain_layernorm_tile(float* xs, int c, const float* gamma, const float* beta, float eps,
                                                     Src src) {
    if (c <= 128) plain_layernorm_tile_n<T, TM, 4>(xs, c, gamma, beta, eps, src);
    else plain_layernorm_tile_n<T, TM, kPlainMaxC / 32>(xs, c, gamma, beta, eps, src);
}

// A K slice of the weights on its way from global memory to ws[k][column]: thread = one column (a weight row) and
// kQuads groups of four k.  kCols columns; row(col) -> that column's weight row, or null.
template <typename T, int kCols> struct PlainWeights {
    static constexpr int kQuads = kPlainKC * kCols / (4 * kPlainThreads);
    const T* row;
    int col, kq;
    float4 r[kQuads];
    template <typename Row> __device__ __forceinline__ void init(Row rowof) {
        col = threadIdx.x % kCols;
        kq = threadIdx.x / kCols * (4 * kQuads);
        row = rowof(col);
    }
    __device__ __forceinline__ void fetch(int k0, int K) {
#pragma unroll
        for (int i = 0; i < kQuads; ++i)      // K is a multiple of 8: a quad is whole or absent
            r[i] = row != nullptr && k0 + kq + 4 * i < K ? load_f4(row + k0 + kq + 4 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __device__ __forceinline__ void put(float* ws) const {
#pragma unroll
        for (int i = 0; i < kQuads; ++i) {
            float* p = ws + (kq + 4 * i) * (kCols + 4) + col;
            p[0] = r[i].x; p[kCols + 4] = r[i].y; p[2 * (kCols + 4)] = r[i].z; p[3 * (kCols + 4)] = r[i].w;
        }
    }
};

// acc[i][j] += sum_k xs[k][position i] * W[column j][k]; kCols = 128: a thread's columns are 4 ty + j of the first
// 64 and of the second 64, kCols = 64: 4 ty + j.  All threads of the block take part.
template <typename T, int TM, int kCols, typename Row>
__device__ __forceinline__ void plain_product(f32x2 (&acc)[TM / 2][kCols / 16], const float* xs, float* ws, int K, int tx, int ty,
                                              Row rowof) {
    constexpr int kWP = kCols + 4;
    PlainWeights<T, kCols> w;
    w.init(rowof);
    w.fetch(0, K);
    w.put(ws);
    __syncthreads();                      // also publishes the caller's xs
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += kPlainKC, buf ^= 1) {
        const bool more = k0 + kPlainKC < K;
        if (more) w.fetch(k0 + kPlainKC, K);
        const float* xk = xs + k0 * PlainTile<TM>::kPitch;
        const float* wk = ws + buf * kPlainKC * kWP + ty * 4;
        const int kn = min(kPlainKC, K - k0);
        for (int k8 = 0; k8 < kn; k8 += 8) {
#pragma unroll
            for (int kk = 0; kk < 8; ++kk) {
                f32x2 x[TM / 2];
                plain_frag<TM>(x, xk + (k8 + kk) * PlainTile<TM>::kPitch, tx);
#pragma unroll
                for (int v = 0; v < kCols / 64; ++v)
                    plain_fma4<TM>(acc, 4 * v, x, *reinterpret_cast<const float4*>(wk + (k8 + kk) * kWP + v * 64));
            }
        }
        if (more) w.put(ws + (buf ^ 1) * kPlainKC * kWP);
        __syncthreads();
    }
}

struct PlainTm1Params {
    int B, rows, N, c, row0, incoming, mask_kind;
    int h;      // planes per batch element = rows of the four [h, c] projection matrices
    const uint8_t* mask;
    const float *gamma, *beta;
    float eps;
    const void *w_left, *w_left_gate, *w_right, *w_right_gate;
    PlaneView a, b;
};

// Positions are walked in the order of the OPERAND PLANES (outgoing: z row, then column; incoming: z column, then
// row), 16 TM consecutive ones per block whatever the row length, so no tile has padding but the very last
// and a plane row is written contiguously in both directions.  blockIdx.y = side * ceil(h / 64) + channel group.
template <typename T, int TM>
__global__ void __launch_bounds__(kPlainThreads, 2) plain_tm1_kernel(const T* __restrict__ z, PlainTm1Params p) {
    constexpr int kPos = PlainTile<TM>::kPos, kPitch = PlainTile<TM>::kPitch;
    extern __shared__ __align__(16) float psm[];
    __shared__ float keep[kPos];
    float* xs = psm;
    float* ws = psm + max(p.c, kPlainCh) * kPitch;
    griddep_wait();
    griddep_launch_dependents();
    const int c = p.c, groups = (p.h + kPlainCh - 1) / kPlainCh;
    const int side = (int)blockIdx.y / groups, ch0 = ((int)blockIdx.y % groups) * kPlainCh;
    const int n_run = p.incoming ? p.rows : p.N, n_fixed = p.incoming ? p.N : p.rows;
    const long long first = (long long)blockIdx.x * kPos, total = (long long)p.B * p.rows * p.N;
    const int npos = (int)min((long long)kPos, total - first);
    const int f0 = (int)(first / n_run), t0 = (int)(first % n_run);
    auto place = [&](int pos, int& b, int& f, int& t) {
        const unsigned u = (unsigned)(t0 + pos);
        const unsigned fb = (unsigned)f0 + u / (unsigned)n_run;
        t = (int)(u % (unsigned)n_run);
        b = (int)(fb / (unsigned)n_fixed);
        f = (int)(fb % (unsigned)n_fixed);
    };
    plain_layernorm_tile<T, TM>(xs, c, p.gamma, p.beta, p.eps, [&](int pos, const T* (&x)[4]) {
        int b, f, t;
        place(pos, b, f, t);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            x[q] = pos + q < npos
                ? z + (((long long)b * p.rows + (p.incoming ? t : f)) * p.N + (p.incoming ? f : t)) * c : nullptr;
            if (++t == n_run) {
                t = 0;
                if (++f == n_fixed) { f = 0; ++b; }
            }
        }
    });
    if (threadIdx.x < npos) {
        float k = 1.f;
        if (p.mask_kind != 0) {
            int b, f, t;
            place(threadIdx.x, b, f, t);
            const long long zr = p.row0 + (p.incoming ? t : f), zc = p.incoming ? f : t, mb = (long long)b * p.N;
            k = (p.mask_kind == 1 ? (p.mask[mb + zr] != 0 && p.mask[mb + zc] != 0) : p.mask[(mb + zr) * p.N + zc] != 0)
                    ? 1.f : 0.f;
        }
        keep[threadIdx.x] = k;
    }
    int tx, ty;
    plain_thread_xy(tx, ty);
    f32x2 acc[TM / 2][8];
#pragma unroll
    for (int i = 0; i < TM / 2; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;      // the pair (+0.f, +0.f)
    const T* wp = static_cast<const T*>(side == 0 ? p.w_left : p.w_right);
    const T* wg = static_cast<const T*>(side == 0 ? p.w_left_gate : p.w_right_gate);
    plain_product<T, TM, 2 * kPlainCh>(acc, xs, ws, c, tx, ty, [&](int col) -> const T* {
        const int o = ch0 + (col & (kPlainCh - 1));
        return o < p.h ? (col < kPlainCh ? wp : wg) + (long long)o * c : nullptr;
    });
    // gate in registers, then through shared memory (the dead x tile) so that a warp writes runs of 32 positions
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int pos = plain_pos<TM>(tx, i);
            xs[(ty * 4 + j) * kPitch + pos] = pos < npos ? plain_acc<TM>(acc, i, j) * sigmoid_ref(plain_acc<TM>(acc, i, 4 + j)) * keep[pos] : 0.f;
        }
    __syncthreads();
    const PlaneView& v = side == 0 ? p.a : p.b;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < kPos / 32; ++i) {
        const int pos = i * 32 + lane;
        if (pos >= npos) break;
        int b, f, t;
        place(pos, b, f, t);
        T* dst = static_cast<T*>(v.base) + v.offset((long long)b * p.h + ch0 + warp * 8, f, t);
        for (int k = 0; k < 8 && ch0 + warp * 8 + k < p.h; ++k)
            dst[k * v.plane_stride] = store_t<T>(xs[(warp * 8 + k) * kPitch + pos]);
    }
}

// tri[p][i][j] = sum_k a[p][i][k] * b[p][j][k].  grid (ceil(rows_b / BT), ceil(rows_a / BT), planes), BT = 16 TM;
// a thread owns TM rows x TM columns, K goes through shared memory 16 at a time, double-buffered, turned into
// [k][row] on the way.
constexpr int kPlainCtK = 16;
template <typename T, int TM>
__global__ void __launch_bounds__(kPlainThreads, 2) plain_contract_kernel(PlaneView a, PlaneView b, PlaneView d) {
    constexpr int BT = PlainTile<TM>::kPos, kPitch = PlainTile<TM>::kPitch;
    constexpr int kPer = kPlainCtK * BT / kPlainThreads;      // k per thread and operand: 8 (128 rows) or 4 (64 rows)
    __shared__ __align__(16) float sa[2][kPlainCtK * kPitch], sb[2][kPlainCtK * kPitch];
    griddep_wait();
    griddep_launch_dependents();
    const long long plane = blockIdx.z;
    const int i0 = blockIdx.y * BT, j0 = blockIdx.x * BT, K = (int)a.cols;
    int tx, ty;
    plain_thread_xy(tx, ty);
    const int row = threadIdx.x % BT, kq = threadIdx.x / BT * kPer;
    const bool quads_a = a.quads(), quads_b = b.quads();
    float4 ra[kPer / 4], rb[kPer / 4];
    auto fetch4 = [&](const PlaneView& v, bool quads, int r, int k) -> float4 {
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r >= v.rows || k >= K) return x;
        const T* base = static_cast<const T*>(v.base);
        if (quads && k + 3 < K) {
            x = load_f4(base + v.offset(plane, r, k));
        } else {                      // nothing past the last column is read: the caller's memory may end there
            x.x = load_f<T>(base + v.offset(plane, r, k));
            if (k + 1 < K) x.y = load_f<T>(base + v.offset(plane, r, k + 1));
            if (k + 2 < K) x.z = load_f<T>(base + v.offset(plane, r, k + 2));
            if (k + 3 < K) x.w = load_f<T>(base + v.offset(plane, r, k + 3));
        }
        return x;
    };
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < kPer / 4; ++i) {
            ra[i] = fetch4(a, quads_a, i0 + row, k0 + kq + 4 * i);
            rb[i] = fetch4(b, quads_b, j0 + row, k0 + kq + 4 * i);
        }
    };
    auto put = [&](int buf) {
#pragma unroll
        for (int i = 0; i < kPer / 4; ++i) {
            float* pa = &sa[buf][(kq + 4 * i) * kPitch + row];
            float* pb = &sb[buf][(kq + 4 * i) * kPitch + row];
            pa[0] = ra[i].x; pa[kPitch] = ra[i].y; pa[2 * kPitch] = ra[i].z; pa[3 * kPitch] = ra[i].w;
            pb[0] = rb[i].x; pb[kPitch] = rb[i].y; pb[2 * kPitch] = rb[i].z; pb[3 * kPitch] = rb[i].w;
        }
    };
    f32x2 acc[TM / 2][TM];      // [pair of rows of b][row of a]
#pragma unroll
    for (int i = 0; i < TM / 2; ++i)
#pragma unroll
        for (int j = 0; j < TM; ++j) acc[i][j] = 0ull;
    fetch(0);
    put(0);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += kPlainCtK, buf ^= 1) {
        const bool more = k0 + kPlainCtK < K;
        if (more) fetch(k0 + kPlainCtK);
#pragma unroll
        for (int kk = 0; kk < kPlainCtK; ++kk) {       // k past the end: both operands are zero
            f32x2 x[TM / 2];
            plain_frag<TM>(x, &sb[buf][kk * kPitch], tx);
#pragma unroll
            for (int v = 0; v < TM / 4; ++v)
                plain_fma4<TM>(acc, 4 * v, x, *reinterpret_cast<const float4*>(&sa[buf][kk * kPitch + v * 64 + ty * 4]));
        }
        if (more) put(buf ^ 1);
        __syncthreads();
    }
    const bool quads_d = d.quads();
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int r = i0 + plain_pos<TM>(ty, i);
        if (r >= d.rows) continue;
#pragma unroll
        for (int v = 0; v < TM / 4; ++v) {
            const int j = j0 + v * 64 + tx * 4;
            float y[4];
            f2_unpack(acc[2 * v][i], y[0], y[1]);
            f2_unpack(acc[2 * v + 1][i], y[2], y[3]);
            T* base = static_cast<T*>(d.base);
            if (quads_d && j + 3 < d.cols) {
                store_f4(base + d.offset(plane, r, j), make_float4(y[0], y[1], y[2], y[3]));
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (j + e < d.cols) base[d.offset(plane, r, j + e)] = store_t<T>(y[e]);
            }
        }
    }
}

struct PlainTm2Params {
    int B, rows, N, c;
    int h;      // channels of tri / LayerNorm_out / in_features of w_out (c, or 2c for the bidirectional block)
    const float *gamma_in, *beta_in, *gamma_out, *beta_out;
    float eps_in, eps_out;
    const void *w_gate, *w_out;
    PlaneView tri;
    const void* drop_scale;   // [B, 1, N, c] row-broadcast multiplier of the block output, or null
};

// 16 TM consecutive positions of z per block, 64 output channels (blockIdx.y).  The z tile is normalised and
// multiplied first, then the tri tile (already [channel][position] in memory) takes its place in shared memory.
template <typename T, int TM>
__global__ void __launch_bounds__(kPlainThreads, 2)
plain_tm2_kernel(const T* __restrict__ z, T* __restrict__ out, const T* __restrict__ residual, PlainTm2Params p) {
    constexpr int kPos = PlainTile<TM>::kPos, kPitch = PlainTile<TM>::kPitch, kParts = kPlainThreads / kPos;
    extern __shared__ __align__(16) float psm[];
    __shared__ float red[2][kParts][kPos];
    const int c = p.c, h = p.h;
    float* xs = psm;
    float* ws = psm + max(c, h) * kPitch;
    griddep_wait();
    griddep_launch_dependents();
    const int o0 = blockIdx.y * kPlainCh;
    const long long first = (long long)blockIdx.x * kPos, total = (long long)p.B * p.rows * p.N;
    const int npos = (int)min((long long)kPos, total - first);
    const int f0 = (int)(first / p.N), t0 = (int)(first % p.N);
    auto place = [&](int pos, int& b, int& r, int& s) {
        const unsigned u = (unsigned)(t0 + pos);
        const unsigned br = (unsigned)f0 + u / (unsigned)p.N;
        s = (int)(u % (unsigned)p.N);
        b = (int)(br / (unsigned)p.rows);
        r = (int)(br % (unsigned)p.rows);
    };
    int tx, ty;
    plain_thread_xy(tx, ty);
    f32x2 g[TM / 2][4], v[TM / 2][4];
#pragma unroll
    for (int i = 0; i < TM / 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) g[i][j] = v[i][j] = 0ull;
    plain_layernorm_tile<T, TM>(xs, c, p.gamma_in, p.beta_in, p.eps_in,
                                [&](int pos, const T* (&x)[4]) {
#pragma unroll
                                    for (int q = 0; q < 4; ++q) x[q] = pos + q < npos ? z + (first + pos + q) * c : nullptr;
                                });
    plain_product<T, TM, kPlainCh>(g, xs, ws, c, tx, ty, [&](int col) -> const T* {
        return o0 + col < c ? static_cast<const T*>(p.w_gate) + (long long)(o0 + col) * c : nullptr;
    });
    {
        // tri tile: thread = one position and every kParts-th channel; the position's sums meet in `red`
        const int pos = threadIdx.x % kPos, part = threadIdx.x / kPos;
        float* col = xs + pos;
        float s[4] = {0.f, 0.f, 0.f, 0.f};
        const T* src = nullptr;
        if (pos < npos) {
            int b, r, q;
            place(pos, b, r, q);
            src = static_cast<const T*>(p.tri.base) + p.tri.offset((long long)b * h, r, q);
        }
        for (int k0 = part; k0 < h; k0 += 4 * kParts) {
            float x[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int ch = k0 + e * kParts;
                x[e] = src != nullptr && ch < h ? load_f<T>(src + ch * p.tri.plane_stride) : 0.f;
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (k0 + e * kParts < h) col[(k0 + e * kParts) * kPitch] = x[e];
                s[e] += x[e];
            }
        }
        red[0][part][pos] = (s[0] + s[1]) + (s[2] + s[3]);
        __syncthreads();
        float mean = 0.f;
#pragma unroll
        for (int k = 0; k < kParts; ++k) mean += red[0][k][pos];
        mean /= (float)h;
        float q2[4] = {0.f, 0.f, 0.f, 0.f};
        for (int k0 = part; k0 < h; k0 += 4 * kParts)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (k0 + e * kParts < h) {
                    const float d = col[(k0 + e * kParts) * kPitch] - mean;
                    q2[e] = fmaf(d, d, q2[e]);
                }
        red[1][part][pos] = (q2[0] + q2[1]) + (q2[2] + q2[3]);
        __syncthreads();
        float var = 0.f;
#pragma unroll
        for (int k = 0; k < kParts; ++k) var += red[1][k][pos];
        const float rstd = 1.0f / sqrtf(var / (float)h + p.eps_out);
#pragma unroll 4
        for (int ch = part; ch < h; ch += kParts)
            col[ch * kPitch] = round_t<T>((col[ch * kPitch] - mean) * rstd * p.gamma_out[ch] + p.beta_out[ch]);
    }
    plain_product<T, TM, kPlainCh>(v, xs, ws, h, tx, ty, [&](int col) -> const T* {
        return o0 + col < c ? static_cast<const T*>(p.w_out) + (long long)(o0 + col) * h : nullptr;
    });
    const int o = o0 + ty * 4;
    if (o >= c) return;         // c is a multiple of 8: four channels are whole or absent
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int pos = plain_pos<TM>(tx, i);
        if (pos >= npos) continue;
        float y[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) y[j] = sigmoid_ref(plain_acc<TM>(g, i, j)) * plain_acc<TM>(v, i, j);
        if (p.drop_scale != nullptr) {   // applied to the rounded block output, as out * scale would
            int b, r, s;
            place(pos, b, r, s);
            const float4 ds = load_f4(static_cast<const T*>(p.drop_scale) + ((long long)b * p.N + s) * c + o);
            y[0] = round_t<T>(y[0]) * ds.x; y[1] = round_t<T>(y[1]) * ds.y;
            y[2] = round_t<T>(y[2]) * ds.z; y[3] = round_t<T>(y[3]) * ds.w;
        }
        if (residual != nullptr) {
            const float4 rs = load_f4(residual + (first + pos) * c + o);
            y[0] = round_t<T>(y[0]) + rs.x; y[1] = round_t<T>(y[1]) + rs.y;
            y[2] = round_t<T>(y[2]) + rs.z; y[3] = round_t<T>(y[3]) + rs.w;
        }
        store_f4(out + (first + pos) * c + o, make_float4(y[0], y[1], y[2], y[3]));
    }
}

}  // namespace trimul
