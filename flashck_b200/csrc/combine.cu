// Split-KV combine: O = sum_s w_s * O_s / sum_s w_s with w_s = exp(LSE_s - max_s LSE_s);
// LSE = max + log(sum).  The default strides are those of the reference's combine arguments
// (attention_kernels/fmha_fwd_split_kv_combine/fmha_fwd_split_kv_combine_jinja.h:125-140): lse_acc
// [bs,hq,S,rows], o_acc [bs,hq,S,rows,dv].  The strided form also reads partials gathered from several GPUs
// ([rank][...] layouts) and can leave the result in fp32, which is what a rank contributes to such a gather.
// The partials in use are read once: from half a megabyte (one token of 32 heads, 32 splits) to some 10-30 MB (9888 rows of
// dv 128 with 2-6 splits), mostly out of L2.  What bounds the kernel is its chain of memory round trips.  Three forms (launch_t picks):
// two (batch, head, row) rows per warp for at most 16 splits and 128 columns (combine_pair_kernel), several warps per row for rows
// with many splits as long as all rows together stay within 16 warps per SM (combine_wide_kernel), one warp per row for the rest.
#include "kernels.h"

namespace fck {

namespace {

template <typename T> struct Out4;
template <> struct Out4<__half> {
    static __device__ __forceinline__ void store(__half* p, float4 v) {
        uint2 pk = make_uint2(Elem<__half>::pack2(v.x, v.y), Elem<__half>::pack2(v.z, v.w));
        *reinterpret_cast<uint2*>(p) = pk;
    }
};
template <> struct Out4<__nv_bfloat16> {
    static __device__ __forceinline__ void store(__nv_bfloat16* p, float4 v) {
        uint2 pk = make_uint2(Elem<__nv_bfloat16>::pack2(v.x, v.y), Elem<__nv_bfloat16>::pack2(v.z, v.w));
        *reinterpret_cast<uint2*>(p) = pk;
    }
};
template <> struct Out4<float> {
    static __device__ __forceinline__ void store(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
};

struct CombineDev {
    const float* lse_acc;
    const float* o_acc;
    void* o;
    float* lse;
    int64_t items;
    int rows, hq, dv, S;
    int64_t lb, lh, ls, lr;  // lse_acc strides: batch, head, split, row
    int64_t ob, oh, os, orr; // o_acc strides (elements): batch, head, split, row
};

template <typename T>
__global__ void __launch_bounds__(128) combine_kernel(const CombineDev p) {
    pdl_wait();  // the split kernel's partials are complete and visible (no-op after an ordinary launch)
    const int lane = threadIdx.x & 31;
    const int64_t item = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (item >= p.items) return;
    // item = (b*hq + h)*rows + r
    const int r = (int)(item % p.rows);
    const int64_t bh = item / p.rows;
    const int h = (int)(bh % p.hq);
    const int64_t b = bh / p.hq;
    const int S = p.S;
    const float* lrow = p.lse_acc + b * p.lb + h * p.lh + r * p.lr;
    const float ninf = -INFINITY;

    float m = ninf;
    for (int s = lane; s < S; s += 32) m = fmaxf(m, lrow[s * p.ls]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));

    T* orow = (T*)p.o + ((b * p.rows + r) * p.hq + h) * (int64_t)p.dv;
    const int nvec = p.dv >> 2;  // float4 chunks
    if (m == ninf) {             // no split saw a key: O = 0, LSE = -inf
        for (int c = lane; c < nvec; c += 32) Out4<T>::store(orow + 4 * c, make_float4(0.f, 0.f, 0.f, 0.f));
        if (p.lse && lane == 0) p.lse[item] = ninf;
        return;
    }
    float sum = 0.f;
    for (int s = lane; s < S; s += 32) {
        const float ls = lrow[s * p.ls];
        sum += (ls == ninf) ? 0.f : expf(ls - m);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    const float inv = 1.f / sum;

    float4 acc[2];
    acc[0] = make_float4(0.f, 0.f, 0.f, 0.f);
    acc[1] = acc[0];
    const float* obase = p.o_acc + b * p.ob + h * p.oh + r * p.orr;
    const bool c0 = lane < nvec, c1 = lane + 32 < nvec;
    // Lane s of a group of 32 splits holds that split's weight, so the row loop below has no load on its way to the
    // next address: four splits' rows are fetched together.  A weight of zero marks an empty split (LSE = -inf),
    // whose o_acc slot is never read -- it may hold anything.
    for (int s0 = 0; s0 < S; s0 += 32) {
        float wl = 0.f;
        if (s0 + lane < S) {
            const float ls = lrow[(s0 + lane) * p.ls];
            wl = (ls == ninf) ? 0.f : expf(ls - m) * inv;
        }
        const int cnt = min(32, S - s0);
        for (int j0 = 0; j0 < cnt; j0 += 4) {
            float w[4];
            float4 x[4][2];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                w[u] = __shfl_sync(0xffffffffu, wl, (j0 + u) & 31);
                if (j0 + u >= cnt) w[u] = 0.f;
                const float4* src = reinterpret_cast<const float4*>(obase + (int64_t)(s0 + j0 + u) * p.os);
                x[u][0] = (w[u] != 0.f && c0) ? src[lane] : make_float4(0.f, 0.f, 0.f, 0.f);
                x[u][1] = (w[u] != 0.f && c1) ? src[lane + 32] : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    acc[j].x += w[u] * x[u][j].x;
                    acc[j].y += w[u] * x[u][j].y;
                    acc[j].z += w[u] * x[u][j].z;
                    acc[j].w += w[u] * x[u][j].w;
                }
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int c = lane + 32 * j;
        if (c < nvec) Out4<T>::store(orow + 4 * c, acc[j]);
    }
    if (p.lse && lane == 0) p.lse[item] = m + logf(sum);
}

// Two rows per warp, for at most 16 splits and 128 columns (most merges: many rows of a few splits): half a warp holds a row's LSEs,
// one a lane, so that maximum, sum and weights need no second look at memory, and its 16 lanes take two float4 of every partial
// row.  The first kFirst splits' rows are requested before the LSEs have come (nearly every row has that many; an empty split's
// slot may hold anything and is dropped by its weight).  What bounds it is two memory round trips per warp and the waves of
// warps: behind 270 tokens of 32 heads in 16 slots, 2-6 of them in use, append + split + merge 237 -> 229 us; 48 rows x 32 heads in 8
// slots at hdim 64, split + merge 74.6 -> 72.6.  The order of the sums is that of combine_kernel.
template <typename T>
__global__ void __launch_bounds__(128) combine_pair_kernel(const CombineDev p) {
    constexpr int kFirst = 2;
    const int lane = threadIdx.x & 31, sub = lane & 15;
    const int64_t item = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 2 + (lane >> 4);
    const bool exists = item < p.items;
    const int64_t it = exists ? item : p.items - 1;  // (an odd last row: the other half walks along and stores nothing)
    const int r = (int)(it % p.rows);
    const int64_t bh = it / p.rows;
    const int h = (int)(bh % p.hq);
    const int64_t b = bh / p.hq;
    const int S = p.S, nvec = p.dv >> 2;
    const float* lrow = p.lse_acc + b * p.lb + h * p.lh + r * p.lr;
    const float4* obase = reinterpret_cast<const float4*>(p.o_acc + b * p.ob + h * p.oh + r * p.orr);
    const int64_t os4 = p.os >> 2;
    const bool c0 = sub < nvec, c1 = sub + 16 < nvec;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const float ninf = -INFINITY;
    pdl_wait();  // the split kernel's partials are complete and visible (no-op after an ordinary launch)

    float4 x[4][2];
#pragma unroll
    for (int u = 0; u < kFirst; ++u) {
        x[u][0] = (u < S && c0) ? obase[u * os4 + sub] : zero;
        x[u][1] = (u < S && c1) ? obase[u * os4 + sub + 16] : zero;
    }
    const float ls = sub < S ? lrow[sub * p.ls] : ninf;
    float m = ls;
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
    const float e = (ls == ninf) ? 0.f : expf(ls - m);
    float sum = e;
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    const float wl = m == ninf ? 0.f : e * (1.f / sum);
    // splits in use by either row of the warp
    const uint32_t used = __ballot_sync(0xffffffffu, ls != ninf);
    const int cnt = 32 - __clz((used | used >> 16) & 0xffffu);

    float4 acc[2] = {zero, zero};
    for (int j0 = 0; j0 < cnt; j0 += 4) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (j0 == 0 && u < kFirst) continue;
            const bool live = used >> ((lane & 16) + ((j0 + u) & 15)) & 1u;  // (only splits below S are in use)
            x[u][0] = (live && c0) ? obase[(j0 + u) * os4 + sub] : zero;
            x[u][1] = (live && c1) ? obase[(j0 + u) * os4 + sub + 16] : zero;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const float w = __shfl_sync(0xffffffffu, wl, (lane & 16) + ((j0 + u) & 15));
            if (w != 0.f) {
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    acc[j].x += w * x[u][j].x;
                    acc[j].y += w * x[u][j].y;
                    acc[j].z += w * x[u][j].z;
                    acc[j].w += w * x[u][j].w;
                }
            }
        }
    }
    if (!exists) return;
    T* orow = (T*)p.o + ((b * p.rows + r) * p.hq + h) * (int64_t)p.dv;
    if (c0) Out4<T>::store(orow + 4 * sub, acc[0]);  // (no split saw a key: zeros)
    if (c1) Out4<T>::store(orow + 4 * (sub + 16), acc[1]);
    if (p.lse && sub == 0) p.lse[item] = m == ninf ? ninf : m + logf(sum);
}

// Several warps per row (one CTA = one row), for rows with many splits: a warp that walks 94 splits four rows at a time
// pays a memory round trip for every four.  Warp w takes splits w, w + W, ...; it requests its first kAhead rows before
// it has seen any LSE (a split without keys may hold anything: its row is dropped by its weight of zero, not multiplied),
// so that a row of up to W * kAhead splits costs one round trip for LSE and partials together, and a longer one another for
// every further W * kAhead.  The LSEs of all slots and the partials of the first W * kAhead are read whether a split has keys or
// not; of the later ones a warp skips every kAhead in which none has.
// Merging one token of 32 heads over 128 split slots, 94 in use: 16.4 us with one warp per row, 3.3 us with 16 (back to
// back in a graph; 24.5 us alone behind its split kernel before).
template <typename T, int W>
__global__ void __launch_bounds__(W * 32) combine_wide_kernel(const CombineDev p) {
    constexpr int kAhead = 4;
    extern __shared__ float4 part[];  // [W][dv / 4]: the warps' weighted sums
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t item = blockIdx.x;
    const int r = (int)(item % p.rows);
    const int64_t bh = item / p.rows;
    const int h = (int)(bh % p.hq);
    const int64_t b = bh / p.hq;
    const int S = p.S;
    const float* lrow = p.lse_acc + b * p.lb + h * p.lh + r * p.lr;
    const float* obase = p.o_acc + b * p.ob + h * p.oh + r * p.orr;
    const int nvec = p.dv >> 2;
    const bool c0 = lane < nvec, c1 = lane + 32 < nvec;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const float ninf = -INFINITY;

    float4 x[kAhead][2];
    auto fetch = [&](int j0) {  // this warp's splits j0 .. j0 + kAhead - 1
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int s = (j0 + u) * W + warp;
            const float4* src = reinterpret_cast<const float4*>(obase + (int64_t)s * p.os);
            x[u][0] = (s < S && c0) ? src[lane] : zero;
            x[u][1] = (s < S && c1) ? src[lane + 32] : zero;
        }
    };
    fetch(0);
    float mine = lane * W + warp < S ? lrow[(int64_t)(lane * W + warp) * p.ls] : ninf;  // lane j: split j * W + warp
    // maximum and sum of weights over all splits (every warp for itself: they are at most a few loads per lane)
    float l4[4], m = ninf;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        l4[u] = lane + 32 * u < S ? lrow[(int64_t)(lane + 32 * u) * p.ls] : ninf;
        m = fmaxf(m, l4[u]);
    }
    for (int s = lane + 128; s < S; s += 32) m = fmaxf(m, lrow[s * p.ls]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
    T* orow = (T*)p.o + ((b * p.rows + r) * p.hq + h) * (int64_t)p.dv;
    if (m == ninf) {  // no split saw a key: O = 0, LSE = -inf (the same in every warp)
        for (int c = threadIdx.x; c < nvec; c += W * 32) Out4<T>::store(orow + 4 * c, zero);
        if (p.lse && threadIdx.x == 0) p.lse[item] = ninf;
        return;
    }
    float sum = 0.f;
#pragma unroll
    for (int u = 0; u < 4; ++u) sum += (l4[u] == ninf) ? 0.f : expf(l4[u] - m);
    for (int s = lane + 128; s < S; s += 32) {
        const float ls = lrow[s * p.ls];
        sum += (ls == ninf) ? 0.f : expf(ls - m);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    const float inv = 1.f / sum;

    float4 acc[2] = {zero, zero};
    for (int j0 = 0; j0 * W + warp < S; j0 += kAhead) {
        if (j0 > 0) {
            if ((j0 & 31) == 0) mine = (j0 + lane) * W + warp < S ? lrow[(int64_t)((j0 + lane) * W + warp) * p.ls] : ninf;
            // (the splits in use come first: behind them there is nothing to fetch)
            if (!__any_sync(0xffffffffu, mine != ninf && lane >= (j0 & 31) && lane < (j0 & 31) + kAhead)) continue;
            fetch(j0);
        }
        const float wl = (mine == ninf) ? 0.f : expf(mine - m) * inv;
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const float w = __shfl_sync(0xffffffffu, wl, (j0 + u) & 31);
            if (w == 0.f) continue;  // (warp-uniform)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                acc[j].x += w * x[u][j].x;
                acc[j].y += w * x[u][j].y;
                acc[j].z += w * x[u][j].z;
                acc[j].w += w * x[u][j].w;
            }
        }
    }
    if (c0) part[warp * nvec + lane] = acc[0];
    if (c1) part[warp * nvec + lane + 32] = acc[1];
    __syncthreads();
    for (int c = threadIdx.x; c < nvec; c += W * 32) {
        float4 t = part[c];
#pragma unroll
        for (int w = 1; w < W; ++w) {
            const float4 y = part[w * nvec + c];
            t.x += y.x; t.y += y.y; t.z += y.z; t.w += y.w;
        }
        Out4<T>::store(orow + 4 * c, t);
    }
    if (p.lse && threadIdx.x == 0) p.lse[item] = m + logf(sum);
}

template <typename T>
cudaError_t launch_t(const CombineDev& d, cudaStream_t stream) {
    // Warps per row: as many as still find two splits each, while the rows together stay within 16 warps per SM; more
    // warps than that only queue, and the other rows hide a row's round trips.  Measured (us with 1 / 4 / 8 / 16 warps,
    // dv 128): 32 rows x 128 slots 16.4 / 4.9 / 3.7 / 3.3; 256 x 75 9.6 / 4.1 / 3.7 / 4.4; 512 x 20 4.2 / 3.1 / 3.6 /
    // 6.0; 2048 x 16 4.4 / 5.5 / 9.5 / 18; 2048 x 6 3.6 / 5.4 / 9.1 / 17.
    // (The order of a row's fp32 sum follows from W, and so from the number of rows in the call.)
    const int64_t warps_ok = (int64_t)sm_count() * 16 / (d.items > 0 ? d.items : 1);
    const dim3 g((unsigned)d.items);
    const size_t row = d.dv * sizeof(float);
    if (warps_ok >= 16 && d.S > 32) return launch_dependent(combine_wide_kernel<T, 16>, g, dim3(512), 16 * row, stream, d);
    if (warps_ok >= 8 && d.S > 16) return launch_dependent(combine_wide_kernel<T, 8>, g, dim3(256), 8 * row, stream, d);
    if (warps_ok >= 4 && d.S > 8) return launch_dependent(combine_wide_kernel<T, 4>, g, dim3(128), 4 * row, stream, d);
    const int warps = 4;
    if (d.S <= 16 && d.dv <= 128)
        return launch_dependent(combine_pair_kernel<T>, dim3((unsigned)((d.items + 2 * warps - 1) / (2 * warps))),
                                dim3(warps * 32), 0, stream, d);
    return launch_dependent(combine_kernel<T>, dim3((unsigned)((d.items + warps - 1) / warps)), dim3(warps * 32), 0, stream, d);
}

}  // namespace

int launch_combine(const CombineParams& p, cudaStream_t stream) {
    FCK_REQUIRE(p.dv % 4 == 0 && p.dv <= 256, FLASHCK_ERR_UNSUPPORTED,
                "combine: v_head_dim must be a multiple of 4 and <= 256 (got %lld)", (long long)p.dv);
    FCK_REQUIRE(p.num_splits >= 1, FLASHCK_ERR_INVALID_ARGUMENT, "combine: num_splits must be >= 1");
    FCK_REQUIRE(p.dtype == FLASHCK_DTYPE_BFLOAT16 || p.dtype == FLASHCK_DTYPE_FLOAT16 || p.dtype == FLASHCK_DTYPE_FLOAT32,
                FLASHCK_ERR_UNSUPPORTED, "combine: output dtype must be 3 (float16), 4 (bfloat16) or 7 (float32)");
    CombineDev d;
    d.lse_acc = p.lse_acc; d.o_acc = p.o_acc; d.o = p.o; d.lse = p.lse;
    d.items = p.bs * p.hq * p.rows;
    d.rows = (int)p.rows; d.hq = (int)p.hq; d.dv = (int)p.dv; d.S = (int)p.num_splits;
    if (p.strided) {
        d.lb = p.lse_strides[0]; d.lh = p.lse_strides[1]; d.ls = p.lse_strides[2]; d.lr = p.lse_strides[3];
        d.ob = p.o_strides[0]; d.oh = p.o_strides[1]; d.os = p.o_strides[2]; d.orr = p.o_strides[3];
        FCK_REQUIRE(d.ob % 4 == 0 && d.oh % 4 == 0 && d.os % 4 == 0 && d.orr % 4 == 0, FLASHCK_ERR_INVALID_ARGUMENT,
                    "combine: o_acc strides must be multiples of 4 elements");
    } else {
        d.lr = 1; d.ls = p.rows; d.lh = p.num_splits * p.rows; d.lb = p.hq * d.lh;
        d.orr = p.dv; d.os = p.rows * p.dv; d.oh = p.num_splits * d.os; d.ob = p.hq * d.oh;
    }
    if (d.items == 0) return FLASHCK_OK;
    if (p.dtype == FLASHCK_DTYPE_BFLOAT16) FCK_CUDA(launch_t<__nv_bfloat16>(d, stream));
    else if (p.dtype == FLASHCK_DTYPE_FLOAT16) FCK_CUDA(launch_t<__half>(d, stream));
    else FCK_CUDA(launch_t<float>(d, stream));
    return FLASHCK_OK;
}

}  // namespace fck
