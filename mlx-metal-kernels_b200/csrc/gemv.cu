// Quantized matvec / skinny GEMM for decode: host-side dispatch and the general kernel.
//
//   y[b, n] = sum_k x[b, k] * (code[n, k] - zero[n, k/G]) * scale[n, k/G]
//
// Group sizes 32 / 64 / 128 with 16-byte aligned rows run on tensor cores: one to four batch rows on integer products of the raw
// codes (gemv_i8.cuh), five and more on tcgen05 (qgemm_ts.cu; bf16 rows when the caller gives scratch for their fp16 form), what
// neither takes - scales that are not fp16 - on fp16 mma.sync (gemv_fast.cuh, up to 16 batch rows per launch).  Everything else runs the general kernel
// below, which follows the reference arithmetic literally.
#include "gemv_params.cuh"

#include <algorithm>
#include <cmath>

namespace b200q {

// Defined in api.cu
int rmsnorm_residual_launch(const void* x, const void* residual, const void* weight, void* y, void* z_out,
                            int64_t rows, int64_t D, float eps, int dtype, int w_dtype, cudaStream_t stream);

int gemv_read_status(int reset, cudaStream_t stream) {
    const int a = gemv_q4_read_status(reset, stream);
    const int b = gemv_q8_read_status(reset, stream);
    const int c = qgemm_ts_read_status(reset, stream);
    const int d = gemv_i8_q4_read_status(reset, stream);
    const int e = gemv_i8_q8_read_status(reset, stream);
    for (int v : {a, b, c, d})
        if (v != 0) return v;
    return e;
}

namespace {

__device__ __forceinline__ float round_act(float v, int dtype) {
    return dtype == B200Q_F16 ? __half2float(__float2half_rn(v)) : __bfloat162float(__float2bfloat16_rn(v));
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ---------------------------------------------------------------------------------------------
// Generic kernel: any K / group size / alignment.  One warp per (output row), all batch rows.
// Follows the reference: W = cast(fp32(code - zero) * scale) in the activation dtype, fp32 sum.
// ---------------------------------------------------------------------------------------------
template <bool GATE_UP>
__global__ void __launch_bounds__(256) qgemv_generic_kernel(const __grid_constant__ GemvParams p, int bits) {
    constexpr int MATS = GATE_UP ? 2 : 1;
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= p.N) return;
    const float fmax_act = p.act_dtype == B200Q_F16 ? 65504.0f : 3.3895313892515355e38f;
    for (int b = 0; b < p.B; ++b) {
        float acc[MATS];
#pragma unroll
        for (int m = 0; m < MATS; ++m) acc[m] = 0.0f;
        for (int k = lane; k < p.K; k += 32) {
            const float xv = load_as_f32(p.x, p.act_dtype, (int64_t)b * p.K + k);
            const int gi = min(k / p.G, p.Gn - 1);
#pragma unroll
            for (int m = 0; m < MATS; ++m) {
                float q;
                if (bits == 4) {
                    const uint8_t byte = p.w[m][row * p.row_bytes + (k >> 1)];
                    q = (float)((k & 1) ? (byte >> 4) : (byte & 0x0F));
                } else {
                    q = (float)p.w[m][row * p.row_bytes + k];
                }
                const float s = load_as_f32(p.s[m], p.scale_dtype, row * p.Gn + gi);
                float w = p.z[m] != nullptr
                              ? __fmul_rn(__fsub_rn(q, load_as_f32(p.z[m], p.scale_dtype, row * p.Gn + gi)), s)
                              : __fmul_rn(q, s);
                w = round_act(w, p.act_dtype);
                acc[m] = fmaf(xv, w, acc[m]);
            }
        }
        float val[MATS];
#pragma unroll
        for (int m = 0; m < MATS; ++m) {
            const float s = warp_sum(acc[m]);
            val[m] = round_act(fminf(fmaxf(s, -fmax_act), fmax_act), p.act_dtype);
        }
        if (lane == 0) {
            const int64_t o = (int64_t)b * p.N + row;
            auto store = [&](void* base, float v) {
                if (p.act_dtype == B200Q_F16) reinterpret_cast<__half*>(base)[o] = __float2half_rn(v);
                else reinterpret_cast<__nv_bfloat16*>(base)[o] = __float2bfloat16_rn(v);
            };
            if (GATE_UP) {
                if (p.gate_out != nullptr) store(p.gate_out, val[0]);
                if (p.up_out != nullptr) store(p.up_out, val[MATS - 1]);
                if (p.act_out != nullptr) {
                    const float silu = val[0] / (1.0f + expf(-val[0]));
                    store(p.act_out, silu * val[MATS - 1]);
                }
            } else {
                float v = val[0];
                if (p.residual != nullptr) v = load_as_f32(p.residual, p.act_dtype, o) + v;
                store(p.y, v);
            }
        }
    }
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

template <bool GATE_UP>
int launch_generic(const GemvParams& p, int bits, cudaStream_t stream) {
    const int warps = 8;
    const int grid = (int)((p.N + warps - 1) / warps);
    qgemv_generic_kernel<GATE_UP><<<grid, warps * 32, 0, stream>>>(p, bits);
    return finish_launch();
}

// The general kernel has no norm prologue: the caller runs the stand-alone rmsnorm kernel first when
// the tensor-core kernel does not apply.
bool fast_path_ok(const GemvParams& p) {
    if (tuning_get("gemv.force_generic")) return false;
    if (p.G != 32 && p.G != 64 && p.G != 128) return false;
    if (p.K % p.G != 0 || p.row_bytes % 16 != 0) return false;
    if (p.B > 64) return false;
    if (!aligned16(p.x) || !aligned16(p.w[0]) || (p.w[1] != nullptr && !aligned16(p.w[1]))) return false;
    if (p.res_in != nullptr && !aligned16(p.res_in)) return false;
    if (p.z_out != nullptr && !aligned16(p.z_out)) return false;
    if (p.normed_out != nullptr && !aligned16(p.normed_out)) return false;
    return true;
}

// Which kernel takes a launch: "gemv.ts" = 1 sends everything the tcgen05 kernel supports to it, -1 nothing, 0 (default) the batches
// of gemv.ts_min_batch rows and more.  Default 5: the integer kernel has no instance above four rows, and against the fp16 mma.sync
// kernel tcgen05 wins from there on (fp16 rows, 14336 x 4096 q4: 14.2 against 18.9 us at five rows; 4096 x 14336: 15.0 against 26.2).
// One region of bf16 rows goes the other way: their weights take two terms there, which doubles the chain of chunks, and with a
// row tile for more than half of the SMs no K split can shorten it; up to eight rows are one launch of the mma.sync kernel.
// mma.sync / tcgen05, us, eight rows of q4, groups of 64: 11008 x 4096 20.4 / 22.2, gate and up 28.6 / 39.5; 11008 x 7168 32.8 / 35.3;
// outside: 11008 x 2048 15.0 / 13.1, 9344 x 4096 18.7 / 15.7, 2048 x 8192 22.3 / 13.4.  The region is coarse: q8 (14336 x 4096 26.5 / 22.0)
// and groups of 32 (11008 x 4096 26.0 / 22.7) would be faster with tcgen05 inside it, 11008 x 8192 (34.4 / 39.9) with mma.sync outside.
bool prefer_ts(const GemvParams& p) {
    const int mode = tuning_get("gemv.ts");
    if (mode < 0) return false;
    if (mode > 0) return true;
    const int min_b = tuning_get("gemv.ts_min_batch");
    if (min_b > 0) return p.B >= min_b;
    if (p.B < 5) return false;
    const int64_t rows_full = (int64_t)p.N * std::max(1, tuning_get("ts.tp_world"));      // of the unsharded matrix: a shard takes the same kernel
    const bool scale_rows = p.scale_dtype == B200Q_F16 && p.Gn % 8 == 0 && aligned16(p.s[0]) && aligned16(p.z[0]) && aligned16(p.s[1]) && aligned16(p.z[1]);
    return !(p.act_dtype == B200Q_BF16 && p.B <= 8 && scale_rows && rows_full > 64 * sm_count() && p.K > 2048 && p.K < 8192);
}

// bf16 rows in fp16 for the tcgen05 kernel: one power of two per row brings the largest element to [2^13, 2^14); bf16 has 8
// significant bits, so everything down to 2^-20 of the largest element is exact.  One CTA per row.
__global__ void __launch_bounds__(256) rows_to_fp16_kernel(const uint16_t* __restrict__ x, __half* __restrict__ out, float* __restrict__ scale, int K) {
    __shared__ float part[8];
    pdl_launch_dependents();
    pdl_wait();
    const size_t row = (size_t)blockIdx.x * K;
    float mx = 0.0f;
    for (int k = threadIdx.x * 8; k < K; k += 256 * 8) {
        const uint4 u = *reinterpret_cast<const uint4*>(x + row + k);
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) mx = fmaxf(mx, fmaxf(fabsf(__uint_as_float(w[i] << 16)), fabsf(__uint_as_float(w[i] & 0xFFFF0000u))));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = mx;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i) mx = fmaxf(mx, part[i]);
    int ex = 0;
    if (mx > 0.0f && mx < INFINITY) frexpf(mx, &ex);
    ex = max(-100, min(114, ex - 14));
    const float sc = exp2f((float)ex), down = exp2f((float)-ex);
    if (threadIdx.x == 0) scale[blockIdx.x] = sc;
    for (int k = threadIdx.x * 8; k < K; k += 256 * 8) {
        const uint4 u = *reinterpret_cast<const uint4*>(x + row + k);
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
        __half2 h[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(__uint_as_float(w[i] << 16) * down, __uint_as_float(w[i] & 0xFFFF0000u) * down);
        *reinterpret_cast<uint4*>(out + row + k) = *reinterpret_cast<const uint4*>(h);
    }
}
int rows_to_fp16(const void* x, void* out, float* scale, int rows, int K, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(rows);
    cfg.blockDim = dim3(256);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = tuning_get("no_pdl") ? 0 : 1;
    if (cudaLaunchKernelEx(&cfg, rows_to_fp16_kernel, (const uint16_t*)x, (__half*)out, scale, K) != cudaSuccess) return B200Q_ERR_LAUNCH;
    return finish_launch();
}

int dispatch_fast(int bits, GemvParams& p, bool gate_up, cudaStream_t stream) {
    if (p.B <= 4 && tuning_get("gemv.i8") >= 0) {
        const int rc = bits == 4 ? gemv_i8_q4(p, gate_up, stream) : gemv_i8_q8(p, gate_up, stream);
        if (rc != B200Q_ERR_UNSUPPORTED) return rc;      // rows that do not fit into its shared memory
    }
    if (p.B > 16) return B200Q_ERR_UNSUPPORTED;
    return bits == 4 ? gemv_fast_q4(p, gate_up, stream) : gemv_fast_q8(p, gate_up, stream);
}

thread_local void* t_scratch = nullptr;          // b200q_scratch_next: for the next matvec / gate-up call of this thread
thread_local size_t t_scratch_bytes = 0;
struct ScratchGuard {                            // a call that ends early must not leave its scratch to the next one
    ~ScratchGuard() { t_scratch = nullptr; t_scratch_bytes = 0; }
};

constexpr int kMinApart = 5;                     // rows from which on the norm, or the conversion of bf16 rows, is a launch of its own
size_t scratch_rows(int rows, int64_t K) { return ((size_t)rows * K * 2 + 255) / 256 * 256; }
size_t scratch_scales(int rows) { return ((size_t)rows * 4 + 255) / 256 * 256; }

// rows b0 .. b0 + bn of a problem
GemvParams slice(const GemvParams& a, int b0, int bn) {
    GemvParams p = a;
    auto in = [&](const void* base, size_t width) -> const void* { return base ? static_cast<const uint8_t*>(base) + (size_t)b0 * width * 2 : nullptr; };
    auto out = [&](void* base, size_t width) -> void* { return base ? static_cast<uint8_t*>(base) + (size_t)b0 * width * 2 : nullptr; };
    p.x = in(a.x, a.K); p.res_in = in(a.res_in, a.K);
    p.z_out = out(a.z_out, a.K); p.normed_out = out(a.normed_out, a.K);
    p.residual = in(a.residual, a.N);
    p.y = out(a.y, a.N); p.gate_out = out(a.gate_out, a.N); p.up_out = out(a.up_out, a.N); p.act_out = out(a.act_out, a.N);
    p.B = bn;
    return p;
}

// All rows of a problem (all.B of them) through the kernels.
int run_rows(int bits, GemvParams all, bool gate_up, cudaStream_t stream) {
    void* scratch = t_scratch;
    const size_t scratch_bytes = t_scratch_bytes;
    const bool tp_used = all.tp_in.world > 0 || all.tp_out.world > 0;
    const bool tensor_cores = !tuning_get("gemv.force_generic");
    const bool bf = all.act_dtype == B200Q_BF16;
    // the scratch: bf16 rows as fp16 and their powers of two, then normalised rows
    const size_t rows_bytes = scratch_rows(all.B, all.K), fp16_bytes = bf ? rows_bytes + scratch_scales(all.B) : 0;
    const bool usable = scratch != nullptr && aligned16(scratch), room = !bf || (usable && scratch_bytes >= fp16_bytes);
    void* normed = all.normed_out;
    if (normed == nullptr && usable && scratch_bytes >= fp16_bytes + rows_bytes) normed = static_cast<uint8_t*>(scratch) + fp16_bytes;
    // From five rows on the norm is a launch of its own where there is a buffer for its rows, the caller's or scratch: inside the matvec
    // kernels every CTA would repeat it, and only mma.sync kernels of up to 16 rows have it at all (4096 -> 2 x 14336 q4, cold calls by
    // events: 8 rows 53 us fused, 36 apart; 32 rows 188 and 38).
    auto norm_first = [&]() -> int {
        if (all.norm_w == nullptr || normed == nullptr) return B200Q_OK;
        const int rc = rmsnorm_residual_launch(all.x, all.res_in, all.norm_w, normed, all.z_out, all.B, all.K, all.eps, all.act_dtype,
                                               all.norm_w_dtype, stream);
        all.x = normed;
        all.norm_w = nullptr; all.res_in = nullptr; all.z_out = nullptr; all.normed_out = nullptr;
        return rc;
    };
    const bool ts = !tp_used && tensor_cores && prefer_ts(all);
    if (ts) {
        GemvParams probe = all;
        if (bf) probe.col_scale = reinterpret_cast<const float*>(scratch);
        if (probe.norm_w != nullptr) probe.x = normed;
        if (room && probe.x != nullptr && qgemm_ts_applies(probe, gate_up)) {
            int rc = norm_first();
            if (rc != B200Q_OK) return rc;
            GemvParams p = all;
            if (bf) {
                float* cs = reinterpret_cast<float*>(static_cast<uint8_t*>(scratch) + rows_bytes);
                rc = rows_to_fp16(all.x, scratch, cs, all.B, all.K, stream);
                if (rc != B200Q_OK) return rc;
                p.x = scratch;
                p.col_scale = cs;
            }
            rc = qgemm_ts(bits, p, gate_up, stream);
            if (rc != B200Q_ERR_UNSUPPORTED) return rc;
        }
    }
    if ((ts || (!tp_used && all.B >= kMinApart && tuning_get("gemv.ts") >= 0)) && fast_path_ok(slice(all, 0, std::min(all.B, 16)))) {
        const int rc = norm_first();
        if (rc != B200Q_OK) return rc;
    }
    int chunk = 16;      // batch rows per launch; halved when a kernel's shared-memory plan does not fit
    for (int b0 = 0; b0 < all.B;) {
        GemvParams p = slice(all, b0, std::min(chunk, all.B - b0));
        const bool fast = fast_path_ok(p);
        int rc = fast ? dispatch_fast(bits, p, gate_up, stream) : B200Q_ERR_UNSUPPORTED;
        if (rc == B200Q_ERR_UNSUPPORTED && tp_used) return rc;      // exchanges exist only in the tensor-core kernels
        if (rc == B200Q_ERR_UNSUPPORTED && p.B > 1 && fast) {
            chunk = (p.B + 1) / 2;
            continue;
        }
        if (rc == B200Q_ERR_UNSUPPORTED) {
            if (!fast) p = slice(all, b0, all.B - b0);              // the general kernel takes all rows at once
            if (p.norm_w != nullptr) {
                // generic route: materialise the normalised rows first (normed_out is required as the buffer)
                if (p.normed_out == nullptr) return B200Q_ERR_UNSUPPORTED;
                rc = rmsnorm_residual_launch(p.x, p.res_in, p.norm_w, p.normed_out, p.z_out, p.B, p.K, p.eps, p.act_dtype, p.norm_w_dtype, stream);
                if (rc != B200Q_OK) return rc;
                p.x = p.normed_out;
                p.norm_w = nullptr; p.res_in = nullptr; p.z_out = nullptr; p.normed_out = nullptr;
            }
            rc = gate_up ? launch_generic<true>(p, bits, stream) : launch_generic<false>(p, bits, stream);
        }
        if (rc != B200Q_OK) return rc;
        b0 += p.B;
    }
    return B200Q_OK;
}

void set_tp(GemvParams& p, int in_slot, int out_slot) {
    if (out_slot >= 0) p.tp_out = tp_slot(out_slot)->out;
    if (in_slot >= 0) {
        const TpOut& src = tp_slot(in_slot)->out;
        p.tp_in.flags = src.flags[src.rank];
        p.tp_in.epoch = src.epoch;
        p.tp_in.world = src.world;
        p.tp_in.spin_limit = (uint32_t)std::max(0, tuning_get("tp.spin_limit"));
        p.tp_in.packets = src.packets;
    }
}

}  // namespace

void scratch_next(void* ptr, size_t bytes) {
    t_scratch = ptr;
    t_scratch_bytes = ptr != nullptr ? bytes : 0;
}
size_t scratch_bytes_impl(int rows, int64_t K, int act_dtype) {
    if (K <= 0 || act_dtype != B200Q_BF16 || rows < kMinApart) return 0;
    return scratch_rows(rows, K) + scratch_scales(rows);
}
size_t norm_scratch_bytes_impl(int rows, int64_t K, int act_dtype) {
    if (K <= 0 || !is_act_dtype(act_dtype) || rows < kMinApart) return 0;
    return scratch_bytes_impl(rows, K, act_dtype) + scratch_rows(rows, K);
}

int qmatvec_impl(int bits, const void* x, const uint8_t* codes, const void* scales, const void* zeros,
                 const void* residual, void* y, int B, int64_t N, int64_t K, int group_size, int act_dtype,
                 int scale_dtype, const void* residual_in, const void* norm_weight, int norm_w_dtype, float eps,
                 void* z_out, void* normed_out, cudaStream_t stream) {
    const ScratchGuard guard;
    int tp_in_slot = -1, tp_out_slot = -1;
    tp_take(&tp_in_slot, &tp_out_slot);
    if ((bits != 4 && bits != 8) || x == nullptr || codes == nullptr || scales == nullptr ||
        (y == nullptr && tp_out_slot < 0))
        return B200Q_ERR_BAD_ARG;
    if ((tp_in_slot >= 0 || tp_out_slot >= 0) && B > 16) return B200Q_ERR_UNSUPPORTED;
    if (B <= 0 || N <= 0 || K <= 0 || group_size <= 0 || !is_act_dtype(act_dtype) || !is_scale_dtype(scale_dtype))
        return B200Q_ERR_BAD_ARG;
    if (norm_weight != nullptr && !is_scale_dtype(norm_w_dtype)) return B200Q_ERR_BAD_ARG;
    if (norm_weight == nullptr && (residual_in != nullptr || z_out != nullptr || normed_out != nullptr))
        return B200Q_ERR_BAD_ARG;
    if (N > INT32_MAX || K > INT32_MAX) return B200Q_ERR_UNSUPPORTED;
    GemvParams p = {};
    p.x = x; p.res_in = residual_in; p.norm_w = norm_weight; p.eps = eps; p.norm_w_dtype = norm_w_dtype;
    p.z_out = z_out; p.normed_out = normed_out;
    p.w[0] = codes; p.s[0] = scales; p.z[0] = zeros;
    p.residual = residual; p.y = y;
    p.B = B; p.N = (int)N; p.K = (int)K; p.G = group_size; p.Gn = (int)((K + group_size - 1) / group_size);
    p.act_dtype = act_dtype; p.scale_dtype = scale_dtype;
    p.row_bytes = bits == 4 ? (int)((K + 1) / 2) : (int)K;
    set_tp(p, tp_in_slot, tp_out_slot);
    return run_rows(bits, p, false, stream);
}

int gate_up_impl(int bits, const void* x, const uint8_t* gate_codes, const uint8_t* up_codes, const void* gate_scales,
                 const void* up_scales, const void* gate_zeros, const void* up_zeros, void* gate_out, void* up_out,
                 void* act_out, const void* residual_in, const void* norm_weight, float eps, void* z_out,
                 void* normed_out, int rows, int64_t N, int64_t K, int group_size, int act_dtype, int scale_dtype,
                 int norm_w_dtype, cudaStream_t stream) {
    const ScratchGuard guard;
    int tp_in_slot = -1, tp_out_slot = -1;
    tp_take(&tp_in_slot, &tp_out_slot);
    if ((bits != 4 && bits != 8) || x == nullptr || gate_codes == nullptr || up_codes == nullptr ||
        gate_scales == nullptr || up_scales == nullptr)
        return B200Q_ERR_BAD_ARG;
    if ((tp_in_slot >= 0 || tp_out_slot >= 0) && rows > 16) return B200Q_ERR_UNSUPPORTED;
    if (rows <= 0 || N <= 0 || K <= 0 || group_size <= 0 || !is_act_dtype(act_dtype) || !is_scale_dtype(scale_dtype))
        return B200Q_ERR_BAD_ARG;
    if (norm_weight != nullptr && !is_scale_dtype(norm_w_dtype)) return B200Q_ERR_BAD_ARG;
    if (norm_weight == nullptr && (residual_in != nullptr || z_out != nullptr || normed_out != nullptr))
        return B200Q_ERR_BAD_ARG;
    if (N > INT32_MAX || K > INT32_MAX) return B200Q_ERR_UNSUPPORTED;
    GemvParams p = {};
    p.x = x; p.res_in = residual_in; p.norm_w = norm_weight; p.eps = eps; p.norm_w_dtype = norm_w_dtype;
    p.z_out = z_out; p.normed_out = normed_out;
    p.w[0] = gate_codes; p.w[1] = up_codes;
    p.s[0] = gate_scales; p.s[1] = up_scales;
    p.z[0] = gate_zeros; p.z[1] = up_zeros;
    p.gate_out = gate_out; p.up_out = up_out; p.act_out = act_out;
    p.B = rows; p.N = (int)N; p.K = (int)K; p.G = group_size; p.Gn = (int)((K + group_size - 1) / group_size);
    p.act_dtype = act_dtype; p.scale_dtype = scale_dtype;
    p.row_bytes = bits == 4 ? (int)((K + 1) / 2) : (int)K;
    set_tp(p, tp_in_slot, tp_out_slot);
    return run_rows(bits, p, true, stream);
}

}  // namespace b200q
