// The bandwidth-bound tail of the convolution path: pooling, fully_connected
// (reference order), softmax, eltwise, reorder, lrn and standalone activation.
// The *_ref kernels take any layout through pitches; pooling_i8_byxf is the
// feature-innermost fast path with 16-byte accesses per lane.
#include <algorithm>
#include <cuda_fp16.h>
#include "engine.hpp"
#include "reorder_tile.hpp"
#include "sm100_ptx.cuh"

namespace b200 {

// Launch with programmatic stream serialisation: the kernel's blocks may be scheduled while the previous kernel of the stream
// drains, so it executes griddepcontrol.wait before it touches memory.
template <class... Params, class... Args>
static cudaError_t launch_dependent(void (*kernel)(Params...), dim3 grid, int threads, cudaStream_t s, Args... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid; cfg.blockDim = dim3((unsigned)threads); cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

static inline int grid_for(int64_t total, int threads, const cldnn_b200_ctx_impl* ctx)
{
    int64_t blocks = (total + threads - 1) / threads;
    const int64_t cap = (int64_t)ctx->prop.multiProcessorCount * 16;
    if (blocks > cap) blocks = cap;
    return blocks < 1 ? 1 : (int)blocks;
}

// ---------------------------------------------------------------------------------
// pooling, any layout.  int8: cl_kernels/pooling_gpu_int8_ref.cl:35-131;
// float: cl_kernels/pooling_gpu_ref.cl:36-201.
// ---------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t pool_divisor(const cldnn_b200_pool_params& p, int ox, int oy, uint32_t n)
{
    if (p.div_mode == CLDNN_B200_DIV_DYNAMIC) return n ? n : 1u;
    if (p.div_mode == CLDNN_B200_DIV_DYNAMIC_WITH_PADDING) {
        const int hend = min(oy + p.size_y, p.in.y + p.pad_y), wend = min(ox + p.size_x, p.in.x + p.pad_x);
        const uint32_t d = (uint32_t)((hend - oy) * (wend - ox));
        return d ? d : 1u;
    }
    return (uint32_t)(p.size_x * p.size_y);
}

// element index -> coordinates, x innermost (planar layouts) or f innermost (byxf)
__device__ __forceinline__ void decode_bfyx(int64_t idx, int F, int Y, int X, bool f_inner, int& b, int& f, int& y, int& x)
{
    if (f_inner) { f = (int)(idx % F); int64_t t = idx / F; x = (int)(t % X); t /= X; y = (int)(t % Y); b = (int)(t / Y); }
    else { x = (int)(idx % X); int64_t t = idx / X; y = (int)(t % Y); t /= Y; f = (int)(t % F); b = (int)(t / F); }
}

__global__ void __launch_bounds__(256)
pooling_ref_kernel(const __grid_constant__ cldnn_b200_pool_params p, const void* in, void* out)
{
    const int64_t total = (int64_t)p.out.b * p.out.f * p.out.y * p.out.x;
    const bool int_in = is_int8(p.in.dtype);
    const bool f_inner = p.in.pf == 1 && p.out.pf == 1;             // consecutive threads follow the innermost dimension of the layout
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
        int b, f, y, x;
        decode_bfyx(idx, p.out.f, p.out.y, p.out.x, f_inner, b, f, y, x);
        const int ox = x * p.stride_x - p.pad_x, oy = y * p.stride_y - p.pad_y;
        if (ox + p.size_x < 0 || ox >= p.in.x || oy + p.size_y < 0 || oy >= p.in.y) continue;
        int32_t ri = p.mode == CLDNN_B200_POOL_MAX ? -128 : 0;
        float rf = p.mode == CLDNN_B200_POOL_MAX ? (p.in.dtype == CLDNN_B200_F16 ? -65504.0f : -3.402823466e38f) : 0.0f;
        uint32_t n = 0;
        for (int j = 0; j < p.size_y; ++j) {
            const int iy = oy + j; if (iy < 0 || iy >= p.in.y) continue;
            for (int i = 0; i < p.size_x; ++i) {
                const int ix = ox + i; if (ix < 0 || ix >= p.in.x) continue;
                const int64_t ii = tidx(p.in, b, f, iy, ix);
                if (int_in) { const int32_t v = load_as_int(in, p.in.dtype, ii); ri = p.mode == CLDNN_B200_POOL_MAX ? max(ri, v) : ri + v; }
                else { const float v = load_as_float(in, p.in.dtype, ii); rf = p.mode == CLDNN_B200_POOL_MAX ? fmaxf(rf, v) : __fadd_rn(rf, v); }
                ++n;
            }
        }
        const uint32_t div = pool_divisor(p, ox, oy, n);
        const int64_t oi = tidx(p.out, b, f, y, x);
        if (int_in) {
            if (p.mode == CLDNN_B200_POOL_AVG) ri = (int32_t)round_half_away(__fdiv_rn((float)ri, (float)div));
            if (p.out.dtype == CLDNN_B200_U8) ((uint8_t*)out)[oi] = (uint8_t)act_int(p.act, (int32_t)(uint8_t)ri, p.act_m, p.act_n);
            else if (p.out.dtype == CLDNN_B200_I8) ((int8_t*)out)[oi] = (int8_t)act_int(p.act, (int32_t)(int8_t)ri, p.act_m, p.act_n);
            else store_sat_int(out, p.out.dtype, oi, act_int(p.act, ri, p.act_m, p.act_n));
        } else {
            if (p.mode == CLDNN_B200_POOL_AVG) rf = __fdiv_rn(rf, (float)div);
            store_sat_float(out, p.out.dtype, oi, act_float(p.act, rf, p.act_m, p.act_n));
        }
    }
}

static bool pooling_ref_supports(const void* vp)
{
    const auto& p = *(const cldnn_b200_pool_params*)vp;
    return p.size_x >= 1 && p.size_y >= 1 && p.stride_x >= 1 && p.stride_y >= 1 && p.in.f == p.out.f && p.in.b == p.out.b;
}
static int one_tune(const void*) { return 1; }

static int32_t pooling_ref_prepare(cldnn_b200_ctx_impl* ctx, const void* vp, const cldnn_b200_args* a, cldnn_b200_prepared_impl* out)
{
    const cldnn_b200_pool_params p = *(const cldnn_b200_pool_params*)vp;
    if (!a->input0 || !a->output) return fail(CLDNN_B200_INVALID_ARG, "pooling_ref: input and output are required");
    const void* in = a->input0; void* o = a->output;
    const int grid = grid_for((int64_t)p.out.b * p.out.f * p.out.y * p.out.x, 256, ctx);
    out->fn = [p, in, o, grid](cudaStream_t s) { pooling_ref_kernel<<<grid, 256, 0, s>>>(p, in, o); return cudaGetLastError(); };
    return CLDNN_B200_SUCCESS;
}
const KernelDef kdef_pooling_ref = {"pooling_ref", sizeof(cldnn_b200_pool_params), pooling_ref_supports, one_tune, nullptr, pooling_ref_prepare};

// ---------------------------------------------------------------------------------
// pooling, 8-bit, feature-innermost (byxf) fast path: each thread owns 16
// consecutive features of one output pixel and moves them with one 128-bit
// load per window tap and one 128-bit store.  Same arithmetic as
// pooling_gpu_int8_ref.cl.
// ---------------------------------------------------------------------------------
template <bool kUnsigned>
__device__ __forceinline__ void unpack16(const uint4& v, int32_t (&e)[16])
{
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const uint32_t byte = (w[i >> 2] >> ((i & 3) * 8)) & 0xffu;
        e[i] = kUnsigned ? (int32_t)byte : (int32_t)(int8_t)byte;
    }
}

// Item walk of the grid-stride loops over (batch, y, x, feature vector): the first item and the stride are
// decomposed once, every later item follows by digit-wise addition with carries (a division by a run-time
// divisor costs more instructions than the pooling of one item).
struct ItemWalk {
    int f, x, y, b, sf, sx, sy, sb, nf, nx, ny;
    __device__ __forceinline__ void init(uint32_t first, uint32_t stride, int fv, int X, int Y)
    {
        nf = fv; nx = X; ny = Y;
        f = (int)(first % (uint32_t)fv); uint32_t t = first / (uint32_t)fv;
        x = (int)(t % (uint32_t)X); t /= (uint32_t)X; y = (int)(t % (uint32_t)Y); b = (int)(t / (uint32_t)Y);
        sf = (int)(stride % (uint32_t)fv); t = stride / (uint32_t)fv;
        sx = (int)(t % (uint32_t)X); t /= (uint32_t)X; sy = (int)(t % (uint32_t)Y); sb = (int)(t / (uint32_t)Y);
    }
    __device__ __forceinline__ void next()
    {
        f += sf; int c = f >= nf ? 1 : 0; f -= c ? nf : 0;
        x += sx + c; c = x >= nx ? 1 : 0; x -= c ? nx : 0;
        y += sy + c; c = y >= ny ? 1 : 0; y -= c ? ny : 0;
        b += sb + c;
    }
};

// Running maximum of four packed bytes kept as two words of 16-bit lanes, for the three-input 16-bit-pair maximum of
// the hardware: the odd bytes are compared through the raw word (the upper byte of a lane decides, the lower byte is
// ignored at the end), the even bytes are moved into the upper bytes of the lanes first.
template <bool kUnsigned>
struct ByteMax {
    uint32_t odd = kUnsigned ? 0u : 0x80008000u, even = kUnsigned ? 0u : 0x80008000u;
    static __device__ __forceinline__ uint32_t up(uint32_t w) { return __byte_perm(w, 0u, 0x2404); }    // bytes 0, 2 -> bytes 1, 3
    static __device__ __forceinline__ uint32_t max3(uint32_t a, uint32_t b, uint32_t c) { return kUnsigned ? __vimax3_u16x2(a, b, c) : __vimax3_s16x2(a, b, c); }
    __device__ __forceinline__ void add3(uint32_t a, uint32_t b, uint32_t c)
    {
        odd = max3(odd, max3(a, b, c), odd);
        even = max3(even, max3(up(a), up(b), up(c)), even);
    }
    // relu: signed bytes, negative maxima become 0
    __device__ __forceinline__ uint32_t result(bool relu) const
    {
        uint32_t o = odd, e = even;
        if (!kUnsigned && relu) { o = __vimax3_s16x2_relu(o, o, o); e = __vimax3_s16x2_relu(e, e, e); }
        return __byte_perm(o, e, 0x3715);                                                              // e.b1, o.b1, e.b3, o.b3
    }
};

template <bool kUnsignedIn>
__global__ void __launch_bounds__(256)
pooling_i8_byxf_kernel(const __grid_constant__ cldnn_b200_pool_params p, const uint8_t* __restrict__ in, uint8_t* __restrict__ out)
{
    ptx::griddep_launch_dependents();
    const int fv = p.in.f / 16;
    const int64_t total = (int64_t)p.out.b * p.out.y * p.out.x * fv;
    const bool fast_max = p.mode == CLDNN_B200_POOL_MAX && (p.act == CLDNN_B200_ACT_NONE || p.act == CLDNN_B200_ACT_RELU);
    // (32-bit index arithmetic: a 64-bit division costs more instructions than the pooling itself; the host admits < 2^31 items)
    ItemWalk it; it.init(blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x, fv, p.out.x, p.out.y);
    for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < (uint32_t)total; idx += gridDim.x * blockDim.x, it.next()) {
        const int f16 = it.f, x = it.x, y = it.y, b = it.b;
        const int ox = x * p.stride_x - p.pad_x, oy = y * p.stride_y - p.pad_y;
        if (ox + p.size_x < 0 || ox >= p.in.x || oy + p.size_y < 0 || oy >= p.in.y) continue;
        if (fast_max) {
            // maximum of the valid taps on packed bytes, no unpacking to 32 bits: the stored bits are the bits of the
            // largest input (the conversion to the output type wraps), ReLU on a signed output is one more max
            const int j0 = max(0, -oy), j1 = min(p.size_y, p.in.y - oy), i0 = max(0, -ox), i1 = min(p.size_x, p.in.x - ox);
            const uint8_t* src = in + tidx(p.in, b, f16 * 16, oy, ox);
            ByteMax<kUnsignedIn> bm[4];
            if (p.size_x == 3 && p.size_y == 3 && j0 < j1 && i0 < i1) {
                // 3x3 window: taps outside the input are replaced by the nearest valid tap (a repeated element does not
                // change a maximum), so the nine loads carry no branches and are all in flight together
                uint4 v[9];
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const int64_t ro = (int64_t)min(max(j, j0), j1 - 1) * p.in.py;
#pragma unroll
                    for (int i = 0; i < 3; ++i)
                        v[j * 3 + i] = __ldg((const uint4*)(src + ro + (int64_t)min(max(i, i0), i1 - 1) * p.in.px));
                }
#pragma unroll
                for (int k = 0; k < 9; k += 3) {
                    bm[0].add3(v[k].x, v[k + 1].x, v[k + 2].x); bm[1].add3(v[k].y, v[k + 1].y, v[k + 2].y);
                    bm[2].add3(v[k].z, v[k + 1].z, v[k + 2].z); bm[3].add3(v[k].w, v[k + 1].w, v[k + 2].w);
                }
            } else
            for (int j = j0; j < j1; ++j) {
#pragma unroll 3
                for (int i = i0; i < i1; ++i) {
                    const uint4 v = __ldg((const uint4*)(src + (int64_t)j * p.in.py + (int64_t)i * p.in.px));
                    bm[0].add3(v.x, v.x, v.x); bm[1].add3(v.y, v.y, v.y); bm[2].add3(v.z, v.z, v.z); bm[3].add3(v.w, v.w, v.w);
                }
            }
            const bool relu = p.act == CLDNN_B200_ACT_RELU && p.out.dtype == CLDNN_B200_I8;
            const uint4 m = make_uint4(bm[0].result(relu), bm[1].result(relu), bm[2].result(relu), bm[3].result(relu));
            *(uint4*)(out + tidx(p.out, b, f16 * 16, y, x)) = m;
            continue;
        }
        int32_t r[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) r[i] = p.mode == CLDNN_B200_POOL_MAX ? -128 : 0;
        uint32_t n = 0;
        const int taps = p.size_x * p.size_y;
        if (p.mode == CLDNN_B200_POOL_AVG && ox >= 0 && oy >= 0 && ox + p.size_x <= p.in.x && oy + p.size_y <= p.in.y && taps <= 256) {
            // whole window inside the input: sums of at most 256 bytes fit 16-bit lanes, so two masks and two additions
            // take a word of four bytes (signed bytes are summed as byte + 128 and the 128s taken out at the end);
            // eight taps are loaded per batch so that a long window (a global average) is not one load latency per tap
            const uint8_t* src = in + tidx(p.in, b, f16 * 16, oy, ox);
            uint32_t a[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
            int ti = 0, tj = 0;
            for (int t0 = 0; t0 < taps; t0 += 8) {
                uint4 v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    v[u] = make_uint4(0u, 0u, 0u, 0u);
                    if (t0 + u < taps) {
                        v[u] = __ldg((const uint4*)(src + (int64_t)tj * p.in.py + (int64_t)ti * p.in.px));
                        if (!kUnsignedIn) { v[u].x ^= 0x80808080u; v[u].y ^= 0x80808080u; v[u].z ^= 0x80808080u; v[u].w ^= 0x80808080u; }
                    }
                    if (++ti == p.size_x) { ti = 0; ++tj; }
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const uint32_t w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
                    for (int k = 0; k < 4; ++k) { a[2 * k] += w[k] & 0x00ff00ffu; a[2 * k + 1] += (w[k] >> 8) & 0x00ff00ffu; }
                }
            }
            n = (uint32_t)taps;
            const int32_t off = kUnsignedIn ? 0 : 128 * taps;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                r[4 * k + 0] = (int32_t)(a[2 * k] & 0xffffu) - off;     r[4 * k + 1] = (int32_t)(a[2 * k + 1] & 0xffffu) - off;
                r[4 * k + 2] = (int32_t)(a[2 * k] >> 16) - off;         r[4 * k + 3] = (int32_t)(a[2 * k + 1] >> 16) - off;
            }
        } else
        for (int j = 0; j < p.size_y; ++j) {
            const int iy = oy + j; if (iy < 0 || iy >= p.in.y) continue;
            for (int i = 0; i < p.size_x; ++i) {
                const int ix = ox + i; if (ix < 0 || ix >= p.in.x) continue;
                const uint4 v = __ldg((const uint4*)(in + tidx(p.in, b, f16 * 16, iy, ix)));
                int32_t e[16]; unpack16<kUnsignedIn>(v, e);
#pragma unroll
                for (int k = 0; k < 16; ++k) r[k] = p.mode == CLDNN_B200_POOL_MAX ? max(r[k], e[k]) : r[k] + e[k];
                ++n;
            }
        }
        const float div = (float)pool_divisor(p, ox, oy, n);
        uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            int32_t v = r[k];
            if (p.mode == CLDNN_B200_POOL_AVG) v = (int32_t)round_half_away(__fdiv_rn((float)v, div));
            // convert_char / convert_uchar wrap, then the activation runs on the 8-bit value
            v = p.out.dtype == CLDNN_B200_U8 ? (int32_t)(uint8_t)v : (int32_t)(int8_t)v;
            v = act_int(p.act, v, p.act_m, p.act_n);
            w[k >> 2] |= ((uint32_t)v & 0xffu) << ((k & 3) * 8);
        }
        *(uint4*)(out + tidx(p.out, b, f16 * 16, y, x)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// Averages over long windows of few outputs (global pooling): the kernel above walks a window of 49 taps in one thread, and 1280 features
// of one image are 80 threads: 9.5 us for 63 KB.  Here a block takes one output pixel of up to 256
// features, 16 threads share each vector of 16 features tap by tap, and the partial sums (packed as above: at most 256 taps
// keep every 16-bit lane exact, in any order) meet in shared memory.
constexpr int kWinSlices = 16, kWinVecs = 16;
template <bool kUnsignedIn>
__global__ void __launch_bounds__(kWinSlices * kWinVecs)
pooling_i8_window_kernel(const __grid_constant__ cldnn_b200_pool_params p, const uint8_t* __restrict__ in, uint8_t* __restrict__ out)
{
    __shared__ uint32_t part[kWinSlices][kWinVecs][8];
    ptx::griddep_launch_dependents();
    const int fv = p.in.f / 16, groups = (fv + kWinVecs - 1) / kWinVecs;
    uint32_t t = blockIdx.x;
    const int g = (int)(t % (uint32_t)groups); t /= (uint32_t)groups;
    const int x = (int)(t % (uint32_t)p.out.x); t /= (uint32_t)p.out.x;
    const int y = (int)(t % (uint32_t)p.out.y), b = (int)(t / (uint32_t)p.out.y);
    const int ox = x * p.stride_x, oy = y * p.stride_y, taps = p.size_x * p.size_y;
    {
        const int vec = threadIdx.x % kWinVecs, slice = threadIdx.x / kWinVecs;
        uint32_t a[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
        if (g * kWinVecs + vec < fv) {
            const uint8_t* src = in + tidx(p.in, b, (g * kWinVecs + vec) * 16, oy, ox);
#pragma unroll 4
            for (int i = slice; i < taps; i += kWinSlices) {
                const int tj = i / p.size_x, ti = i - tj * p.size_x;
                uint4 v = __ldg((const uint4*)(src + (int64_t)tj * p.in.py + (int64_t)ti * p.in.px));
                if (!kUnsignedIn) { v.x ^= 0x80808080u; v.y ^= 0x80808080u; v.z ^= 0x80808080u; v.w ^= 0x80808080u; }
                const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) { a[2 * k] += w[k] & 0x00ff00ffu; a[2 * k + 1] += (w[k] >> 8) & 0x00ff00ffu; }
            }
        }
        *reinterpret_cast<uint4*>(&part[slice][vec][0]) = make_uint4(a[0], a[1], a[2], a[3]);
        *reinterpret_cast<uint4*>(&part[slice][vec][4]) = make_uint4(a[4], a[5], a[6], a[7]);
    }
    __syncthreads();
    // one feature per thread: byte k of its vector lies in lane (k & 3) >> 1 of word 2 * (k / 4) + (k & 1)
    const int vec = threadIdx.x / 16, k = threadIdx.x % 16, f = (g * kWinVecs + vec) * 16 + k;
    if (f >= p.in.f) return;
    uint32_t s = 0u;
#pragma unroll
    for (int i = 0; i < kWinSlices; ++i) s += part[i][vec][2 * (k >> 2) + (k & 1)];
    int32_t v = (int32_t)((k & 2) ? s >> 16 : s & 0xffffu) - (kUnsignedIn ? 0 : 128 * taps);
    v = (int32_t)round_half_away(__fdiv_rn((float)v, (float)pool_divisor(p, ox, oy, (uint32_t)taps)));
    v = p.out.dtype == CLDNN_B200_U8 ? (int32_t)(uint8_t)v : (int32_t)(int8_t)v;
    v = act_int(p.act, v, p.act_m, p.act_n);
    out[tidx(p.out, b, f, y, x)] = (uint8_t)v;
}
static int64_t pooling_i8_window_blocks(const cldnn_b200_pool_params& p)
{
    return (int64_t)p.out.b * p.out.y * p.out.x * ((p.in.f / 16 + kWinVecs - 1) / kWinVecs);
}
// Whole windows of 16 to 256 taps inside the input (below that a window is too short to share), as many blocks as are resident at once (eight
// per SM), up to twice that for the longest windows.  Beyond, one thread per output vector fills the device by itself and a block per output
// pixel only adds work, the more the fewer features it has.  Over 1959 shapes (windows of 4 to 16, 16 .. 2048 features, 1 .. 256 images) the rule
// is never behind the general kernel and on average 0.6 % behind the better of the two (at worst 1.49): 7x7 of 1280 features, one image, 9.5 -> 3.5
// us; 16x16 of 256 features, 64 images, 29 -> 6.3; but 4x4 stride 4 of 64 features at 112x112, 64 images (50 k blocks), 21 us in general and 119 here.
static bool pooling_i8_by_window(const cldnn_b200_pool_params& p, int sms)
{
    const int taps = p.size_x * p.size_y;
    return p.mode == CLDNN_B200_POOL_AVG && taps >= kWinSlices && taps <= 256 && p.size_x > 0 && p.pad_x == 0 && p.pad_y == 0 && p.out.x > 0 && p.out.y > 0 && p.out.b > 0 &&
           (p.out.x - 1) * p.stride_x + p.size_x <= p.in.x && (p.out.y - 1) * p.stride_y + p.size_y <= p.in.y &&
           pooling_i8_window_blocks(p) * 256 <= (int64_t)8 * sms * (256 + taps);
}

static bool pooling_i8_byxf_supports(const void* vp)
{
    const auto& p = *(const cldnn_b200_pool_params*)vp;
    if (!pooling_ref_supports(vp)) return false;
    if (!is_int8(p.in.dtype) || !is_int8(p.out.dtype)) return false;
    if (p.in.pf != 1 || p.out.pf != 1 || p.in.f % 16) return false;
    const int64_t pitches[] = {p.in.px, p.in.py, p.in.pb, p.in.offset, p.out.px, p.out.py, p.out.pb, p.out.offset};
    for (int64_t v : pitches) if (v % 16) return false;
    if ((int64_t)p.out.b * p.out.y * p.out.x * (p.in.f / 16) >= 0x7fffffffLL) return false;      // 32-bit item index
    return true;
}

static int32_t pooling_i8_byxf_prepare(cldnn_b200_ctx_impl* ctx, const void* vp, const cldnn_b200_args* a, cldnn_b200_prepared_impl* out)
{
    const cldnn_b200_pool_params p = *(const cldnn_b200_pool_params*)vp;
    if (!a->input0 || !a->output) return fail(CLDNN_B200_INVALID_ARG, "pooling_i8_byxf: input and output are required");
    if (((uintptr_t)a->input0 | (uintptr_t)a->output) & 15) return fail(CLDNN_B200_INVALID_ARG, "pooling_i8_byxf: buffers must be 16-byte aligned");
    const uint8_t* in = (const uint8_t*)a->input0; uint8_t* o = (uint8_t*)a->output;
    const int grid = grid_for((int64_t)p.out.b * p.out.y * p.out.x * (p.in.f / 16), 256, ctx);
    const bool uns = p.in.dtype == CLDNN_B200_U8;
    if (pooling_i8_by_window(p, ctx->prop.multiProcessorCount)) {
        const unsigned blocks = (unsigned)pooling_i8_window_blocks(p);
        out->fn = [p, in, o, blocks, uns](cudaStream_t s) {
            if (uns) pooling_i8_window_kernel<true><<<blocks, kWinSlices * kWinVecs, 0, s>>>(p, in, o);
            else pooling_i8_window_kernel<false><<<blocks, kWinSlices * kWinVecs, 0, s>>>(p, in, o);
            return cudaGetLastError();
        };
        return CLDNN_B200_SUCCESS;
    }
    out->fn = [p, in, o, grid, uns](cudaStream_t s) {
        if (uns) pooling_i8_byxf_kernel<true><<<grid, 256, 0, s>>>(p, in, o);
        else pooling_i8_byxf_kernel<false><<<grid, 256, 0, s>>>(p, in, o);
        return cudaGetLastError();
    };
    return CLDNN_B200_SUCCESS;
}
const KernelDef kdef_pooling_i8_byxf = {"pooling_i8_byxf", sizeof(cldnn_b200_pool_params), pooling_i8_byxf_supports, one_tune, nullptr, pooling_i8_byxf_prepare};

// ---------------------------------------------------------------------------------
// pooling, fp16, feature-innermost (byxf): each thread owns 8 consecutive features of one
// output pixel, one 128-bit load per window tap and one 128-bit store; the maximum on
// packed halves, the average accumulated in fp32.  Same arithmetic as pooling_gpu_ref.cl
// (its half accumulator for the average is replaced by a float one: tolerance parity).
// ---------------------------------------------------------------------------------
template <int S>
__device__ __forceinline__ void pool_max_clamped(const __half* src, int64_t px, int64_t py, int i0, int i1, int j0, int j1, __half2 (&m)[4])
{
    uint4 v[S * S];
#pragma unroll
    for (int j = 0; j < S; ++j) {
        const int64_t ro = (int64_t)min(max(j, j0), j1 - 1) * py;
#pragma unroll
        for (int i = 0; i < S; ++i)
            v[j * S + i] = __ldg(reinterpret_cast<const uint4*>(src + ro + (int64_t)min(max(i, i0), i1 - 1) * px));
    }
#pragma unroll
    for (int t = 0; t < S * S; ++t) {
        const __half2* h = reinterpret_cast<const __half2*>(&v[t]);
#pragma unroll
        for (int k = 0; k < 4; ++k) m[k] = __hmax2(m[k], h[k]);
    }
}

__global__ void __launch_bounds__(256)
pooling_f16_byxf_kernel(const __grid_constant__ cldnn_b200_pool_params p, const __half* __restrict__ in, __half* __restrict__ out)
{
    ptx::griddep_launch_dependents();
    const int fv = p.in.f / 8;
    const int64_t total = (int64_t)p.out.b * p.out.y * p.out.x * fv;
    const bool is_max = p.mode == CLDNN_B200_POOL_MAX;
    ItemWalk it; it.init(blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x, fv, p.out.x, p.out.y);
    for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < (uint32_t)total; idx += gridDim.x * blockDim.x, it.next()) {   // < 2^31 items (host check)
        const int f8 = it.f, x = it.x, y = it.y, b = it.b;
        const int ox = x * p.stride_x - p.pad_x, oy = y * p.stride_y - p.pad_y;
        if (ox + p.size_x < 0 || ox >= p.in.x || oy + p.size_y < 0 || oy >= p.in.y) continue;
        const int j0 = max(0, -oy), j1 = min(p.size_y, p.in.y - oy), i0 = max(0, -ox), i1 = min(p.size_x, p.in.x - ox);
        const __half* src = in + tidx(p.in, b, f8 * 8, oy, ox);
        const __half2 lowest = __half2half2(__ushort_as_half((unsigned short)0xfbffu));      // -65504, the reference's HALF_MIN start value
        __half2 m[4] = {lowest, lowest, lowest, lowest};
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        uint32_t n = 0;
        const bool sq3 = p.size_x == 3 && p.size_y == 3, sq2 = p.size_x == 2 && p.size_y == 2;
        if (is_max && (sq3 || sq2) && j0 < j1 && i0 < i1) {
            // small square window: taps outside the input are replaced by the nearest valid tap (a repeated element
            // does not change a maximum), so the loads carry no branches and are all in flight together
            if (sq3) pool_max_clamped<3>(src, p.in.px, p.in.py, i0, i1, j0, j1, m);
            else pool_max_clamped<2>(src, p.in.px, p.in.py, i0, i1, j0, j1, m);
        } else
        for (int j = j0; j < j1; ++j) {
            for (int i = i0; i < i1; ++i) {
                const uint4 v = __ldg(reinterpret_cast<const uint4*>(src + (int64_t)j * p.in.py + (int64_t)i * p.in.px));
                const __half2* h = reinterpret_cast<const __half2*>(&v);
                if (is_max) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) m[k] = __hmax2(m[k], h[k]);
                } else {
#pragma unroll
                    for (int k = 0; k < 4; ++k) { const float2 f = __half22float2(h[k]); acc[2 * k] += f.x; acc[2 * k + 1] += f.y; }
                }
                ++n;
            }
        }
        if (is_max && (p.act == CLDNN_B200_ACT_NONE || p.act == CLDNN_B200_ACT_RELU)) {
            // the maximum is one of the inputs: stored as it is (ReLU: one more packed maximum), no trip through fp32
            if (p.act == CLDNN_B200_ACT_RELU) {
                const __half2 zero = __float2half2_rn(0.0f);
#pragma unroll
                for (int k = 0; k < 4; ++k) m[k] = __hmax2(m[k], zero);
            }
            *reinterpret_cast<uint4*>(out + tidx(p.out, b, f8 * 8, y, x)) = *reinterpret_cast<const uint4*>(m);
            continue;
        }
        float r[8];
        if (is_max) {
#pragma unroll
            for (int k = 0; k < 4; ++k) { const float2 f = __half22float2(m[k]); r[2 * k] = f.x; r[2 * k + 1] = f.y; }
        } else {
            const float div = (float)pool_divisor(p, ox, oy, n);
#pragma unroll
            for (int k = 0; k < 8; ++k) r[k] = __fdiv_rn(acc[k], div);
        }
        __half2 o[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            o[k] = __floats2half2_rn(act_float(p.act, r[2 * k], p.act_m, p.act_n), act_float(p.act, r[2 * k + 1], p.act_m, p.act_n));
        *reinterpret_cast<uint4*>(out + tidx(p.out, b, f8 * 8, y, x)) = *reinterpret_cast<const uint4*>(o);
    }
}

static bool pooling_f16_byxf_supports(const void* vp)
{
    const auto& p = *(const cldnn_b200_pool_params*)vp;
    if (!pooling_ref_supports(vp)) return false;
    if (p.in.dtype != CLDNN_B200_F16 || p.out.dtype != CLDNN_B200_F16) return false;
    if (p.in.pf != 1 || p.out.pf != 1 || p.in.f % 8) return false;
    const int64_t pitches[] = {p.in.px, p.in.py, p.in.pb, p.in.offset, p.out.px, p.out.py, p.out.pb, p.out.offset};
    for (int64_t v : pitches) if (v % 8) return false;
    if ((int64_t)p.out.b * p.out.y * p.out.x * (p.in.f / 8) >= 0x7fffffffLL) return false;       // 32-bit item index
    return true;
}

static int32_t pooling_f16_byxf_prepare(cldnn_b200_ctx_impl* ctx, const void* vp, const cldnn_b200_args* a, cldnn_b200_prepared_impl* out)
{
    const cldnn_b200_pool_params p = *(const cldnn_b200_pool_params*)vp;
    if (!a->input0 || !a->output) return fail(CLDNN_B200_INVALID_ARG, "pooling_f16_byxf: input and output are required");
    if (((uintptr_t)a->input0 | (uintptr_t)a->output) & 15) return fail(CLDNN_B200_INVALID_ARG, "pooling_f16_byxf: buffers must be 16-byte aligned");
    const __half* in = (const __half*)a->input0; __half* o = (__half*)a->output;
    const int grid = grid_for((int64_t)p.out.b * p.out.y * p.out.x * (p.in.f / 8), 256, ctx);
    out->fn = [p, in, o, grid](cudaStream_t s) { pooling_f16_byxf_kernel<<<grid, 256, 0, s>>>(p, in, o); return cudaGetLastError(); };
    return CLDNN_B200_SUCCESS;
}
const KernelDef kdef_pooling_f16_byxf = {"pooling_f16_byxf", sizeof(cldnn_b200_pool_params), pooling_f16_byxf_supports, one_tune, nullptr, pooling_f16_byxf_prepare};

// ---------------------------------------------------------------------------------
// fully_connected in the reference's order (cl_kernels/fully_connected_gpu_bfyx_ref.cl:18-84):
// one warp per output, lanes stride the reduction, shuffle-reduce (integer sums
// are order-independent; float sums are tolerance-checked).
// ---------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
fc_ref_kernel(const __grid_constant__ cldnn_b200_fc_params p, const void* in, const void* w, const void* bias,
              const float* quant, const float* calib, void* out)
{
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t total = (int64_t)p.out.b * p.out.f;
    const int K = p.in.f * p.in.y * p.in.x;
    for (int64_t bo = warp; bo < total; bo += nwarps) {
        const int b = (int)(bo / p.out.f), o = (int)(bo % p.out.f);
        int32_t acc_i = 0; float acc_f = 0.f;
        for (int k = lane; k < K; k += 32) {
            const int x = k % p.in.x, y = (k / p.in.x) % p.in.y, f = k / (p.in.x * p.in.y);
            const int64_t ii = tidx(p.in, b, f, y, x);
            const int64_t wi = p.w_offset + (int64_t)o * p.w_po + (int64_t)f * p.w_pi + (int64_t)y * p.w_py + (int64_t)x * p.w_px;
            if (p.quantization) acc_i += load_as_int(in, p.in.dtype, ii) * load_as_int(w, p.w_dtype, wi);
            else acc_f += load_as_float(in, p.in.dtype, ii) * load_as_float(w, p.w_dtype, wi);
        }
#pragma unroll
        for (int s = 16; s; s >>= 1) { acc_i += __shfl_xor_sync(0xffffffffu, acc_i, s); acc_f += __shfl_xor_sync(0xffffffffu, acc_f, s); }
        if (lane) continue;
        const int64_t oi = tidx(p.out, b, o, 0, 0);
        if (p.quantization) {
            int32_t r = acc_i;
            if (p.bias_dtype != CLDNN_B200_NONE) {
                float t = __fmul_rn(__fmul_rn((float)acc_i, quant[o]), p.i_qf);
                t = __fadd_rn(t, load_as_float(bias, p.bias_dtype, o));
                t = __fmul_rn(t, p.calibration ? calib[o] : p.o_qf);
                r = sat_i32_from_float(round_half_away(t), -128, 127);
            } else r = min(127, max(-128, r));
            store_sat_int(out, p.out.dtype, oi, act_int(p.act, r, p.act_m, p.act_n));
        } else {
            float v = acc_f;
            if (p.bias_dtype != CLDNN_B200_NONE) v += load_as_float(bias, p.bias_dtype, o);
            store_sat_float(out, p.out.dtype, oi, act_float(p.act, v, p.act_m, p.act_n));
        }
    }
}
static bool fc_ref_supports(const void* vp) { const auto& p = *(const cldnn_b200_fc_params*)vp; return p.in.b == p.out.b && p.out.f >= 1; }
static int32_t fc_ref_prepare(cldnn_b200_ctx_impl* ctx, const void* vp, const cldnn_b200_args* a, cldnn_b200_prepared_impl* out)
{
    const cldnn_b200_fc_params p = *(const cldnn_b200_fc_params*)vp;
    if (!a->input0 || !a->output || !a->weights) return fail(CLDNN_B200_INVALID_ARG, "fc_ref: input, output and weights are required");
    if (p.quantization && p.bias_dtype != CLDNN_B200_NONE && !a->weights_quantization_factors) return fail(CLDNN_B200_INVALID_ARG, "fc_ref: quantization factors missing");
    if (p.calibration && !a->output_calibration_factors) return fail(CLDNN_B200_INVALID_ARG, "fc_ref: calibration factors missing");
    const void* in = a->input0; const void* w = a->weights; const void* bias = a->bias; void* o = a->output;
    const float* q = a->weights_quantization_factors; const float* c = a->output_calibration_factors;
    const int grid = grid_for((int64_t)p.out.b * p.out.f * 32, 256, ctx);
    out->fn = [=](cudaStream_t s) { fc_ref_kernel<<<grid, 256, 0, s>>>(p, in, w, bias, q, c, o); return cudaGetLastError(); };
    return CLDNN_B200_SUCCESS;
}
const KernelDef kdef_fc_ref = {"fc_ref", sizeof(cldnn_b200_fc_params), fc_ref_supports, one_tune, nullptr, fc_ref_prepare};

// ---------------------------------------------------------------------------------
// softmax over features (cl_kernels/softmax_gpu_ref.cl:22-58): one warp per
// (b, y, x) row; max, sum and normalise with warp shuffles, float accumulation.
// ---------------------------------------------------------------------------------
// set index + position inside the set -> coordinates, by the scope of normalisation (api/C/softmax.h:34-40)
__device__ __forceinline__ void softmax_coords(const cldnn_b200_softmax_params& p, int64_t set, int i, int& b, int& f, int& y, int& x)
{
    const int F = p.in.f, Y = p.in.y, X = p.in.x;
    switch (p.dimension) {
    case CLDNN_B200_SOFTMAX_X:   x = i; y = (int)(set % Y); f = (int)((set / Y) % F); b = (int)(set / ((int64_t)Y * F)); break;
    case CLDNN_B200_SOFTMAX_Y:   y = i; x = (int)(set % X); f = (int)((set / X) % F); b = (int)(set / ((int64_t)X * F)); break;
    case CLDNN_B200_SOFTMAX_FYX: x = i % X; y = (i / X) % Y; f = i / (X * Y); b = (int)set; break;
    default:                     f = i; x = (int)(set % X); y = (int)((set / X) % Y); b = (int)(set / ((int64_t)X * Y)); break;
    }
}
__host__ __device__ inline int64_t softmax_len(const cldnn_b200_softmax_params& p)
{
    switch (p.dimension) {
    case CLDNN_B200_SOFTMAX_X: return p.in.x;
    case CLDNN_B200_SOFTMAX_Y: return p.in.y;
    case CLDNN_B200_SOFTMAX_FYX: return (int64_t)p.in.f * p.in.y * p.in.x;
    default: return p.in.f;
    }
}

__global__ void __launch_bounds__(256)
softmax_kernel(const __grid_constant__ cldnn_b200_softmax_params p, const void* in, void* out)
{
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int len = (int)softmax_len(p);
    const int64_t sets = len > 0 ? ((int64_t)p.in.b * p.in.f * p.in.y * p.in.x) / len : 0;
    for (int64_t r = warp; r < sets; r += nwarps) {
        int b, f, y, x;
        float mx = -3.402823466e38f;
        for (int i = lane; i < len; i += 32) { softmax_coords(p, r, i, b, f, y, x); mx = fmaxf(mx, load_as_float(in, p.in.dtype, tidx(p.in, b, f, y, x))); }
#pragma unroll
        for (int s = 16; s; s >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, s));
        float den = 0.f;
        for (int i = lane; i < len; i += 32) { softmax_coords(p, r, i, b, f, y, x); den += expf(load_as_float(in, p.in.dtype, tidx(p.in, b, f, y, x)) - mx); }
#pragma unroll
        for (int s = 16; s; s >>= 1) den += __shfl_xor_sync(0xffffffffu, den, s);
        for (int i = lane; i < len; i += 32) {
            softmax_coords(p, r, i, b, f, y, x);
            const float e = expf(load_as_float(in, p.in.dtype, tidx(p.in, b, f, y, x)) - mx);
            store_sat_float(out, p.out.dtype, tidx(p.out, b, f, y, x), __fdiv_rn(e, den));
        }
    }
}
// One block per row for long rows (classification heads): every thread keeps its elements in registers, two block
// reductions (max, sum) through shared memory, one pass over memory in, one out.
constexpr int kSoftmaxPerThread = 8;
__global__ void __launch_bounds__(256)
softmax_row_kernel(const __grid_constant__ cldnn_b200_softmax_params p, const void* in, void* out)
{
    __shared__ float red[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t rows = (int64_t)p.in.b * p.in.y * p.in.x;
    for (int64_t r = blockIdx.x; r < rows; r += gridDim.x) {
        const int x = (int)(r % p.in.x), y = (int)((r / p.in.x) % p.in.y), b = (int)(r / ((int64_t)p.in.x * p.in.y));
        float v[kSoftmaxPerThread];
        float mx = -3.402823466e38f;
#pragma unroll
        for (int i = 0; i < kSoftmaxPerThread; ++i) {
            const int f = threadIdx.x + i * 256;
            v[i] = f < p.in.f ? load_as_float(in, p.in.dtype, tidx(p.in, b, f, y, x)) : -3.402823466e38f;
            mx = fmaxf(mx, v[i]);
        }
#pragma unroll
        for (int s = 16; s; s >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, s));
        if (lane == 0) red[warp] = mx;
        __syncthreads();
        mx = red[0];
#pragma unroll
        for (int w = 1; w < 8; ++w) mx = fmaxf(mx, red[w]);
        __syncthreads();
        float den = 0.f;
#pragma unroll
        for (int i = 0; i < kSoftmaxPerThread; ++i) {
            const int f = threadIdx.x + i * 256;
            v[i] = f < p.in.f ? expf(v[i] - mx) : 0.f;
        }
        // the reference adds the exponentials of one row in feature order on one work-item; a tree sum differs from it in
        // the last bits only, inside the tolerance softmax is compared with
#pragma unroll
        for (int i = 0; i < kSoftmaxPerThread; ++i) den += v[i];
#pragma unroll
        for (int s = 16; s; s >>= 1) den += __shfl_xor_sync(0xffffffffu, den, s);
        if (lane == 0) red[warp] = den;
        __syncthreads();
        den = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) den += red[w];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kSoftmaxPerThread; ++i) {
            const int f = threadIdx.x + i * 256;
            if (f < p.in.f) store_sat_float(out, p.out.dtype, tidx(p.out, b, f, y, x), __fdiv_rn(v[i], den));
        }
    }
}
static bool softmax_supports(const void* vp)
{
    const auto& p = *(const cldnn_b200_softmax_params*)vp;
    return is_fp(p.in.dtype) && is_fp(p.out.dtype) && p.in.f == p.out.f && p.in.x == p.out.x && p.in.y == p.out.y && p.in.b == p.out.b &&
           p.dimension >= CLDNN_B200_SOFTMAX_F && p.dimension <= CLDNN_B200_SOFTMAX_FYX && softmax_len(p) < 0x7fffffffLL;
}
static int32_t softmax_prepare(cldnn_b200_ctx_impl* ctx, const void* vp, const cldnn_b200_args* a, cldnn_b200_prepared_impl* out)
{
    const cldnn_b200_softmax_params p = *(const cldnn_b200_softmax_params*)vp;
    if (!a->input0 || !a->output) return fail(CLDNN_B200_INVALID_ARG, "softmax: input and output are required");
    const void* in = a->input0; void* o = a->output;
    const int64_t len = softmax_len(p);
    const int64_t sets = len > 0 ? ((int64_t)p.in.b * p.in.f * p.in.y * p.in.x) / len : 0;
    const int grid = grid_for(sets * 32, 256, ctx);
    // the block-per-row kernel normalises over f; over a 1x1 map the whole-image scope is the same thing
    const bool over_f = p.dimension == CLDNN_B200_SOFTMAX_F || (p.dimension == CLDNN_B200_SOFTMAX_FYX && p.in.x == 1 && p.in.y == 1);
    const int64_t rows = (int64_t)p.in.b * p.in.y * p.in.x;
    const bool by_row = over_f && p.in.f >= 256 && p.in.f <= 256 * kSoftmaxPerThread && rows <= (int64_t)ctx->prop.multiProcessorCount * 32;
    const int row_grid = (int)(rows < 1 ? 1 : rows);
    out->fn = [=](cudaStream_t s) {
        if (by_row) softmax_row_kernel<<<row_grid, 256, 0, s>>>(p, in, o);
        else softmax_kernel<<<grid, 256, 0, s>>>(p, in, o);
        return cudaGetLastError();
    };
    return CLDNN_B200_SUCCESS;
}
const KernelDef kdef_softmax = {"softmax", sizeof(cldnn_b200_softmax_params), softmax_supports, one_tune, nullptr, softmax_prepare};

// ---------------------------------------------------------------------------------
// eltwise (cl_kernels/generic_eltwise_ref.cl:198-330)
// ---------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
eltwise_ref_kernel(const __grid_constant__ cldnn_b200_eltwise_params p, const void* in0, const void* in1, const float* calib, void* out)
{
    const int64_t total = (int64_t)p.out.b * p.out.f * p.out.y * p.out.x;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
        // iterate in the output's memory order of its innermost axis
        int b, f, y, x;
        if (p.out.pf == 1) { f = (int)(idx % p.out.f); int64_t t = idx / p.out.f; x = (int)(t % p.out.x); t /= p.out.x; y = (int)(t % p.out.y); b = (int)(t / p.out.y); }
        else { x = (int)(idx % p.out.x); int64_t t = idx / p.out.x; y = (int)(t % p.out.y); t /= p.out.y; f = (int)(t % p.out.f); b = (int)(t / p.out.f); }
        const int64_t i0 = tidx(p.in0, b % p.in0.b, f % p.in0.f, ((int64_t)y * p.stride_y0) % p.in0.y, ((int64_t)x * p.stride_x0) % p.in0.x);
        const int64_t i1 = tidx(p.in1, b % p.in1.b, f % p.in1.f, ((int64_t)y * p.stride_y1) % p.in1.y, ((int64_t)x * p.stride_x1) % p.in1.x);
        const int64_t oi = tidx(p.out, b, f, y, x);
        if (p.quantization) {
            const int32_t a = load_as_int(in0, p.in0.dtype, i0), c = load_as_int(in1, p.in1.dtype, i1);
            int32_t r;
            switch (p.mode) {
            case CLDNN_B200_ELTW_SUB: r = a - c; break;
            case CLDNN_B200_ELTW_MAX: r = max(a, c); break;
            case CLDNN_B200_ELTW_MIN: r = min(a, c); break;
            case CLDNN_B200_ELTW_PROD: r = a * c; break;
            default: r = a + c; break;
            }
            r = sat_i32_from_float(round_half_away(__fmul_rn((float)r, p.calibration ? calib[f] : p.o_qf)), -128, 127);
            store_sat_int(out, p.out.dtype, oi, act_int(p.act, r, p.act_m, p.act_n));
            continue;
        }
        const float a = load_as_float(in0, p.in0.dtype, i0), c = load_as_float(in1, p.in1.dtype, i1);
        float r;
        switch (p.mode) {
        case CLDNN_B200_ELTW_SUB: r = __fsub_rn(a, c); break;
        case CLDNN_B200_ELTW_MAX: r = fmaxf(a, c); break;
        case CLDNN_B200_ELTW_MIN: r = fminf(a, c); break;
        case CLDNN_B200_ELTW_PROD: r = __fmul_rn(a, c); break;
        default: r = __fadd_rn(a, c); break;
        }
        if (is_fp(p.out.dtype)) store_sat_float(out, p.out.dtype, oi, act_float(p.act, r, p.act_m, p.act_n));
        else store_sat_int(out, p.out.dtype, oi, act_int(p.act, (int32_t)r, p.act_m, p.act_n));
    }
}
static bool eltwise_supports(const void* vp) { const auto& p = *(const cldnn_b200_eltwise_params*)vp; return p.stride_x0 >= 1 && p.stride_y0 >= 1 && p.stride_x1 >= 1 && p.stride_y1 >= 1; }
static int32_t eltwise_prepare(cldnn_b200_ctx_impl* ctx, const void* vp, const cldnn_b200_args* a, cldnn_b200_prepared_impl* out)
{
    const cldnn_b200_eltwise_params p = *(const cldnn_b200_eltwise_params*)vp;
    if (!a->input0 || !a->input1 || !a->output) return fail(CLDNN_B200_INVALID_ARG, "eltwise_ref: two inputs and an output are required");
    if (p.quantization && p.calibration && !a->output_calibration_factors) return fail(CLDNN_B200_INVALID_ARG, "eltwise_ref: calibration factors missing");
    const void* i0 = a->input0; const void* i1 = a->input1; void* o = a->output; const float* c = a->output_calibration_factors;
    const int grid = grid_for((int64_t)p.out.b * p.out.f * p.out.y * p.out.x, 256, ctx);
    out->fn = [=](cudaStream_t s) { eltwise_ref_kernel<<<grid, 256, 0, s>>>(p, i0, i1, c, o); return cudaGetLastError(); };
    return CLDNN_B200_SUCCESS;
}
const KernelDef kdef_eltwise_ref = {"eltwise_ref", sizeof(cldnn_b200_eltwise_params), eltwise_supports, one_tune, nullptr, eltwise_prepare};

// ---------------------------------------------------------------------------------
// eltwise over equal dense layouts, 16 bytes per thread (the role of eltwise_simple_vload8.cl among the reference's kernels):
// both inputs and the output have the same sizes, pitches and element size, so the tensors are walked as flat arrays.
// 8-bit: the requantising form of generic_eltwise_ref.cl (integer operation, * O_QF or calibrations[f], round, saturate to
// char, activation, saturating store); fp16: the floating form.  Activations none / ReLU; features innermost when the
// factors are per feature.  Same results as eltwise_ref, element for element.
// ---------------------------------------------------------------------------------
template <bool kHalf>
__global__ void __launch_bounds__(256)
eltwise_vec_kernel(const __grid_constant__ cldnn_b200_eltwise_params p, const uint4* __restrict__ in0, const uint4* __restrict__ in1,
                   const float* __restrict__ calib, uint4* __restrict__ out, int64_t vectors, int32_t stored_f)
{
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < vectors; v += (int64_t)gridDim.x * blockDim.x) {
        const uint4 a = in0[v], c = in1[v];
        uint4 r;
        if (kHalf) {
            const __half2* ah = reinterpret_cast<const __half2*>(&a); const __half2* ch = reinterpret_cast<const __half2*>(&c);
            __half2* rh = reinterpret_cast<__half2*>(&r);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 x = __half22float2(ah[i]), y = __half22float2(ch[i]);
                float2 z;
                switch (p.mode) {
                case CLDNN_B200_ELTW_SUB: z = make_float2(__fsub_rn(x.x, y.x), __fsub_rn(x.y, y.y)); break;
                case CLDNN_B200_ELTW_MAX: z = make_float2(fmaxf(x.x, y.x), fmaxf(x.y, y.y)); break;
                case CLDNN_B200_ELTW_MIN: z = make_float2(fminf(x.x, y.x), fminf(x.y, y.y)); break;
                case CLDNN_B200_ELTW_PROD: z = make_float2(__fmul_rn(x.x, y.x), __fmul_rn(x.y, y.y)); break;
                default: z = make_float2(__fadd_rn(x.x, y.x), __fadd_rn(x.y, y.y)); break;
                }
                if (p.act == CLDNN_B200_ACT_RELU) { z.x = fmaxf(0.0f, z.x); z.y = fmaxf(0.0f, z.y); }
                rh[i] = __floats2half2_rn(z.x, z.y);
            }
        } else {
            const uint8_t* ab = reinterpret_cast<const uint8_t*>(&a); const uint8_t* cb = reinterpret_cast<const uint8_t*>(&c);
            uint8_t* rb = reinterpret_cast<uint8_t*>(&r);
            const int f0 = p.calibration ? (int)((v * 16) % stored_f) : 0;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int32_t x = p.in0.dtype == CLDNN_B200_U8 ? (int32_t)ab[i] : (int32_t)(int8_t)ab[i];
                const int32_t y = p.in1.dtype == CLDNN_B200_U8 ? (int32_t)cb[i] : (int32_t)(int8_t)cb[i];
                int32_t z;
                switch (p.mode) {
                case CLDNN_B200_ELTW_SUB: z = x - y; break;
                case CLDNN_B200_ELTW_MAX: z = max(x, y); break;
                case CLDNN_B200_ELTW_MIN: z = min(x, y); break;
                case CLDNN_B200_ELTW_PROD: z = x * y; break;
                default: z = x + y; break;
                }
                // a feature lane beyond the tensor's feature count (padding of the layout) has no factor: it stays what the operation gives on zeros
                const float factor = p.calibration ? (f0 + i < p.out.f ? calib[f0 + i] : 1.0f) : p.o_qf;
                z = sat_i32_from_float(round_half_away(__fmul_rn((float)z, factor)), -128, 127);
                if (p.act == CLDNN_B200_ACT_RELU) z = max(z, 0);
                rb[i] = p.out.dtype == CLDNN_B200_U8 ? (uint8_t)max(z, 0) : (uint8_t)(int8_t)z;
            }
        }
        out[v] = r;
    }
}
static bool same_dense(const cldnn_b200_tensor& a, const cldnn_b200_tensor& b)
{
    return a.b == b.b && a.f == b.f && a.y == b.y && a.x == b.x && a.pb == b.pb && a.pf == b.pf && a.py == b.py && a.px == b.px && a.offset == 0 && b.offset == 0;
}
// bytes of the tensor when it is one dense block (no padding between rows, images): 0 otherwise
static int64_t dense_elems(const cldnn_b200_tensor& t)
{
    if (t.pf == 1) return (t.py == t.px * t.x && t.pb == t.py * t.y && t.px >= t.f) ? t.pb * t.b : 0;        // byxf, features possibly padded
    if (t.px == 1) return (t.py == t.x && t.pf == t.py * t.y && t.pb == t.pf * t.f) ? t.pb * t.b : 0;          // bfyx
    return 0;
}
static bool eltwise_vec_supports(const void* vp)
{
    const auto& p = *(const cldnn_b200_eltwise_params*)vp;
    if (p.stride_x0 != 1 || p.stride_y0 != 1 || p.stride_x1 != 1 || p.stride_y1 != 1) return false;
    if (!same_dense(p.in0, p.out) || !same_dense(p.in1, p.out)) return false;
    if (p.act != CLDNN_B200_ACT_NONE && p.act != CLDNN_B200_ACT_RELU) return false;
    const bool half = p.in0.dtype == CLDNN_B200_F16 && p.in1.dtype == CLDNN_B200_F16 && p.out.dtype == CLDNN_B200_F16 && !p.quantization;
    const bool bytes = is_int8(p.in0.dtype) && is_int8(p.in1.dtype) && is_int8(p.out.dtype) && p.quantization;
    if (!half && !bytes) return false;
    const int64_t n = dense_elems(p.out);
    if (n <= 0 || (n * (half ? 2 : 1)) % 16) return false;
    if (bytes && p.calibration && (p.out.pf != 1 || p.out.px % 16)) return false;          // per-feature factors: 16 consecutive features per vector
    return true;
}
static int32_t eltwise_vec_prepare(cldnn_b200_ctx_impl* ctx, const void* vp, const cldnn_b200_args* a, cldnn_b200_prepared_impl* out)
{
    const cldnn_b200_eltwise_params p = *(const cldnn_b200_eltwise_params*)vp;
    if (!eltwise_vec_supports(vp)) return fail(CLDNN_B200_UNSUPPORTED_FORMAT, "eltwise_byxf: equal dense layouts, strides 1, 8-bit requantising or fp16 form, NONE / ReLU only");
    if (!a->input0 || !a->input1 || !a->output) return fail(CLDNN_B200_INVALID_ARG, "eltwise_byxf: two inputs and an output are required");
    if (p.quantization && p.calibration && !a->output_calibration_factors) return fail(CLDNN_B200_INVALID_ARG, "eltwise_byxf: calibration factors missing");
    if (((uintptr_t)a->input0 | (uintptr_t)a->input1 | (uintptr_t)a->output) & 15) return fail(CLDNN_B200_INVALID_ARG, "eltwise_byxf: buffers must be 16-byte aligned");
    const bool half = p.in0.dtype == CLDNN_B200_F16;
    const int64_t vectors = dense_elems(p.out) * (half ? 2 : 1) / 16;
    const uint4* i0 = (const uint4*)a->input0; const uint4* i1 = (const uint4*)a->input1; uint4* o = (uint4*)a->output; const float* c = a->output_calibration_factors;
    const int32_t sf = (int32_t)(p.out.pf == 1 ? p.out.px : 1);
    const int grid = grid_for(vectors, 256, ctx);
    if (half) out->fn = [=](cudaStream_t s) { eltwise_vec_kernel<true><<<grid, 256, 0, s>>>(p, i0, i1, c, o, vectors, sf); return cudaGetLastError(); };
    else out->fn = [=](cudaStream_t s) { eltwise_vec_kernel<false><<<grid, 256, 0, s>>>(p, i0, i1, c, o, vectors, sf); return cudaGetLastError(); };
    return CLDNN_B200_SUCCESS;
}
const KernelDef kdef_eltwise_byxf = {"eltwise_byxf", sizeof(cldnn_b200_eltwise_params), eltwise_vec_supports, one_tune, nullptr, eltwise_vec_prepare};

// ---------------------------------------------------------------------------------
// reorder (cl_kernels/reorder_data.cl:72-128).  Threads walk the destination in
// its own memory order so writes coalesce; a destination feature beyond the
// source's feature count is written as zero (feature padding of the new layout).
// ---------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
reorder_ref_kernel(const __grid_constant__ cldnn_b200_reorder_params p, const void* in, void* out)
{
    const int64_t total = (int64_t)p.out.b * p.out.f * p.out.y * p.out.x;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
        int b, f, y, x;
        if (p.out.pf == 1) { f = (int)(idx % p.out.f); int64_t t = idx / p.out.f; x = (int)(t % p.out.x); t /= p.out.x; y = (int)(t % p.out.y); b = (int)(t / p.out.y); }
        else if (p.out.pb == 1) { b = (int)(idx % p.out.b); int64_t t = idx / p.out.b; f = (int)(t % p.out.f); t /= p.out.f; x = (int)(t % p.out.x); y = (int)(t / p.out.x); }
        else { x = (int)(idx % p.out.x); int64_t t = idx / p.out.x; y = (int)(t % p.out.y); t /= p.out.y; f = (int)(t % p.out.f); b = (int)(t / p.out.f); }
        const int64_t oi = tidx(p.out, b, f, y, x);
        if (f >= p.in.f) { store_sat_int(out, p.out.dtype, oi, 0); continue; }
        const int64_t ii = tidx(p.in, b, f, y, x);
        if (!is_fp(p.in.dtype) && !p.has_mean) { store_sat_int(out, p.out.dtype, oi, load_as_int(in, p.in.dtype, ii)); continue; }
        float v = load_as_float(in, p.in.dtype, ii);
        if (p.has_mean) v = __fsub_rn(v, p.mean[f < 4 ? f : 3]);
        store_sat_float(out, p.out.dtype, oi, v);
    }
}
// The same between a planar layout (bfyx) and a feature-innermost one (byxf) of equal element type, 1 or 2 bytes: per image a
// transposition of features x pixels.  Walking the destination in order (the kernel above) reads one element per 32-byte sector
// of the source: 32 x 512 x 28 x 28 halves (51 MB moved) took 95 us.  Here a block moves a tile of 64 features x 64 pixels through
// shared memory, both sides in vectors along their contiguous axis: 16 bytes of features, VB bytes of pixels (16, 4 or one
// element, whatever the planes' size keeps aligned).  13 - 18 us for the same tensor, 2.9 - 4.0 TB/s; tiles are small so that one
// image still makes many blocks.
// (No early release of dependents: weights are packed with this kernel, and convolutions fetch weights before they wait.)
constexpr int kTilePitch = kTileP + 2;
template <class T, int VB, bool kToByxf>
__global__ void __launch_bounds__(256)
reorder_tile_kernel(const T* __restrict__ in, T* __restrict__ out, int F, int Fs, int HW, int64_t plane_pf, int64_t plane_pb, int64_t inner_px, int64_t inner_pb)
{
    constexpr int VP = VB / (int)sizeof(T), VF = 16 / (int)sizeof(T);          // elements per vector: planar side, byxf side
    __shared__ T tile[kTileF][kTilePitch];
    ptx::griddep_wait();
    const int f0 = blockIdx.x * kTileF, p0 = blockIdx.y * kTileP, b = blockIdx.z;
    auto planar = [&](bool load) {
        for (int i = threadIdx.x; i < kTileF * (kTileP / VP); i += 256) {
            const int f = i / (kTileP / VP), p = (i - f * (kTileP / VP)) * VP;
            if (p0 + p >= HW || (!load && f0 + f >= F)) continue;              // planes hold whole vectors
            union { T e[VP]; uint4 q[(VB + 15) / 16]; uint32_t w[(VB + 3) / 4]; } v;
            const int64_t at = b * plane_pb + (int64_t)(f0 + f) * plane_pf + p0 + p;
            if (load) {
                if (f0 + f >= F) { for (int k = 0; k < VP; ++k) v.e[k] = T(0); }
                else if (VB == 16) v.q[0] = *reinterpret_cast<const uint4*>(in + at);
                else if (VB == 4) v.w[0] = *reinterpret_cast<const uint32_t*>(in + at);
                else v.e[0] = in[at];
#pragma unroll
                for (int k = 0; k < VP; ++k) tile[f][p + k] = v.e[k];
            } else {
#pragma unroll
                for (int k = 0; k < VP; ++k) v.e[k] = tile[f][p + k];
                if (VB == 16) *reinterpret_cast<uint4*>(out + at) = v.q[0];
                else if (VB == 4) *reinterpret_cast<uint32_t*>(out + at) = v.w[0];
                else out[at] = v.e[0];
            }
        }
    };
    auto inner = [&](bool load) {
        for (int i = threadIdx.x; i < kTileP * (kTileF / VF); i += 256) {
            const int p = i / (kTileF / VF), f = (i - p * (kTileF / VF)) * VF;
            if (p0 + p >= HW || f0 + f >= (load ? F : Fs)) continue;           // (written features are in whole vectors)
            union { T e[VF]; uint4 q; } v;
            const int64_t at = b * inner_pb + (int64_t)(p0 + p) * inner_px + f0 + f;
            if (load) {
                if (f0 + f + VF <= F) {
                    v.q = *reinterpret_cast<const uint4*>(in + at);
#pragma unroll
                    for (int k = 0; k < VF; ++k) tile[f + k][p] = v.e[k];
                } else
                    for (int k = 0; k < F - (f0 + f); ++k) tile[f + k][p] = in[at + k];   // what lies behind the last feature need not belong to the tensor
            } else {
#pragma unroll
                for (int k = 0; k < VF; ++k) v.e[k] = tile[f + k][p];
                *reinterpret_cast<uint4*>(out + at) = v.q;
            }
        }
    };
    if (kToByxf) planar(true); else inner(true);
    __syncthreads();
    if (kToByxf) inner(false); else planar(false);
}

template <class T, bool kToByxf>
static std::function<cudaError_t(cudaStream_t)> reorder_tile_launch(const ReorderTilePlan& t, const void* in, void* out)
{
    auto* k = t.vector == 16 ? reorder_tile_kernel<T, 16, kToByxf> : (t.vector == 4 ? reorder_tile_kernel<T, 4, kToByxf> : reorder_tile_kernel<T, (int)sizeof(T), kToByxf>);
    const T* src = (const T*)in + t.in_offset; T* dst = (T*)out + t.out_offset;
    return [=](cudaStream_t s) {
        return launch_dependent(k, dim3(t.grid_x, t.grid_y, t.grid_z), 256, s, src, dst, t.features, t.stored, t.pixels, t.plane_pf, t.plane_pb, t.inner_px, t.inner_pb);
    };
}

// the tile kernel's launch, or an empty function when the two layouts are not its pair
static std::function<cudaError_t(cudaStream_t)> reorder_tile_form(const cldnn_b200_reorder_params& p, const void* in, void* out)
{
    ReorderTilePlan t;
    if (!reorder_tile_plan(p, (uintptr_t)in, (uintptr_t)out, t)) return {};
    if (t.element == 1) return t.to_inner ? reorder_tile_launch<uint8_t, true>(t, in, out) : reorder_tile_launch<uint8_t, false>(t, in, out);
    return t.to_inner ? reorder_tile_launch<uint16_t, true>(t, in, out) : reorder_tile_launch<uint16_t, false>(t, in, out);
}

static bool reorder_supports(const void* vp) { const auto& p = *(const cldnn_b200_reorder_params*)vp; return p.in.b == p.out.b && p.in.y == p.out.y && p.in.x == p.out.x && p.out.f >= p.in.f; }
static int32_t reorder_prepare(cldnn_b200_ctx_impl* ctx, const void* vp, const cldnn_b200_args* a, cldnn_b200_prepared_impl* out)
{
    const cldnn_b200_reorder_params p = *(const cldnn_b200_reorder_params*)vp;
    if (!a->input0 || !a->output) return fail(CLDNN_B200_INVALID_ARG, "reorder_ref: input and output are required");
    const void* in = a->input0; void* o = a->output;
    out->fn = reorder_tile_form(p, in, o);
    if (out->fn) return CLDNN_B200_SUCCESS;
    const int grid = grid_for((int64_t)p.out.b * p.out.f * p.out.y * p.out.x, 256, ctx);
    out->fn = [=](cudaStream_t s) { reorder_ref_kernel<<<grid, 256, 0, s>>>(p, in, o); return cudaGetLastError(); };
    return CLDNN_B200_SUCCESS;
}
const KernelDef kdef_reorder_ref = {"reorder_ref", sizeof(cldnn_b200_reorder_params), reorder_supports, one_tune, nullptr, reorder_prepare};

// ---------------------------------------------------------------------------------
// lrn across channels (cl_kernels/lrn_gpu_across_channel_ref.cl:26-66)
// ---------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
lrn_ref_kernel(const __grid_constant__ cldnn_b200_lrn_params p, const void* in, void* out)
{
    const int64_t total = (int64_t)p.in.b * p.in.f * p.in.y * p.in.x;
    const int pad = (p.size - 1) / 2;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
        int b, f, y, x;
        decode_bfyx(idx, p.in.f, p.in.y, p.in.x, p.in.pf == 1 && p.out.pf == 1, b, f, y, x);
        float acc = 0.f;
        for (int i = 0; i < p.size; ++i) {
            const int ff = f - pad + i; if (ff < 0 || ff >= p.in.f) continue;
            const float v = load_as_float(in, p.in.dtype, tidx(p.in, b, ff, y, x));
            acc = __fadd_rn(acc, __fmul_rn(v, v));
        }
        acc = __fadd_rn(__fmul_rn(acc, __fdiv_rn(p.alpha, (float)p.size)), p.k);
        const float v = load_as_float(in, p.in.dtype, tidx(p.in, b, f, y, x));
        store_sat_float(out, p.out.dtype, tidx(p.out, b, f, y, x), v * powf(acc, -p.beta));
    }
}
// 8 consecutive features f0 .. f0 + 7 of one pixel (`src`) normalised over a window of 5: one 128-bit load and the two neighbours on
// either side with one 32-bit load each.
__device__ __forceinline__ uint4 lrn5_f16(const __half* src, int f0, int features, float scale, float k0, float beta)
{
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(src));
    float val[12];                                               // features f0 - 2 .. f0 + 9
    {
        const __half2* h = reinterpret_cast<const __half2*>(&v);
#pragma unroll
        for (int k = 0; k < 4; ++k) { const float2 f = __half22float2(h[k]); val[2 + 2 * k] = f.x; val[3 + 2 * k] = f.y; }
        float2 lo = make_float2(0.f, 0.f), hi = make_float2(0.f, 0.f);
        if (f0 >= 2) lo = __half22float2(__ldg(reinterpret_cast<const __half2*>(src - 2)));
        if (f0 + 8 < features) hi = __half22float2(__ldg(reinterpret_cast<const __half2*>(src + 8)));
        if (f0 + 9 >= features) hi.y = 0.f;
        val[0] = lo.x; val[1] = lo.y; val[10] = hi.x; val[11] = hi.y;
    }
    float sq[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) sq[k] = val[k] * val[k];
    float pair[11];
#pragma unroll
    for (int k = 0; k < 11; ++k) pair[k] = sq[k] + sq[k + 1];
    float r[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        // (flushing a subnormal power to zero changes nothing: times a half it rounds to a half zero)
        const float e = -beta * __log2f(fmaf(pair[k] + pair[k + 2] + sq[k + 4], scale, k0));
        float w; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(w) : "f"(e));
        r[k] = val[k + 2] * w;
    }
    __half2 o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) o[k] = __floats2half2_rn(r[2 * k], r[2 * k + 1]);
    return *reinterpret_cast<const uint4*>(o);
}
// The same for fp16 in the feature-innermost (byxf) layout, window 5: a thread owns 8 consecutive features of one pixel, keeps the squares
// in fp32 and writes 8 halves; x^-beta = exp2(-beta * log2(x)) on the special-function unit (the reference's
// native_powr is as loosely specified).
__global__ void __launch_bounds__(256)
lrn_f16_byxf_kernel(const __grid_constant__ cldnn_b200_lrn_params p, const __half* __restrict__ in, __half* __restrict__ out)
{
    ptx::griddep_launch_dependents();
    const int fv = p.in.f / 8;
    const int64_t total = (int64_t)p.in.b * p.in.y * p.in.x * fv;
    const float scale = __fdiv_rn(p.alpha, (float)p.size);
    ItemWalk it; it.init(blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x, fv, p.in.x, p.in.y);
    for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < (uint32_t)total; idx += gridDim.x * blockDim.x, it.next()) {   // < 2^31 items (host check)
        const int f8 = it.f, x = it.x, y = it.y, b = it.b;
        const int f0 = f8 * 8;
        const uint4 o = lrn5_f16(in + tidx(p.in, b, f0, y, x), f0, p.in.f, scale, p.k, p.beta);
        *reinterpret_cast<uint4*>(out + tidx(p.out, b, f0, y, x)) = o;
    }
}
static bool lrn_f16_byxf_supports(const void* vp)
{
    const auto& p = *(const cldnn_b200_lrn_params*)vp;
    if (p.size != 5 || p.in.dtype != CLDNN_B200_F16 || p.out.dtype != CLDNN_B200_F16) return false;
    if (p.in.pf != 1 || p.out.pf != 1 || p.in.f % 8) return false;
    const int64_t pitches[] = {p.in.px, p.in.py, p.in.pb, p.in.offset, p.out.px, p.out.py, p.out.pb, p.out.offset};
    for (int64_t v : pitches) if (v % 8) return false;
    if ((int64_t)p.in.b * p.in.y * p.in.x * (p.in.f / 8) >= 0x7fffffffLL) return false;         // 32-bit item index
    return true;
}
static int32_t lrn_f16_byxf_prepare(cldnn_b200_ctx_impl* ctx, const void* vp, const cldnn_b200_args* a, cldnn_b200_prepared_impl* out)
{
    const cldnn_b200_lrn_params p = *(const cldnn_b200_lrn_params*)vp;
    if (!a->input0 || !a->output) return fail(CLDNN_B200_INVALID_ARG, "lrn_f16_byxf: input and output are required");
    if (((uintptr_t)a->input0 | (uintptr_t)a->output) & 15) return fail(CLDNN_B200_INVALID_ARG, "lrn_f16_byxf: buffers must be 16-byte aligned");
    const __half* in = (const __half*)a->input0; __half* o = (__half*)a->output;
    const int grid = grid_for((int64_t)p.in.b * p.in.y * p.in.x * (p.in.f / 8), 256, ctx);
    out->fn = [p, in, o, grid](cudaStream_t s) { lrn_f16_byxf_kernel<<<grid, 256, 0, s>>>(p, in, o); return cudaGetLastError(); };
    return CLDNN_B200_SUCCESS;
}

// LRN and the 3x3 stride-2 maximum behind it in one pass (AlexNet's norm + pool): apart, the normalised map is written and read back,
// 149 MB each way at 256 x 96 x 55 x 55.  A block normalises the input rows of a strip of output rows into shared memory, three
// rows at a time (each pixel once: two special-function operations per value make recomputation as dear as the traffic), and pools from
// there.  Values are rounded to half before the maximum, so the result is that of the two kernels apart, bit for bit.
__global__ void __launch_bounds__(256)
lrn_pool_f16_byxf_kernel(const __grid_constant__ cldnn_b200_lrn_pool_params p, const __half* __restrict__ in, __half* __restrict__ out, int strip)
{
    extern __shared__ uint4 s_rows[];                                // [iy % 3][x][feature / 8]
    ptx::griddep_launch_dependents();
    const cldnn_b200_tensor& ti = p.pool.in; const cldnn_b200_tensor& to = p.pool.out;
    // a thread keeps its feature vector and steps over columns: no index arithmetic per value worth mentioning
    const int fv = ti.f / 8, row_items = ti.x * fv, b = blockIdx.y;
    const int f8 = threadIdx.x % fv, x0 = threadIdx.x / fv, xs = blockDim.x / fv, f0 = f8 * 8;
    const int oy0 = blockIdx.x * strip, oy1 = min(oy0 + strip, to.y);
    const float scale = __fdiv_rn(p.lrn_alpha, (float)p.lrn_size);
    const __half* src = in + tidx(ti, b, f0, 0, x0);
    __half* dst = out + tidx(to, b, f0, 0, x0);
    for (int oy = oy0; oy < oy1; ++oy) {
        for (int iy = oy == oy0 ? 2 * oy : 2 * oy + 1; iy < 2 * oy + 3; ++iy) {          // the row above is there from the output row before
            const __half* row = src + (int64_t)iy * ti.py;
            uint4* to_row = s_rows + (iy % 3) * row_items + f8;
            if (x0 < xs)
#pragma unroll 2
                for (int x = x0; x < ti.x; x += xs) to_row[x * fv] = lrn5_f16(row + (int64_t)(x - x0) * ti.px, f0, ti.f, scale, p.lrn_k, p.lrn_beta);
        }
        __syncthreads();
        if (x0 < xs)
            for (int x = x0; x < to.x; x += xs) {
                const __half2 lowest = __half2half2(__ushort_as_half((unsigned short)0xfbffu));   // as the pooling kernel starts
                __half2 m[4] = {lowest, lowest, lowest, lowest};
                const uint4* at = s_rows + 2 * x * fv + f8;
#pragma unroll
                for (int r = 0; r < 3; ++r)
#pragma unroll
                    for (int s = 0; s < 3; ++s) {
                        const uint4 v = at[r * row_items + s * fv];
                        const __half2* h = reinterpret_cast<const __half2*>(&v);
#pragma unroll
                        for (int q = 0; q < 4; ++q) m[q] = __hmax2(m[q], h[q]);
                    }
                *reinterpret_cast<uint4*>(dst + (int64_t)oy * to.py + (int64_t)(x - x0) * to.px) = *reinterpret_cast<const uint4*>(m);
            }
        __syncthreads();
    }
}
static size_t lrn_pool_smem(const cldnn_b200_lrn_pool_params& p) { return (size_t)3 * p.pool.in.x * p.pool.in.f * 2; }
static bool lrn_pool_supports(const void* vp)
{
    const auto& p = *(const cldnn_b200_lrn_pool_params*)vp;
    const cldnn_b200_pool_params& q = p.pool;
    if (p.lrn_size != 5 || q.in.dtype != CLDNN_B200_F16 || q.out.dtype != CLDNN_B200_F16) return false;
    if (q.mode != CLDNN_B200_POOL_MAX || q.size_x != 3 || q.size_y != 3 || q.stride_x != 2 || q.stride_y != 2 || q.pad_x || q.pad_y || q.act != CLDNN_B200_ACT_NONE) return false;
    if (q.in.pf != 1 || q.out.pf != 1 || q.in.f % 8 || q.in.f < 8 || q.in.f > 2048 || q.in.f != q.out.f || q.in.b != q.out.b || q.in.b < 1 || q.in.b > 65535) return false;
    if (q.out.x < 1 || q.out.y < 1 || 2 * q.out.x + 1 > q.in.x || 2 * q.out.y + 1 > q.in.y) return false;   // windows inside the map
    const int64_t pitches[] = {q.in.px, q.in.py, q.in.pb, q.in.offset, q.out.px, q.out.py, q.out.pb, q.out.offset};
    for (int64_t v : pitches) if (v % 8) return false;
    return lrn_pool_smem(p) <= 64 * 1024;
}
static int32_t lrn_pool_prepare(cldnn_b200_ctx_impl* ctx, const void* vp, const cldnn_b200_args* a, cldnn_b200_prepared_impl* out)
{
    const cldnn_b200_lrn_pool_params p = *(const cldnn_b200_lrn_pool_params*)vp;
    if (!lrn_pool_supports(vp)) return fail(CLDNN_B200_UNSUPPORTED_FORMAT, "lrn_pool_f16_byxf: fp16 byxf, up to 2048 features, LRN window 5, 3x3 stride-2 maximum without padding");
    if (!a->input0 || !a->output) return fail(CLDNN_B200_INVALID_ARG, "lrn_pool_f16_byxf: input and output are required");
    if (((uintptr_t)a->input0 | (uintptr_t)a->output) & 15) return fail(CLDNN_B200_INVALID_ARG, "lrn_pool_f16_byxf: buffers must be 16-byte aligned");
    const __half* in = (const __half*)a->input0; __half* o = (__half*)a->output;
    const size_t smem = lrn_pool_smem(p);
    B200_CUDA(raise_smem_limit((const void*)lrn_pool_f16_byxf_kernel, ctx->device, smem));
    // the strip with the least work per wave of resident blocks: 2 * strip + 1 input rows each
    const int64_t per_sm = std::min<int64_t>(8, (int64_t)(ctx->prop.sharedMemPerMultiprocessor / (smem + 1024))), slots = per_sm * ctx->prop.multiProcessorCount;
    int strip = 1; int64_t best = 0;
    for (int r = 1; r <= p.pool.out.y; ++r) {
        const int64_t blocks = (int64_t)p.pool.out.b * ((p.pool.out.y + r - 1) / r), cost = (blocks + slots - 1) / slots * (2 * r + 1);
        if (r == 1 || cost < best) { best = cost; strip = r; }
    }
    const dim3 grid((unsigned)((p.pool.out.y + strip - 1) / strip), (unsigned)p.pool.out.b);
    out->fn = [p, in, o, grid, smem, strip](cudaStream_t s) { lrn_pool_f16_byxf_kernel<<<grid, 256, smem, s>>>(p, in, o, strip); return cudaGetLastError(); };
    return CLDNN_B200_SUCCESS;
}
const KernelDef kdef_lrn_pool_f16_byxf = {"lrn_pool_f16_byxf", sizeof(cldnn_b200_lrn_pool_params), lrn_pool_supports, one_tune, nullptr, lrn_pool_prepare};

static bool lrn_supports(const void* vp) { const auto& p = *(const cldnn_b200_lrn_params*)vp; return p.size >= 1 && is_fp(p.in.dtype); }
static int32_t lrn_prepare(cldnn_b200_ctx_impl* ctx, const void* vp, const cldnn_b200_args* a, cldnn_b200_prepared_impl* out)
{
    const cldnn_b200_lrn_params p = *(const cldnn_b200_lrn_params*)vp;
    if (!a->input0 || !a->output) return fail(CLDNN_B200_INVALID_ARG, "lrn_ref: input and output are required");
    const void* in = a->input0; void* o = a->output;
    const int grid = grid_for((int64_t)p.in.b * p.in.f * p.in.y * p.in.x, 256, ctx);
    out->fn = [=](cudaStream_t s) { lrn_ref_kernel<<<grid, 256, 0, s>>>(p, in, o); return cudaGetLastError(); };
    return CLDNN_B200_SUCCESS;
}
const KernelDef kdef_lrn_ref = {"lrn_ref", sizeof(cldnn_b200_lrn_params), lrn_supports, one_tune, nullptr, lrn_prepare};
const KernelDef kdef_lrn_f16_byxf = {"lrn_f16_byxf", sizeof(cldnn_b200_lrn_params), lrn_f16_byxf_supports, one_tune, nullptr, lrn_f16_byxf_prepare};

// ---------------------------------------------------------------------------------
// standalone activation (cl_kernels/activation_ref.cl)
// ---------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
activation_ref_kernel(const __grid_constant__ cldnn_b200_activation_params p, const void* in, void* out)
{
    const int64_t total = (int64_t)p.in.b * p.in.f * p.in.y * p.in.x;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (int64_t)gridDim.x * blockDim.x) {
        int x = (int)(idx % p.in.x); int64_t t = idx / p.in.x;
        int y = (int)(t % p.in.y); t /= p.in.y;
        int f = (int)(t % p.in.f); int b = (int)(t / p.in.f);
        const int64_t ii = tidx(p.in, b, f, y, x), oi = tidx(p.out, b, f, y, x);
        if (is_fp(p.in.dtype)) store_sat_float(out, p.out.dtype, oi, act_float(p.act, load_as_float(in, p.in.dtype, ii), p.act_m, p.act_n));
        else store_sat_int(out, p.out.dtype, oi, act_int(p.act, load_as_int(in, p.in.dtype, ii), p.act_m, p.act_n));
    }
}
static bool activation_supports(const void*) { return true; }
static int32_t activation_prepare(cldnn_b200_ctx_impl* ctx, const void* vp, const cldnn_b200_args* a, cldnn_b200_prepared_impl* out)
{
    const cldnn_b200_activation_params p = *(const cldnn_b200_activation_params*)vp;
    if (!a->input0 || !a->output) return fail(CLDNN_B200_INVALID_ARG, "activation_ref: input and output are required");
    const void* in = a->input0; void* o = a->output;
    const int grid = grid_for((int64_t)p.in.b * p.in.f * p.in.y * p.in.x, 256, ctx);
    out->fn = [=](cudaStream_t s) { activation_ref_kernel<<<grid, 256, 0, s>>>(p, in, o); return cudaGetLastError(); };
    return CLDNN_B200_SUCCESS;
}
const KernelDef kdef_activation_ref = {"activation_ref", sizeof(cldnn_b200_activation_params), activation_supports, one_tune, nullptr, activation_prepare};

}  // namespace b200
