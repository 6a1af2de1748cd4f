// conv_featrows: convolution with the output FEATURES as the rows of the tensor-core tile and the output pixels as its
// columns, the reduction split over the CTAs of a cluster.  It serves what the pixel-row kernels (conv_i8_tc, conv_f16_tc:
// 128 pixels x up to 256 features per tile, one CTA per tile) cannot spread over the device: inner products (one "pixel" per
// image) and the deep layers of small batches, where a handful of tiles each walk a reduction of many steps while most SMs
// idle.  An inner product reads its weights once and does little else, so what bounds it is how many SMs stream weights: 4096
// outputs are 32 feature tiles, times a split of up to 8.
//   Tile: 128 features (weights, K-major rows as packed for the pixel-row kernels) x `cols` pixels (16 .. 256).  Each of the
//   `split` CTAs of a cluster accumulates its share of the (tap, channel chunk) steps in tensor memory, writes its 128 x cols
//   partial sums to its own shared memory, and after a cluster barrier every CTA adds up and finishes its share of the columns,
//   reading the others' partial sums through distributed shared memory (no workspace in HBM, no atomics; a fixed order of the
//   fp32 sums).  Four consecutive features of one pixel per thread: a warp stores 128 features of a pixel contiguously.
//   Warp 0 loads, warp 1 issues the tensor-core instructions, all eight warps run the epilogue.
// Launched with programmatic stream serialisation: where the parameters are constants of the network (early_params) the weights of the
// first stages are requested and the epilogue's constants read before the previous kernel has finished; activations only after
// griddepcontrol.wait.
#include <cuda.h>
#include <algorithm>
#include <mutex>
#include "conv_featrows.hpp"
#include "conv_tile_cost.hpp"
#include "conv_epilogue.cuh"

namespace b200 {

namespace {

constexpr int kRows = 128;                    // features per tile = TMEM lanes
constexpr int kFrThreads = 256;
constexpr int kFrMaxStages = 12;
constexpr uint32_t kFrErr = 0xa0u;
enum { FR_FLAT = 0, FR_IM2COL = 1, FR_TILED = 2 };

struct alignas(64) FrParams {
    CUtensorMap tmW, tmX[kGroupMaps];         // activations: [0], or one per group (group_maps)
    int32_t mode, N, P, Q;
    int32_t kw, stride_x, stride_y, pad_x, pad_y, dil_x, dil_y;
    int32_t bk, chunks, k_steps, split;
    int32_t n_tiles, cols, valid_cols;        // pixel tiles, columns per tile, columns of a tile that can hold pixels
    int32_t bw, bh, bb, tiles_w, tiles_h;
    uint32_t M_total;
    int32_t stages, a_stage_bytes, b_stage_bytes, tx_bytes, ring_bytes;
    uint32_t sbo, layout_type, idesc, tmem_cols;
    int32_t ofm;
    int32_t early_params;                     // weights and per-feature constants may be read before the previous kernel has ended
    int32_t group_tiles, group_ch;            // grouped: feature tiles per group (0: one group), its input features
    int32_t group_maps;                       // grouped fp16 whose slices end inside a chunk: a tensor map per group
    int64_t out_px, out_py, out_pb, out_off, el_px, el_py, el_pb, el_off;
    int32_t el_sx, el_sy;
    void* out; const void* eltw; const void* bias; const float* quant; const float* calib; const float* ecal;
    uint32_t* status;
    EpiCfg epi;
};

struct FrAux {
    uint64_t full[kFrMaxStages], empty[kFrMaxStages];
    uint64_t tmem_full;
    uint32_t tmem_base, abort;
};

__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ uint4 ld_cluster_v4(uint32_t addr)
{
    uint4 v;
    asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}
template <bool kF16> __device__ __forceinline__ uint32_t add_acc(uint32_t a, uint32_t b)
{
    return kF16 ? __float_as_uint(__uint_as_float(a) + __uint_as_float(b)) : a + b;
}

// the partial sums of four features of one column, added up over the CTAs of the cluster
template <bool kF16, int S>
__device__ __forceinline__ uint4 gather_sums(const uint32_t (&peer)[8], uint32_t off)
{
    uint4 v[S];
#pragma unroll
    for (int r = 0; r < S; ++r) v[r] = ld_cluster_v4(peer[r] + off);
    uint4 s = v[0];
#pragma unroll
    for (int r = 1; r < S; ++r) {
        s.x = add_acc<kF16>(s.x, v[r].x); s.y = add_acc<kF16>(s.y, v[r].y);
        s.z = add_acc<kF16>(s.z, v[r].z); s.w = add_acc<kF16>(s.w, v[r].w);
    }
    return s;
}

// pixel of column `col` of pixel tile `tile`; false: the column holds no pixel
__device__ __forceinline__ bool column_pixel(const FrParams& P, int tile, int col, int& n, int& p, int& q)
{
    if (P.mode == FR_TILED) {
        const int tw = tile % P.tiles_w, t2 = tile / P.tiles_w;
        const int th = t2 % P.tiles_h, tb = t2 / P.tiles_h;
        const int rw = col % P.bw, r2 = col / P.bw;
        q = tw * P.bw + rw; p = th * P.bh + r2 % P.bh; n = tb * P.bb + r2 / P.bh;
        return r2 / P.bh < P.bb && q < P.Q && p < P.P && n < P.N;
    }
    const uint32_t m = (uint32_t)tile * (uint32_t)P.cols + (uint32_t)col, pq = (uint32_t)(P.P * P.Q);
    if (m >= P.M_total) return false;
    n = (int)(m / pq); const int r = (int)(m - (uint32_t)n * pq);
    p = r / P.Q; q = r - p * P.Q;
    return true;
}

template <bool kF16>
__global__ void __launch_bounds__(kFrThreads)
conv_featrows_kernel(const __grid_constant__ FrParams P)
{
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* smem = smem_raw + (base - raw);
    const uint32_t b_base = base + (uint32_t)(P.stages * P.a_stage_bytes);
    FrAux* aux = reinterpret_cast<FrAux*>(smem + P.ring_bytes);
    volatile uint32_t* s_abort = &aux->abort;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int split = P.split;
    const uint32_t rank = split > 1 ? cluster_ctarank() : 0u;
    const int tile = (int)blockIdx.x / split;
    const int m_tile = tile / P.n_tiles, n_tile = tile - m_tile * P.n_tiles;

    if (threadIdx.x == 0) {
        for (int s = 0; s < P.stages; ++s) { mbar_init(smem_u32(&aux->full[s]), 1); mbar_init(smem_u32(&aux->empty[s]), 1); }
        mbar_init(smem_u32(&aux->tmem_full), 1);
        aux->abort = 0u;
        mbar_fence_init();
        prefetch_tensormap(&P.tmW); prefetch_tensormap(&P.tmX[P.group_maps ? m_tile / P.group_tiles : 0]);
    }
    if (warp == 1) { tmem_alloc(smem_u32(&aux->tmem_base), P.tmem_cols); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = aux->tmem_base;
    griddep_launch_dependents();

    // constants of the epilogue: fetched under the previous kernel's tail, unless that kernel may be computing them, and the main loop
    if (!P.early_params) griddep_wait();
    const EpiCfg& c = P.epi;
    const int f = m_tile * kRows + lane * 4;                         // this thread's four features
    const int nf = min(4, P.ofm - f);
    int32_t bi[4] = {0, 0, 0, 0}; float bf[4] = {0.f, 0.f, 0.f, 0.f}, qv[4], cv[4], ev[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const bool v = j < nf;
        if (v && c.bias_dtype != CLDNN_B200_NONE) { if (kF16 || c.bias_dtype == CLDNN_B200_F32) bf[j] = load_as_float(P.bias, c.bias_dtype, f + j); else bi[j] = load_as_int(P.bias, c.bias_dtype, f + j); }
        qv[j] = (!kF16 && v && c.quantization) ? P.quant[f + j] : 1.f;
        cv[j] = (!kF16 && v && c.calibration) ? P.calib[f + j] : 1.f;
        ev[j] = (!kF16 && v && c.eltw_calibration) ? P.ecal[f + j] : 1.f;
    }

    const int k0 = (int)((int64_t)P.k_steps * (int)rank / split), k1 = (int)((int64_t)P.k_steps * ((int)rank + 1) / split);
    const int steps = k1 - k0;
    if (warp == 0) {
        // ------------------------------ TMA producer ------------------------------
        const bool leader = elect_one();
        const int bke = kF16 ? P.bk >> 1 : P.bk;                     // elements per chunk
        const int pre = steps < P.stages ? steps : P.stages;
        auto load_w = [&](int i, int tap, int cc) {
            const uint32_t full = smem_u32(&aux->full[i % P.stages]);
            mbar_expect_tx(full, (uint32_t)P.tx_bytes);
            tma_load_3d(base + (uint32_t)(i % P.stages) * (uint32_t)P.a_stage_bytes, &P.tmW, full, cc * bke, tap, m_tile * kRows);
        };
        int tap = k0 / P.chunks, cc = k0 - tap * P.chunks;
        if (leader) {
            int t = tap, c = cc;
            for (int i = 0; i < pre; ++i) { load_w(i, t, c); if (++c == P.chunks) { c = 0; ++t; } }
        }
        griddep_wait();
        int c_w = 0, c_h = 0, c_n = 0;
        if (P.mode == FR_IM2COL) {
            int n = 0, p = 0, q = 0; column_pixel(P, n_tile, 0, n, p, q);
            c_w = q * P.stride_x - P.pad_x; c_h = p * P.stride_y - P.pad_y; c_n = n;
        } else if (P.mode == FR_TILED) {
            const int tw = n_tile % P.tiles_w, t2 = n_tile / P.tiles_w;
            c_w = tw * P.bw - P.pad_x; c_h = (t2 % P.tiles_h) * P.bh - P.pad_y; c_n = (t2 / P.tiles_h) * P.bb;
        }
        const int group = P.group_tiles ? m_tile / P.group_tiles : 0, g0 = group * P.group_ch;
        const CUtensorMap* tx = P.tmX + (P.group_maps ? group : 0);
        int r = tap / P.kw, s = tap - r * P.kw;
        int issued = pre; bool ok = true;
        for (int i = 0; i < steps; ++i) {
            const int st = i % P.stages;
            if (i >= pre) {
                if (!__all_sync(0xffffffffu, mbar_wait_lean(smem_u32(&aux->empty[st]), (uint32_t)(i / P.stages - 1) & 1u, s_abort, P.status, kFrErr))) { ok = false; break; }
                if (leader) load_w(i, tap, cc);
                issued = i + 1;
            }
            if (leader) {
                const uint32_t full = smem_u32(&aux->full[st]), dst = b_base + (uint32_t)st * (uint32_t)P.b_stage_bytes;
                if (P.mode == FR_FLAT) tma_load_2d(dst, tx, full, g0 + cc * bke, n_tile * P.cols);
                else if (P.mode == FR_IM2COL) tma_load_im2col_4d(dst, tx, full, g0 + cc * bke, c_w, c_h, c_n, (uint16_t)(s * P.dil_x), (uint16_t)(r * P.dil_y));
                else tma_load_4d(dst, tx, full, g0 + cc * bke, c_w + s * P.dil_x, c_h + r * P.dil_y, c_n);
            }
            if (++cc == P.chunks) { cc = 0; ++tap; if (++s == P.kw) { s = 0; ++r; } }
        }
        if (!ok) {
            // unwind: let the copies already in flight land before the CTA's shared memory goes away
            for (int i = issued > P.stages ? issued - P.stages : 0; i < issued; ++i) {
                const uint64_t t0 = globaltimer();
                while (!mbar_try_wait(smem_u32(&aux->full[i % P.stages]), (uint32_t)(i / P.stages) & 1u) && globaltimer() - t0 < 100000000ull) { }
            }
        }
    } else if (warp == 1) {
        // ------------------------------ MMA issuer --------------------------------
        const bool leader = elect_one();
        const int kk = P.bk >> 5;                                    // one instruction consumes 32 bytes of K
        griddep_wait();                                              // (the bounded waits below count their own kernel's time only)
        for (int i = 0; i < steps; ++i) {
            const int st = i % P.stages;
            if (!__all_sync(0xffffffffu, mbar_wait_lean(smem_u32(&aux->full[st]), (uint32_t)(i / P.stages) & 1u, s_abort, P.status, kFrErr + 1u))) break;
            tc_fence_after();
            if (leader) {
                const uint64_t ad = make_smem_desc(base + (uint32_t)st * (uint32_t)P.a_stage_bytes, P.sbo, P.layout_type);
                const uint64_t bd = make_smem_desc(b_base + (uint32_t)st * (uint32_t)P.b_stage_bytes, P.sbo, P.layout_type);
                for (int k = 0; k < kk; ++k) {
                    if (kF16) mma_f16_ss(tmem_base, ad + (uint64_t)(2 * k), bd + (uint64_t)(2 * k), P.idesc, (i | k) ? 1u : 0u);
                    else mma_i8_ss(tmem_base, ad + (uint64_t)(2 * k), bd + (uint64_t)(2 * k), P.idesc, (i | k) ? 1u : 0u);
                }
                tc_commit(smem_u32(&aux->empty[st]));
            }
        }
        if (leader) tc_commit(smem_u32(&aux->tmem_full));            // also after a failed wait: whatever was issued must retire
    }
    __syncwarp();
    griddep_wait();                                                  // the epilogue reads the residual and overwrites pooled buffers
    // ------------------------------ epilogue ----------------------------------
    bool ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&aux->tmem_full), 0u, s_abort, P.status, kFrErr + 2u));
    tc_fence_after();
    uint32_t* dump = reinterpret_cast<uint32_t*>(smem);              // [column][128 features]; the operand ring has been consumed
    {
        const int quad = warp & 3;                                   // TMEM lanes 32 * quad ..
        const uint32_t t_row = tmem_base + ((uint32_t)(quad * 32) << 16);
        for (int c0 = (warp >> 2) * 16; c0 < P.cols && ok; c0 += 32) {
            uint32_t r[16];
            tmem_ld_32x16(t_row + (uint32_t)c0, r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) dump[(c0 + j) * kRows + quad * 32 + lane] = r[j];
        }
    }
    tc_fence_before();
    __syncthreads();
    // Tensor memory goes back before the CTA waits for its cluster: a CTA that holds some never waits for another CTA, so kernels of
    // other streams that allocate on the same SMs (CTA pairs among them) cannot close a circle of waits with this one.
    if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, P.tmem_cols); }
    if (split > 1) cluster_sync_all();
    ok = ok && *s_abort == 0u;
    const int per = (P.valid_cols + split - 1) / split;
    const int lo = (int)rank * per, hi = min(lo + per, P.valid_cols);
    uint32_t peer[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) peer[r] = mapa_rank(smem_u32(dump), (uint32_t)(r < split ? r : 0));
    if (nf > 0 && ok)
        for (int col = lo + warp; col < hi; col += kFrThreads / 32) {
            int n, p, q;
            if (!column_pixel(P, n_tile, col, n, p, q)) continue;
            const uint32_t off = (uint32_t)(col * kRows + lane * 4) * 4u;
            uint4 s4;
            switch (split) {
                case 1: s4 = gather_sums<kF16, 1>(peer, off); break;
                case 2: s4 = gather_sums<kF16, 2>(peer, off); break;
                case 4: s4 = gather_sums<kF16, 4>(peer, off); break;
                default: s4 = gather_sums<kF16, 8>(peer, off); break;
            }
            const uint32_t sv[4] = {s4.x, s4.y, s4.z, s4.w};
            const int64_t o = P.out_off + (int64_t)n * P.out_pb + (int64_t)p * P.out_py + (int64_t)q * P.out_px + f;
            const int64_t e = P.el_off + (int64_t)n * P.el_pb + (int64_t)p * P.el_sy * P.el_py + (int64_t)q * P.el_sx * P.el_px + f;
            if (kF16) {
                __half h[4];
                uint2 ew = make_uint2(0u, 0u);
                if (c.fused_eltw) {
                    if (nf == 4) ew = *reinterpret_cast<const uint2*>(reinterpret_cast<const __half*>(P.eltw) + e);
                    else for (int j = 0; j < nf; ++j) reinterpret_cast<__half*>(&ew)[j] = reinterpret_cast<const __half*>(P.eltw)[e + j];
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float v = act_float(c.act, __uint_as_float(sv[j]) + bf[j], c.act_m, c.act_n);
                    if (c.fused_eltw) v = act_float(c.eltw_act, __half2float(__float2half_rn(v)) + __half2float(reinterpret_cast<const __half*>(&ew)[j]), c.eltw_m, c.eltw_n);
                    h[j] = __float2half_rn(v);
                }
                __half* op = reinterpret_cast<__half*>(P.out) + o;
                if (nf == 4) *reinterpret_cast<uint2*>(op) = *reinterpret_cast<const uint2*>(h);
                else for (int j = 0; j < nf; ++j) op[j] = h[j];
            } else {
                int32_t iv[4]; float fv[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float el = c.fused_eltw && j < nf ? load_as_float(P.eltw, c.eltw_dtype, e + j) : 0.f;
                    fv[j] = epi_quant(c, (int32_t)sv[j] + bi[j], qv[j], bf[j], cv[j], el, ev[j]);
                    iv[j] = c.out_dtype == CLDNN_B200_U8 ? sat_i32_from_float(fv[j], 0, 255) : sat_i32_from_float(fv[j], -128, 127);
                }
                if (nf == 4 && is_int8(c.out_dtype) && ((reinterpret_cast<uintptr_t>(P.out) + (uintptr_t)o) & 3) == 0)
                    *reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(P.out) + o) =
                        (uint32_t)(iv[0] & 0xff) | ((uint32_t)(iv[1] & 0xff) << 8) | ((uint32_t)(iv[2] & 0xff) << 16) | ((uint32_t)(iv[3] & 0xff) << 24);
                else for (int j = 0; j < nf; ++j) store_sat_float(P.out, c.out_dtype, o + j, fv[j]);
            }
        }
    // the others' partial sums are read from their shared memory: nobody leaves before everybody has finished reading
    if (split > 1) cluster_sync_all();
}

typedef CUresult (*FrEncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                    const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                    CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
typedef CUresult (*FrEncodeIm2colFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                     const int*, const int*, cuuint32_t, cuuint32_t, const cuuint32_t*, CUtensorMapInterleave,
                                     CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
FrEncodeTiledFn fr_encode_tiled = nullptr;
FrEncodeIm2colFn fr_encode_im2col = nullptr;

bool fr_entry_points()
{
    static std::once_flag once;
    std::call_once(once, [] {
        void* fn = nullptr; cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qr) == cudaSuccess && qr == cudaDriverEntryPointSuccess)
            fr_encode_tiled = (FrEncodeTiledFn)fn;
        fn = nullptr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeIm2col", &fn, cudaEnableDefault, &qr) == cudaSuccess && qr == cudaDriverEntryPointSuccess)
            fr_encode_im2col = (FrEncodeIm2colFn)fn;
        (void)cudaGetLastError();
    });
    return fr_encode_tiled && fr_encode_im2col;
}

bool fr_pixel_dense(const cldnn_b200_tensor& t) { return t.py == t.px * t.x && t.pb == t.py * t.y; }

// box of bw x bh x bb <= `cols` pixels that needs the fewest tiles
void fr_choose_box(int Q, int Pn, int N, int cols, int& bw, int& bh, int& bb)
{
    double best = -1.0; bw = bh = bb = 1;
    for (int w = 1; w <= Q && w <= cols; ++w)
        for (int h = 1; h <= Pn && w * h <= cols; ++h) {
            const int b = cols / (w * h) < N ? cols / (w * h) : N;
            const double tiles = (double)((Q + w - 1) / w) * ((Pn + h - 1) / h) * ((N + b - 1) / b);
            const double score = ((double)Q * Pn * N) / (tiles * cols) + 1e-4 * w + 1e-6 * h;
            if (score > best) { best = score; bw = w; bh = h; bb = b; }
        }
}

constexpr int kCols[kFrCols] = {16, 32, 64, 128, 256};

}  // namespace

bool fr_plan(const cldnn_b200_conv_params& p, int variant, FrPlan& pl, std::string* why, bool box)
{
    auto no = [&](const char* m) { if (why) *why = m; return false; };
    if (variant < 0 || variant >= kFrVariants) return no("unknown tuning index");
    const bool f16 = p.in.dtype == CLDNN_B200_F16;
    if (!f16 && !(p.quantization || p.calibration || p.has_o_qf)) return no("the feature-row form needs the quantised epilogue");
    if (f16 && (p.out.px % 4 || p.out.py % 4 || p.out.pb % 4 || p.out.offset % 4)) return no("the feature-row form stores four features at a time");
    pl.cols = kCols[variant / kFrSplits]; pl.split = 1 << (variant % kFrSplits);
    const int64_t es = f16 ? 2 : 1, cs = reduction_features(p) * es;
    const int bk = (int)chunk_bytes(cs);
    const int64_t steps = (int64_t)p.kh * p.kw * (cs / bk);
    if (pl.split > steps) return no("fewer reduction steps than CTAs");
    const bool pointwise = p.kh == 1 && p.kw == 1 && p.pad_x == 0 && p.pad_y == 0;
    const bool tiled_ok = (p.stride_x == 1 && p.stride_y == 1) || pointwise;
    const bool im2col_ok = p.pad_x <= 127 && p.pad_y <= 127 && (p.kw - 1) * p.dil_x <= 255 && (p.kh - 1) * p.dil_y <= 255 &&
                           p.stride_x <= 8 && p.stride_y <= 8 && (int64_t)p.in.b * p.in.pb * es >= 131072;
    if (pointwise && p.stride_x == 1 && p.stride_y == 1 && fr_pixel_dense(p.in)) pl.mode = FR_FLAT;
    else if (im2col_ok) pl.mode = FR_IM2COL;
    else if (tiled_ok) pl.mode = FR_TILED;
    else return no("neither im2col nor tiled addressing fits");
    pl.bw = pl.bh = pl.bb = 1;
    if (pl.mode == FR_TILED && box) fr_choose_box(p.out.x, p.out.y, p.out.b, pl.cols, pl.bw, pl.bh, pl.bb);
    return true;
}

// Columns: as many as there are images, up to 128 (past that the partial sums cost more than re-reading the weights, which L2
// serves); fewer while even the widest split leaves SMs idle.  Split: the widest of 8, 4, 2, 1 that gives every CTA at least one
// step (four where several pixel tiles share the weights: the cluster's exchange costs about two steps) and at most two CTAs per
// SM.  Measured over 1 .. 1024 images of the 1000- and 4096-output layers of AlexNet, VGG16 and ResNet-50 (us, pixel-row kernel as
// untuned / best of its tiles / this rule / best variant of this form): fp16 25088 -> 4096 at 16 images 181 / 105 / 37 / 37, at
// 256 images 181 / 109 / 63 / 62; fp16 9216 -> 4096 at 256 images 72 / 45 / 29 / 29; fp16 4096 -> 1000 at 16 images 27 / 23 / 9.2 /
// 9.0; 8-bit 2048 -> 1000 at 256 images 21 / 14 / 8.8 / 8.8, 8-bit 9216 -> 4096 at 1 image 39 / 31 / 10.6 / 10.6.  Where the rule
// comes out at a split of 1 there are as many tiles as SMs without it, and the pixel-row kernel's TMA stores win (fp16 4096 -> 4096
// at 1024 images: 31 against 51); at a split of 2 the two are even (30 against 29 at 512 images) or this form is ahead.
int fr_inner_product_variant(const cldnn_b200_conv_params& p)
{
    if (p.groups != 1 || p.kh != 1 || p.kw != 1 || p.in.x != 1 || p.in.y != 1 || p.pad_x || p.pad_y || p.stride_x != 1 || p.stride_y != 1) return -1;
    const int64_t cs = p.in.px * (p.in.dtype == CLDNN_B200_F16 ? 2 : 1), n = p.out.b, m_tiles = (p.ofm + kRows - 1) / kRows;
    const int64_t steps = cs / chunk_bytes(cs);
    int ci = 0;                                                      // kCols index: 16, 32, 64, 128
    auto n_tiles = [&](int i) { return (n + kCols[i] - 1) / kCols[i]; };
    auto widest = [&](int i) { int s = kFrSplits - 1; while (s > 0 && (int64_t)(n_tiles(i) > 1 ? 4 : 1) * (1 << s) > steps) --s; return s; };
    while (ci < 3 && kCols[ci] < n) ++ci;
    while (ci > 1 && (m_tiles * n_tiles(ci) << widest(ci)) < kCostSMs) --ci;
    int si = widest(ci);
    while (si > 0 && (m_tiles * n_tiles(ci) << si) > 2 * kCostSMs) --si;
    return si > 0 ? ci * kFrSplits + si : -1;
}

// time = launch + (reduction steps of a CTA + epilogue) * (1 + share * CTAs beyond one per SM); constants (us) fitted to every variant of
// the layers conv_tile_cost.hpp is fitted to (root mean square error 5 %).  More CTAs than are resident at once run in waves, which
// the other kernels do better: 256 columns leave room for one CTA per SM, and clusters of eight (four) for about 128 (144) of them
// (fp16 96 -> 256 5x5 at 27x27, 4 images, 256 columns: split of 8, 192 CTAs, 31.0 us; 128 columns, split of 4, 184 CTAs, 18.7).
double fr_cost(const cldnn_b200_conv_params& p, int& variant)
{
    variant = -1;
    struct Cost { double launch, step, step_row, col, gather, exchange_col, exchange, share; };
    constexpr Cost kI8 = {4.89, 0.351, 0.00031, 0.0064, 0.0766, 0.0132, 0.893, 0.44}, kF16 = {4.09, 0.338, 0.00039, 0.0061, 0.0844, 0.0072, 1.37, 0.30};
    const bool f16 = p.in.dtype == CLDNN_B200_F16;
    const Cost& c = f16 ? kF16 : kI8;
    const int64_t cs = reduction_features(p) * (f16 ? 2 : 1), pixels = (int64_t)p.out.b * p.out.y * p.out.x;
    const int64_t bk = chunk_bytes(cs), steps = (int64_t)p.kh * p.kw * (cs / bk), m_tiles = (p.ofm + kRows - 1) / kRows;
    double best = 0.0;
    for (int v = 0; v < kFrVariants; ++v) {
        FrPlan pl;
        const int64_t cols = kCols[v / kFrSplits], split = 1 << (v % kFrSplits), ctas = m_tiles * ((pixels + cols - 1) / cols) * split;
        const int64_t resident = (split == 8 ? 128 : (split == 4 ? 144 : kCostSMs)) * (cols == 256 ? 1 : 2);
        if (ctas > resident || !fr_plan(p, v, pl, nullptr, false)) continue;
        const double valid = (double)std::min(cols, pixels);
        const double main = (double)((steps + split - 1) / split) * (c.step + c.step_row * (double)(kRows + cols) * ((double)bk / 128.0));
        const double epi = c.col * (double)cols + c.gather * valid / (double)split + (split > 1 ? c.exchange_col * valid + c.exchange : 0.0);
        const double t = c.launch + (main + epi) * (1.0 + c.share * std::max(0.0, (double)ctas / (double)kCostSMs - 1.0));
        if (variant < 0 || t < best) { best = t; variant = v; }
    }
    return best;
}

int32_t fr_prepare(cldnn_b200_ctx_impl* ctx, const cldnn_b200_conv_params& p, const cldnn_b200_args* a, const FrPlan& pl, cldnn_b200_prepared_impl* out)
{
    if (!fr_entry_points()) return fail(CLDNN_B200_DEVICE_ERROR, "conv_featrows: the CUDA driver does not export cuTensorMapEncodeTiled/Im2col");
    const bool f16 = p.in.dtype == CLDNN_B200_F16;
    const int64_t es = f16 ? 2 : 1;
    FrParams P{};
    P.mode = pl.mode; P.N = p.out.b; P.P = p.out.y; P.Q = p.out.x;
    P.kw = p.kw; P.stride_x = p.stride_x; P.stride_y = p.stride_y; P.pad_x = p.pad_x; P.pad_y = p.pad_y; P.dil_x = p.dil_x; P.dil_y = p.dil_y;
    const int64_t cs = reduction_features(p) * es, xs = p.in.px * es;   // bytes of K per tap, pixel pitch of the activations
    P.bk = (int)chunk_bytes(cs);
    P.chunks = (int)(cs / P.bk); P.k_steps = p.kh * p.kw * P.chunks; P.split = pl.split;
    P.cols = pl.cols; P.bw = pl.bw; P.bh = pl.bh; P.bb = pl.bb;
    const int64_t pixels = (int64_t)P.N * P.P * P.Q;
    if (pixels < 1 || p.ofm < 1) return fail(CLDNN_B200_INVALID_ARG, "conv_featrows: empty output");
    if (pixels > 0x7fffff00LL) return fail(CLDNN_B200_UNSUPPORTED_SIZE, "conv_featrows: too many output pixels");
    P.M_total = (uint32_t)pixels;
    P.tiles_w = P.tiles_h = 1; P.valid_cols = P.cols;
    if (pl.mode == FR_TILED) {
        P.tiles_w = (P.Q + pl.bw - 1) / pl.bw; P.tiles_h = (P.P + pl.bh - 1) / pl.bh;
        P.n_tiles = P.tiles_w * P.tiles_h * ((P.N + pl.bb - 1) / pl.bb);
        P.valid_cols = pl.bw * pl.bh * pl.bb;
    } else P.n_tiles = (int)((pixels + P.cols - 1) / P.cols);
    const int m_tiles = (p.ofm + kRows - 1) / kRows;
    const int64_t ctas = (int64_t)m_tiles * P.n_tiles * P.split;
    if (ctas > 0x7fffffffLL) return fail(CLDNN_B200_UNSUPPORTED_SIZE, "conv_featrows: too many tiles");
    P.a_stage_bytes = kRows * P.bk; P.b_stage_bytes = (P.cols * P.bk + 1023) / 1024 * 1024;
    P.tx_bytes = P.a_stage_bytes + P.valid_cols * P.bk;
    P.sbo = 8u * (uint32_t)P.bk; P.layout_type = P.bk == 128 ? 2u : (P.bk == 64 ? 4u : 6u);
    // instruction descriptor: A = weights (s8), B = activations (u8 / s8), s32 accumulate; or f16 x f16 -> f32
    P.idesc = f16 ? (1u << 4) : ((2u << 4) | (1u << 7) | ((p.in.dtype == CLDNN_B200_U8 ? 0u : 1u) << 10));
    P.idesc |= ((uint32_t)(P.cols >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24);
    P.tmem_cols = (uint32_t)(P.cols < 32 ? 32 : P.cols);
    P.ofm = p.ofm; P.early_params = p.constant_params;
    if (p.groups > 1) { P.group_tiles = p.ofm / p.groups / kRows; P.group_ch = p.ifm; P.group_maps = slices_overhang(p); }
    const cldnn_b200_tensor& et = p.in_out_opt ? p.out : p.eltw;
    P.out_px = p.out.px; P.out_py = p.out.py; P.out_pb = p.out.pb; P.out_off = p.out.offset;
    if (p.fused_eltw) {
        P.el_px = et.px; P.el_py = et.py; P.el_pb = et.pb; P.el_off = et.offset;
        P.el_sx = p.in_out_opt ? 1 : p.eltw_stride_x; P.el_sy = p.in_out_opt ? 1 : p.eltw_stride_y;
    }
    P.out = a->output; P.eltw = p.in_out_opt ? a->output : a->input1; P.bias = a->bias;
    P.quant = a->weights_quantization_factors; P.calib = a->output_calibration_factors; P.ecal = a->eltw_output_calibration_factors;
    P.status = ctx->d_status; P.epi = make_epi_cfg(p);

    // Operand ring: every step of a CTA in flight at once where that fits.  More CTAs than SMs: two share an SM.  Clusters of four or
    // eight do not fill a GPC evenly, so with one CTA per SM a part of them would wait for a second wave well before the SMs run
    // out (8-bit 512 -> 512 3x3 at 4 images, 16 clusters of eight, ring of five 24 KiB stages: 17.2 us against 10.1 in twice as many CTAs).
    const size_t dump = (size_t)P.cols * kRows * 4, stage = (size_t)P.a_stage_bytes + P.b_stage_bytes;
    const size_t max_smem = (size_t)ctx->prop.sharedMemPerBlockOptin, other = 1024 + sizeof(FrAux);
    const int64_t alone = P.split >= 4 ? ctx->prop.multiProcessorCount / 2 : ctx->prop.multiProcessorCount;
    size_t budget = ctas > alone ? (ctx->prop.sharedMemPerMultiprocessor / 2) - 2048 : max_smem;
    if (budget < other + dump || budget < other + 2 * stage) budget = max_smem;
    if (budget < other + dump || budget < other + 2 * stage) return fail(CLDNN_B200_OUT_OF_RESOURCES, "conv_featrows: not enough shared memory");
    const int most = (P.k_steps + P.split - 1) / P.split;
    int stages = (int)((budget - other) / stage);
    if (stages > kFrMaxStages) stages = kFrMaxStages;
    if (stages > most) stages = most;
    P.stages = stages;
    P.ring_bytes = (int32_t)((stages * stage > dump ? stages * stage : dump) + 15) / 16 * 16;
    const size_t smem = other + P.ring_bytes;

    const CUtensorMapDataType dt = f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8;
    const CUtensorMapSwizzle sw = P.bk == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : (P.bk == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
    const cuuint32_t bke = (cuuint32_t)(P.bk / es);
    void* in_ptr = (char*)const_cast<void*>(a->input0) + p.in.offset * es;
    CUresult cr;
    auto encode_x = [&](CUtensorMap* tm, cuuint64_t features) -> int32_t {      // `features`: where the pixels' reduction ends
        if (pl.mode == FR_FLAT) {
            cuuint64_t dims[2] = {features, (cuuint64_t)P.M_total}; cuuint64_t strides[1] = {(cuuint64_t)xs};
            cuuint32_t box[2] = {bke, (cuuint32_t)P.cols}; cuuint32_t one[2] = {1, 1};
            cr = fr_encode_tiled(tm, dt, 2, in_ptr, dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        } else if (pl.mode == FR_IM2COL) {
            cuuint64_t dims[4] = {features, (cuuint64_t)p.in.x, (cuuint64_t)p.in.y, (cuuint64_t)p.in.b};
            cuuint64_t strides[3] = {(cuuint64_t)xs, (cuuint64_t)(p.in.py * es), (cuuint64_t)(p.in.pb * es)};
            int lower[2] = {-p.pad_x, -p.pad_y};
            int upper[2] = {p.pad_x - (p.kw - 1) * p.dil_x, p.pad_y - (p.kh - 1) * p.dil_y};
            // the box of base pixels must produce exactly Q x P positions per image
            const int q_tm = (p.in.x + upper[0] - lower[0] - 1) / p.stride_x + 1, p_tm = (p.in.y + upper[1] - lower[1] - 1) / p.stride_y + 1;
            if (q_tm != P.Q || p_tm != P.P) return fail(CLDNN_B200_UNSUPPORTED_SIZE, "conv_featrows: im2col traversal does not match the output size");
            cuuint32_t step[4] = {1, (cuuint32_t)p.stride_x, (cuuint32_t)p.stride_y, 1};
            cr = fr_encode_im2col(tm, dt, 4, in_ptr, dims, strides, lower, upper, bke, (cuuint32_t)P.cols, step, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        } else {
            const int sx = p.stride_x, sy = p.stride_y;                  // a pointwise strided convolution reads a strided view of the input
            const bool view = sx != 1 || sy != 1;
            cuuint64_t dims[4] = {features, (cuuint64_t)(view ? P.Q : p.in.x), (cuuint64_t)(view ? P.P : p.in.y), (cuuint64_t)p.in.b};
            cuuint64_t strides[3] = {(cuuint64_t)(xs * sx), (cuuint64_t)(p.in.py * sy * es), (cuuint64_t)(p.in.pb * es)};
            cuuint32_t box[4] = {bke, (cuuint32_t)pl.bw, (cuuint32_t)pl.bh, (cuuint32_t)pl.bb}; cuuint32_t one[4] = {1, 1, 1, 1};
            cr = fr_encode_tiled(tm, dt, 4, in_ptr, dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        }
        if (cr != CUDA_SUCCESS) return fail(CLDNN_B200_DEVICE_ERROR, "conv_featrows: activation tensor map rejected by the driver (CUresult " + std::to_string((int)cr) + ")");
        return CLDNN_B200_SUCCESS;
    };
    for (int g = 0; g < (P.group_maps ? p.groups : 1); ++g)
        if (const int32_t st = encode_x(&P.tmX[g], (cuuint64_t)(P.group_maps ? (g + 1) * p.ifm : p.in.px))) return st;
    {
        cuuint64_t dims[3] = {(cuuint64_t)p.w_px, (cuuint64_t)(p.kh * p.kw), (cuuint64_t)p.ofm};
        cuuint64_t strides[2] = {(cuuint64_t)(p.w_px * es), (cuuint64_t)(p.w_po * es)};
        cuuint32_t box[3] = {bke, 1, (cuuint32_t)kRows}; cuuint32_t one[3] = {1, 1, 1};
        cr = fr_encode_tiled(&P.tmW, dt, 3, (char*)const_cast<void*>(a->weights) + p.w_offset * es, dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (cr != CUDA_SUCCESS) return fail(CLDNN_B200_DEVICE_ERROR, "conv_featrows: weights tensor map rejected by the driver (CUresult " + std::to_string((int)cr) + ")");
    }
    const void* fn = f16 ? (const void*)conv_featrows_kernel<true> : (const void*)conv_featrows_kernel<false>;
    B200_CUDA(raise_smem_limit(fn, ctx->device, smem));
    const unsigned grid = (unsigned)ctas;
    out->fn = [P, fn, grid, smem](cudaStream_t s) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(grid); cfg.blockDim = dim3(kFrThreads); cfg.dynamicSmemBytes = smem; cfg.stream = s;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr; cfg.numAttrs = 1;
        if (P.split > 1) {
            attr[1].id = cudaLaunchAttributeClusterDimension;
            attr[1].val.clusterDim.x = (unsigned)P.split; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
            cfg.numAttrs = 2;
        }
        void* args[1] = {const_cast<FrParams*>(&P)};
        return cudaLaunchKernelExC(&cfg, fn, args);
    };
    out->launches = 1;
    return CLDNN_B200_SUCCESS;
}

}  // namespace b200
