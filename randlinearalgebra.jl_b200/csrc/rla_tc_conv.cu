// rla_tc_conv.cu -- FP32-accurate tensor-core products whose large operand is split into BF16 terms
// inside the kernel.
//
// C = alpha * op(A) * B + beta * C with three BF16 terms per operand (t0 = bf16(x), t1 = bf16(x - t0),
// ...) and FP64 accumulation across chunks of four k-blocks, the products and their order as in
// tc_gemm_f64acc_kernel (rla_tc.cu).  There the terms of A come from HBM: splitting reads 4 bytes
// and writes 6 per element, and the product reads the 6 again.  Here four converter warps
// copy A's Float32 tile ahead with cp.async (three k-blocks of 16 KB), turn it into the
// terms and store them where TMA would have put them (64-byte swizzle), so A is read once, at any
// alignment.  B, the small operand, is split beforehand and loaded by TMA.
//
// Warps: 0 TMA producer of B, 1 MMA issuer, 2 TMEM allocator, 4..11 chunk drain / epilogue (lane
// quarter by warp mod 4, 32 of the 64 columns each), 12..15 converters.  A tile is 128 x 64.
// Bound by the converters' chain per k-block (copy, convert, store, proxy fence, arrive; four warps):
// the tensor pipe is 18 % and the ALU pipe 25 % busy at 65536 x 1024 x 128.
#include "rla_internal.cuh"
#include "rla_kernels.cuh"
#include "rla_tc.cuh"
#include "rla_tc_ptx.cuh"

namespace rla {

constexpr int CV_THREADS = 512, CV_BN = 64, CV_CHUNK = 4, CV_RAW = 4, CV_EPI_WARPS = 8;
constexpr uint32_t CV_RAW_BYTES = TC_BM * TC_BK * 4;  // 16 KB per k-block of A
constexpr uint32_t CV_B_BYTES = CV_BN * TC_BK * 2;
constexpr int NT = 3;  // BF16 terms per operand
constexpr uint32_t CV_TMEM_COLS = 512, CV_STAGE_BYTES = NT * (TC_A_BYTES + CV_B_BYTES);

struct ConvArgs {
    const float *A;  // a_kmajor: element (m, k) at A[k + m*lda]; else at A[m + k*lda]
    int64_t lda;
    int a_vec;       // every 8-element group of A starts on 16 bytes
    int M, N, K;
    void *out;  // element (m, n) at out[m*rs + n*cs]
    int64_t rs, cs;
    int out_f64;
    double alpha, beta;  // beta: read and scaled when beta_on
    int beta_on;
    int stages;
    int *status;
    uint64_t wait_ns;
};

__device__ __forceinline__ void cp_async_zfill(uint32_t dst, const void *src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async4_zfill(uint32_t dst, const void *src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// Converter thread t of 128: four groups of 8 elements of each k-block, in the order in which
// consecutive lanes read consecutive memory.  A group's raw values stay private to the thread,
// so waiting for its own copies is enough.
template <int AK>
__device__ __forceinline__ void conv_warps(const ConvArgs &p, int t, uint32_t raw, unsigned char *raw_gen,
                                           unsigned char *stage_gen, int m0, int kb0, int nkb, uint32_t empty0,
                                           uint32_t afull0) {
    const int lane = t & 31, c = t & 3;
    // A group keeps its rows through all k-blocks: past the last row of A its place in every stage is
    // zeroed once, and it is neither copied nor converted.
    auto off = [&](int u) {  // in the tile: 64-byte rows (of box u when A is not K-major)
        const int row = AK ? u * 32 + (t >> 2) : t >> 2;
        return (AK ? 0u : (uint32_t)u * 2048u) + (uint32_t)row * 64u + (uint32_t)((c ^ ((row >> 1) & 3)) << 4);
    };
    auto live = [&](int u) { return (AK ? m0 + u * 32 + (t >> 2) : m0 + 32 * u + 8 * c) < p.M; };
#pragma unroll
    for (int u = 0; u < 4; ++u)
        if (!live(u))
            for (int s = 0; s < p.stages; ++s)
#pragma unroll
                for (int q = 0; q < NT; ++q)
                    *reinterpret_cast<uint4 *>(stage_gen + (size_t)s * CV_STAGE_BYTES + (size_t)q * TC_A_BYTES + off(u)) =
                        make_uint4(0, 0, 0, 0);
    auto issue = [&](int kb) {
        if (kb < nkb) {
            const int k0 = (kb0 + kb) * TC_BK;
            const uint32_t slot = raw + (uint32_t)(kb % CV_RAW) * CV_RAW_BYTES + (uint32_t)t * 16u;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (!live(u)) continue;
                const int m = AK ? m0 + u * 32 + (t >> 2) : m0 + 32 * u + 8 * c;
                const int k = AK ? k0 + 8 * c : k0 + (t >> 2);
                const int valid = AK ? (m < p.M ? min(8, p.K - k) : 0) : (k < p.K ? min(8, p.M - m) : 0);
                const float *src = valid > 0 ? p.A + (AK ? k + (int64_t)m * p.lda : m + (int64_t)k * p.lda) : p.A;
                const uint32_t d = slot + (uint32_t)u * 4096u;
                if (p.a_vec) {
                    cp_async_zfill(d, src, 4 * max(0, min(4, valid)));
                    cp_async_zfill(d + 2048u, valid > 4 ? src + 4 : src, 4 * max(0, valid - 4));
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        cp_async4_zfill(d + (uint32_t)(i >> 2) * 2048u + (uint32_t)(i & 3) * 4u, i < valid ? src + i : src,
                                        i < valid ? 4 : 0);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int i = 0; i < CV_RAW - 1; ++i) issue(i);
    for (int kb = 0; kb < nkb; ++kb) {
        issue(kb + CV_RAW - 1);
        const int s = kb % p.stages;
        const uint32_t ph = (uint32_t)(kb / p.stages) & 1u;
        if (!__all_sync(FULL, mbar_wait(empty0 + 8u * (uint32_t)s, ph ^ 1u, p.status, p.wait_ns))) break;
        asm volatile("cp.async.wait_group %0;" ::"n"(CV_RAW - 1) : "memory");
        const unsigned char *slot = raw_gen + (size_t)(kb % CV_RAW) * CV_RAW_BYTES + t * 16;
        unsigned char *st = stage_gen + (size_t)s * CV_STAGE_BYTES;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (!live(u)) continue;
            const float4 a = *reinterpret_cast<const float4 *>(slot + u * 4096);
            const float4 b = *reinterpret_cast<const float4 *>(slot + u * 4096 + 2048);
            const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
            uint4 o[NT];
            split_terms8<NT>(v, o);
#pragma unroll
            for (int q = 0; q < NT; ++q)
                *reinterpret_cast<uint4 *>(st + (size_t)q * TC_A_BYTES + off(u)) = o[q];
        }
        // the MMAs read the tile through the async proxy
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(afull0 + 8u * (uint32_t)s) : "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// The 128 x 64 tile (m0, n0) over k-blocks kb0 .. kb0 + nkb - 1.
__device__ __forceinline__ void conv_cta(const CUtensorMap *mb, const ConvArgs &p, int a_kmajor, int m0, int n0, int kb0,
                                         int nkb) {
    extern __shared__ unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t raw0 = smem_u32(smem_raw);
    const uint32_t base = (raw0 + 1023u) & ~1023u;
    unsigned char *gen = smem_raw + (base - raw0);
    const uint32_t ring = base + (uint32_t)p.stages * CV_STAGE_BYTES;
    const uint32_t bars = ring + CV_RAW * CV_RAW_BYTES;
    const uint32_t afull0 = bars, bfull0 = bars + 64u, empty0 = bars + 128u;  // up to 8 stages each
    auto accf_bar = [&](int x) { return bars + 192u + 8u * (uint32_t)x; };
    auto acce_bar = [&](int x) { return bars + 208u + 8u * (uint32_t)x; };
    const uint32_t done_bar = bars + 224u, tmem_slot = bars + 232u;
    volatile uint32_t *tmem_slot_ptr = reinterpret_cast<volatile uint32_t *>(gen + (tmem_slot - base));
    const int nchunks = (nkb + CV_CHUNK - 1) / CV_CHUNK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(afull0 + 8u * s, 4);
            mbar_init(bfull0 + 8u * s, 1);
            mbar_init(empty0 + 8u * s, 1);
        }
        for (int x = 0; x < 2; ++x) {
            mbar_init(accf_bar(x), 1);
            mbar_init(acce_bar(x), CV_EPI_WARPS);
        }
        mbar_init(done_bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
#pragma unroll
        for (int q = 0; q < NT; ++q)
            asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(mb + q)) : "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot),
                     "r"(CV_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot_ptr;

    if (warp == 0) {
        if (lane == 0) {
            int issued = 0;
            for (int kb = 0; kb < nkb; ++kb) {
                const int s = kb % p.stages;
                const uint32_t ph = (uint32_t)(kb / p.stages) & 1u;
                if (!mbar_wait(empty0 + 8u * s, ph ^ 1u, p.status, p.wait_ns)) break;
                issued = kb + 1;
                const uint32_t b0 = base + (uint32_t)s * CV_STAGE_BYTES + NT * TC_A_BYTES;
                mbar_arrive_expect_tx(bfull0 + 8u * s, NT * CV_B_BYTES);
#pragma unroll
                for (int t = 0; t < NT; ++t)
                    tma_load_2d(b0 + (uint32_t)t * CV_B_BYTES, mb + t, bfull0 + 8u * s, (kb0 + kb) * TC_BK, n0);
            }
            for (int kb = max(0, issued - p.stages); kb < issued; ++kb)
                mbar_drain(bfull0 + 8u * (kb % p.stages), (uint32_t)(kb / p.stages) & 1u, p.status);
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {
            // chunk c accumulates into TMEM columns (c & 1) * 64 NT; A_t x [B_0 | .. | B_(NT-1-t)] is
            // one MMA, column group u collects the products with B_u
            const uint32_t a_mn = a_kmajor ? 0 : 1;
            const uint32_t idesc_n[NT] = {idesc_bf16(TC_BM, CV_BN * NT, a_mn, 0),
                                         idesc_bf16(TC_BM, CV_BN * 2, a_mn, 0),
                                         idesc_bf16(TC_BM, CV_BN, a_mn, 0)};
            for (int kb = 0; kb < nkb; ++kb) {
                const int c = kb / CV_CHUNK, x = c & 1;
                const bool first = kb % CV_CHUNK == 0;
                if (first) {
                    if (!mbar_wait(acce_bar(x), ((uint32_t)(c >> 1) & 1u) ^ 1u, p.status, p.wait_ns)) break;
                    tc_fence_after();
                }
                const int s = kb % p.stages;
                const uint32_t ph = (uint32_t)(kb / p.stages) & 1u;
                if (!mbar_wait(bfull0 + 8u * s, ph, p.status, p.wait_ns)) break;
                if (!mbar_wait(afull0 + 8u * s, ph, p.status, p.wait_ns)) break;
                tc_fence_after();
                const uint32_t st = base + (uint32_t)s * CV_STAGE_BYTES;
                const uint32_t d = tmem + (uint32_t)x * CV_BN * NT;
#pragma unroll
                for (int kk = 0; kk < TC_BK / 16; ++kk) {
                    const uint64_t db = sdesc_sw64(st + NT * TC_A_BYTES + kk * 32u, 16u, 512u);  // from B_0 on
#pragma unroll
                    for (int t = 0; t < NT; ++t) {
                        const uint32_t a_t = st + (uint32_t)t * TC_A_BYTES;
                        const uint64_t da = a_kmajor ? sdesc_sw64(a_t + kk * 32u, 16u, 512u)
                                                     : sdesc_sw64(a_t + kk * 1024u, 2048u, 512u);
                        mma_bf16(d, da, db, idesc_n[t], (first && kk == 0 && t == 0) ? 0u : 1u);
                    }
                }
                mma_commit(empty0 + 8u * s);
                if (kb % CV_CHUNK == CV_CHUNK - 1 || kb == nkb - 1) mma_commit(accf_bar(x));
            }
            mma_commit(done_bar);
        }
        __syncwarp();
    } else if (warp >= 4 && warp < 4 + CV_EPI_WARPS) {
        // ---- chunk drain: FP64 sums of 32 rows (TMEM lane quarter) and 32 columns ----
        const int q = warp & 3, h = (warp - 4) >> 2;
        double acc[CV_BN / 2];
#pragma unroll
        for (int j = 0; j < CV_BN / 2; ++j) acc[j] = 0.0;
        bool ok = true;
        for (int c = 0; c < nchunks; ++c) {
            const int x = c & 1;
            ok = __all_sync(FULL, mbar_wait(accf_bar(x), (uint32_t)(c >> 1) & 1u, p.status, p.wait_ns));
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int c0 = 0; c0 < CV_BN / 2; c0 += 16) {
#pragma unroll
                for (int u = 0; u < NT; ++u) {
                    uint32_t r[16];
                    tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(x * CV_BN * NT + u * CV_BN + h * (CV_BN / 2) + c0), r);
#pragma unroll
                    for (int j = 0; j < 16; ++j) acc[c0 + j] += (double)__uint_as_float(r[j]);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acce_bar(x)) : "memory");
        }
        const int row0 = m0 + q * 32, col0 = n0 + h * (CV_BN / 2);
        // element i of a lane at address(i), the old values (beta) of eight read before the first one is
        // written (581667 x 96, K = 27: 1361 us a call one by one, 543 now)
        auto write = [&](auto *base, int count, auto address, auto value) {
            using O = std::remove_reference_t<decltype(*base)>;
            constexpr int STEP = 8;
#pragma unroll
            for (int i0 = 0; i0 < CV_BN / 2; i0 += STEP) {
                if (i0 >= count) break;
                O old[STEP];
                if (p.beta_on) {
#pragma unroll
                    for (int i = 0; i < STEP; ++i)
                        if (i0 + i < count) old[i] = base[address(i0 + i)];
                }
#pragma unroll
                for (int i = 0; i < STEP; ++i)
                    if (i0 + i < count) {
                        double v = value(i0 + i);
                        if (p.beta_on) v += p.beta * (double)old[i];
                        base[address(i0 + i)] = (O)v;
                    }
            }
        };
        auto epilogue = [&](auto *out) {
            if (p.cs == 1 && p.N - col0 >= 16 && ok) {
                // rows of the tile along memory: turned through the operand stages (every copy into
                // them has been consumed), so that a warp writes 32 neighbouring elements of a row
                // (4096 x 30000, K = 200: 1403 us a call; 2004 with a row per lane, whose stores went to
                // 32 lines each; for a few columns those are neighbours)
                double *blk = reinterpret_cast<double *>(gen) + (warp - 4) * 32 * 33;
#pragma unroll
                for (int j = 0; j < CV_BN / 2; ++j) blk[lane * 33 + j] = p.alpha * acc[j];
                __syncwarp();
                if (col0 + lane < p.N)
                    write(out + (int64_t)row0 * p.rs + col0 + lane, min(32, p.M - row0), [&](int i) { return i * p.rs; },
                          [&](int i) { return blk[i * 33 + lane]; });
            } else if (row0 + lane < p.M) {
                write(out + (row0 + lane) * p.rs + col0 * p.cs, min(CV_BN / 2, p.N - col0), [&](int j) { return j * p.cs; },
                      [&](int j) { return ok ? p.alpha * acc[j] : 0.0; });
            }
        };
        if (p.out_f64) epilogue((double *)p.out);
        else epilogue((float *)p.out);
    } else if (warp >= 4 + CV_EPI_WARPS) {
        const int t = threadIdx.x - 32 * (4 + CV_EPI_WARPS);
        unsigned char *ring_gen = gen + (ring - base);
        if (a_kmajor) conv_warps<1>(p, t, ring, ring_gen, gen, m0, kb0, nkb, empty0, afull0);
        else conv_warps<0>(p, t, ring, ring_gen, gen, m0, kb0, nkb, empty0, afull0);
    }
    // every MMA issued (done_bar is committed on every path) has finished before the
    // accumulators are released
    if (threadIdx.x == 64) mbar_drain(done_bar, 0u, p.status);
    tc_fence_before();
    __syncthreads();
    if (warp == 2)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(CV_TMEM_COLS) : "memory");
}

struct ConvMaps {
    CUtensorMap b[NT];
};

// CTA (tile, split): tiles with the N index fastest, so that the CTAs that share rows of A run
// together; split z writes its FP64 partial tile at out + z * stride.
__global__ void __launch_bounds__(CV_THREADS, 1)
conv_gemm_kernel(const __grid_constant__ ConvMaps maps, ConvArgs p, int a_kmajor, int ntl, int nkb, int kbps,
                 int64_t stride) {
    const int tile = blockIdx.x, kb0 = blockIdx.y * kbps;
    if (blockIdx.y) p.out = (double *)p.out + (int64_t)blockIdx.y * stride;
    conv_cta(maps.b, p, a_kmajor, (tile / ntl) * TC_BM, (tile % ntl) * CV_BN, kb0, max(0, min(nkb - kb0, kbps)));
}

// C(m, n) (at C[m*rs + n*cs]) = alpha * sum_s P[s](m, n) + beta * C(m, n), P(m, n) at [m + n*M], splits
// added in order, through 32 x 8 tiles so that both sides are read and written along memory.  One
// thread per element with CR_AHEAD partials in flight: a single tile has up to 64 splits, and their
// latency is all this kernel does (16384 x 100 to 100 rows: 50 us a call, 79 with four elements per
// thread one after another).
constexpr int CR_AHEAD = 16, CR_N = 8;
__global__ void __launch_bounds__(256) conv_reduce_kernel(const double *P, int splits, int64_t stride, int64_t M, int64_t N,
                                                          float *C, int64_t rs, int64_t cs, double alpha, double beta,
                                                          int beta_on) {
    __shared__ double tile[32][CR_N + 1];
    const int64_t tn = (N + CR_N - 1) / CR_N, m0 = blockIdx.x / tn * 32, n0 = blockIdx.x % tn * CR_N;
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
    if (m0 + x < M && n0 + y < N) {
        const double *e = P + m0 + x + (n0 + y) * M;
        double a = 0.0;
        for (int s0 = 0; s0 < splits; s0 += CR_AHEAD) {
            double v[CR_AHEAD];
#pragma unroll
            for (int k = 0; k < CR_AHEAD; ++k) v[k] = __ldg(e + min(s0 + k, splits - 1) * stride);
#pragma unroll
            for (int k = 0; k < CR_AHEAD; ++k)
                if (s0 + k < splits) a += v[k];
        }
        tile[x][y] = a;
    }
    __syncthreads();
    const int i = rs == 1 ? x : (int)threadIdx.x / CR_N, j = rs == 1 ? y : (int)threadIdx.x % CR_N;
    if (m0 + i >= M || n0 + j >= N) return;
    float *c = C + (m0 + i) * rs + (n0 + j) * cs;
    double v = alpha * tile[i][j];
    if (beta_on) v += beta * (double)*c;
    *c = (float)v;
}

// C (M x N, ld ldc) = alpha * op(A) * op(B) + beta * C for Float32 A and B (an FP32-accurate
// product).  The operand with more elements is converted in the kernel; when that is B, the
// transposed product is computed and written with its strides exchanged.  The other one is split
// beforehand into K-major terms in the context's memory pool.  Gaussian A * Omega, A 65536 x 1024,
// Omega 1024 x 128: 289 us a call, 394 us with both operands split in memory.
int gemm_f32_tc(rla_ctx *ctx, int64_t M, int64_t N, int64_t K, const float *A, int64_t lda, int ta, const float *B,
                int64_t ldb, int tb, float *C, int64_t ldc, double alpha, double beta) {
    if (M <= 0 || N <= 0) return RLA_OK;
    if (K <= 0) return gemm<float, float, float, double>(ctx, M, N, K, A, lda, ta, B, ldb, tb, C, ldc, alpha, beta);
    if (M >= (1ll << 31) || K >= (1ll << 31) || N >= (1ll << 31))
        return set_error(ctx, RLA_E_UNSUPPORTED, "tensor-core GEMM: dimension above 2^31");
    // every tile of 64 columns converts its 128 rows of A again: above four of them splitting A once in
    // memory is faster (16000 x 512 to 1000 rows: 389 us converting, 363 us split before), unless K is
    // so short that the FP64 partial tiles of the other kernel cost more (4096 x 30000, converting / split
    // before: K = 16 615 / 1246 us, K = 128 1032 / 1415, K = 256 1446 / 1689)
    if (std::min(M, N) > 4 * CV_BN && K > 256)
        return gemm_f32_tc_presplit(ctx, M, N, K, A, lda, ta, B, ldb, tb, C, ldc, alpha, beta);
    int64_t rs = 1, cs = ldc;
    // The larger operand is converted, unless the other way round fills the tiles so much better that
    // it makes up for splitting the larger one in memory (each tile saved for 64 rows more; 130 x 120,
    // K = 258299: 2 x 2 or 1 x 3 tiles, 398 / 252 us a call)
    const int64_t large = std::max(M, N), small = std::min(M, N);
    auto tiles_of = [](int64_t m, int64_t n) { return ceil_div(m, TC_BM) * ceil_div(n, CV_BN); };
    const bool turn = 64 * (tiles_of(large, small) - tiles_of(small, large)) > large - small;
    if (turn ? N < M : N > M) {  // C' = op(B)' op(A)'
        std::swap(M, N);
        std::swap(A, B);
        std::swap(lda, ldb);
        const int t = ta;
        ta = !tb;
        tb = !t;
        std::swap(rs, cs);
    }
    const int64_t mt = ceil_div(M, TC_BM), ntl = ceil_div(N, CV_BN), nkb = ceil_div(K, TC_BK);
    if (mt * ntl >= (1ll << 31)) return set_error(ctx, RLA_E_UNSUPPORTED, "tensor-core GEMM: grid too large");
    int *status = nullptr;
    RLA_TRY(tc_status_get(ctx, &status));
    const int64_t budget = ctx->smem_optin - 1024 - 256 - (int64_t)CV_RAW * CV_RAW_BYTES;
    const int stages = (int)std::min<int64_t>(4, budget / CV_STAGE_BYTES);
    const size_t smem = 1024 + 256 + (size_t)stages * CV_STAGE_BYTES + CV_RAW * CV_RAW_BYTES;
    // K splits: the rounds of CTAs times the k-blocks of a split (1.2 us each) and of a CTA's start (4),
    // and the sums of the partial tiles (4 us, 16 bytes an element at 4 TB/s).  16384 x 260 to 200 rows,
    // 12 tiles: 117 us a call in 13 splits, 90 in 12; 11234 x 2778 to 244, 88 tiles: 465 in one, 321 in five.
    // At most 64 MB of partial tiles; in a graph capture no more splits than one round holds (a
    // captured scratch must not be grown later, and calls of a round or more never had one).
    const int64_t tiles = mt * ntl, sms = ctx->sm_count;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    RLA_CUDA_TRY(ctx, cudaStreamIsCapturing(ctx->stream, &cap));
    const int64_t most = cap != cudaStreamCaptureStatusNone ? std::max<int64_t>(1, sms / tiles) : 8 * sms / tiles;
    int64_t splits = 1;
    double best = 0.0;
    for (int64_t sp = 1; sp <= std::min(most, nkb / (2 * CV_CHUNK)); ++sp) {
        const int64_t len = ceil_div(ceil_div(nkb, sp), CV_CHUNK) * CV_CHUNK, n = ceil_div(nkb, len);
        if (n > 1 && 8 * M * N * n > (int64_t)64 << 20) break;
        const double us = 1.2 * (ceil_div(tiles * n, sms) * (std::min(len, nkb) + 4)) + (n > 1 ? 4.0 + 4e-6 * M * N * n : 0.0);
        if (sp == 1 || us < best) {
            best = us;
            splits = n;
        }
    }
    const int64_t kbps = ceil_div(ceil_div(nkb, splits), CV_CHUNK) * CV_CHUNK;
    splits = ceil_div(nkb, kbps);
    void *ws = nullptr;
    if (splits > 1) RLA_TRY(scratch_get(ctx, sizeof(double) * (size_t)(M * N * splits), &ws));
    const int64_t ldb2 = ceil_div(K, 8) * 8;
    const size_t nb = (size_t)ldb2 * N;
    bf16 *buf = nullptr;
    RLA_CUDA_TRY(ctx, pool_malloc_s(ctx, (void **)&buf, sizeof(bf16) * 3 * nb + 256, ctx->stream));
    bf16 *b3[3] = {buf, buf + nb, buf + 2 * nb};
    int rc = tb ? split_terms_launch<NT>(ctx, B, N, K, ldb, 1, b3, ldb2) : split_terms_launch<NT>(ctx, B, K, N, ldb, 0, b3, ldb2);
    ConvMaps maps;
    for (int t = 0; t < NT && rc == RLA_OK; ++t) rc = tc_make_map(ctx, &maps.b[t], b3[t], K, N, ldb2, TC_BK, CV_BN);
    auto launch = [&]() -> int {
        const bool part = splits > 1;
        ConvArgs p{A, lda, lda % 4 == 0 && (uintptr_t)A % 16 == 0, (int)M, (int)N, (int)K,
                   part ? ws : (void *)C, part ? 1 : rs, part ? M : cs, part,
                   part ? 1.0 : alpha, beta, !part && beta != 0.0, stages, status, ctx->wait_ns};
        RLA_CUDA_TRY(ctx, set_smem_max(conv_gemm_kernel));
        cudaEvent_t e0 = timing_begin(ctx);
        conv_gemm_kernel<<<dim3((unsigned)tiles, (unsigned)splits), CV_THREADS, smem, ctx->stream>>>(
            maps, p, ta, (int)ntl, (int)nkb, (int)kbps, M * N);
        RLA_TRY(check_launch(ctx, "conv_gemm"));
        timing_end(ctx, 0, e0);
        if (!part) return RLA_OK;
        conv_reduce_kernel<<<(unsigned)(ceil_div(M, 32) * ceil_div(N, CR_N)), 256, 0, ctx->stream>>>(
            (const double *)ws, (int)splits, M * N, M, N, C, rs, cs, alpha, beta, beta != 0.0);
        return check_launch(ctx, "conv_reduce");
    };
    if (rc == RLA_OK) rc = launch();
    cudaFreeAsync(buf, ctx->stream);
    return rc;
}

}  // namespace rla
