// rla_sparse_tile.cu -- SparseSign / CountSketch compress on tiles of 128-byte rows.
//
// Y(b, v) = sum over the entries (j, b) of the sketch of sign(j, b) * X(j, v): every input
// element is used nnz times, so the pass is bound by shared-memory traffic, not by HBM, unless
// one access moves a full row of useful values.  A tile holds R = 640 long indices of 32 (Float32)
// or 16 (Float64) vectors, one 128-byte row per long index, and 8 lanes ("an octet") handle one
// entry with 16-byte accesses: reading row j and adding to the bins of bucket b are then one
// conflict-free wavefront each whatever j and b are, and a warp instruction serves four entries.
// The entries of a chunk of R long indices are kept sorted by bucket (built when the sketch is
// drawn) and cut into groups of four entries of one bucket (of one, when buckets are sparse), the
// last group of a bucket filled up with a row of zeros: a step of the kernel adds one group per octet to its bucket, with no
// branches.  With e = R * nnz / s entries per bucket and chunk and g = ceil(e/4) groups,
//   wavefronts per bucket and chunk = g * (4 rows + 2 bins + 1/4 words).
// Measured (unprofiled call): 150001 -> 1332 (nnz 8) of 333 Float32 columns 254 us, 603 us with one
// output vector per warp and private bins; 3000 -> 100 (nnz 8) of 30011 Float32 rows 297 us,
// 1526 us with lane = vector bins; 4096 -> 512 of 256 Float64 columns 39 against 71 us.  The
// shared-memory pipe is 72 % busy at the second size.  Entry by entry with an end-of-run
// flag instead of filled groups takes fewer wavefronts and half again as many instructions, and came
// out the same (258 and 308 us, when groups took 257 and 307).
// A CTA of 16 warps walks (vector tile, bucket window, chunk) units; each warp owns the
// buckets congruent to it modulo 16, so there are no atomics and the result is reproducible bit
// for bit.  Vectors that are contiguous in j (columns of a column-major A) are transposed on the
// way into shared memory, strided ones (rows) copied as they are.  The next unit's elements are
// loaded into registers while the current one is summed.
//
// The tile takes 80 KB, the bins the rest: a window holds 1040 buckets (R = 640 is the largest
// that leaves 1024); a larger s takes several windows, each staging X again.
#include "rla_internal.cuh"
#include "rla_kernels.cuh"

namespace rla {

constexpr int BL_WARPS = 16;       // warps of the compress CTA, lists per (chunk, window)
constexpr int BL_BUILD_WARPS = 8;  // warps of the plan builder
constexpr int BL_R = 640;          // long indices per chunk
constexpr int BL_MAX_SW = 1040, BL_MAX_WIN = 8, BL_MAX_NNZ = 32;
constexpr int BL_PITCH = 144;      // bytes between bins of consecutive buckets (128 + 16)
constexpr int BL_PF = 10;          // 16-byte loads per thread and unit
static_assert(BL_R * 8 == BL_PF * BL_WARPS * 32, "a unit is BL_PF 16-byte loads per thread");
// Entry word: bits 4..16 byte offset of row j with its swizzle, bits 17..30 offset of the
// bucket's bins in 16-byte units (used from the first word of a group), bit 31 sign.
constexpr uint32_t BL_ROW_MASK = 0x1fff0u, BL_BIN_MASK = 0x3fff0u;
constexpr int BL_BIN_SHIFT = 17;
constexpr uint32_t BL_ZERO_ROW = (uint32_t)BL_R << 7;  // row R of the tile holds zeros
constexpr int BL_SLOW = 1 << 30;   // list flag: two octets may update one bucket in the same step
constexpr int BL_AHEAD = 7;         // steps whose words a lane holds
constexpr int BL_SLACK = 2 * BL_AHEAD * 16;  // words read ahead of the end of a list (and never used)
constexpr int BL_TILE_BYTES = (BL_R + 1) * 128;

template <class T>
struct TileCfg {
    static constexpr int VR = 16 / (int)sizeof(T);  // elements per 16 bytes
    static constexpr int C = 8 * VR;                // vectors per tile
};
template <class T>
struct TileVec;
template <>
struct TileVec<float> {
    using type = float4;
};
template <>
struct TileVec<double> {
    using type = double2;
};

// Row j keeps 16-byte slot q at q ^ swz(j): the transposing stores of a warp (8 lanes along j
// in steps of VR, 4 vectors) then hit distinct banks.
template <class T>
__host__ __device__ constexpr int tile_swz(int j) {
    constexpr int VR = TileCfg<T>::VR;
    return (j / VR + (8 / VR) * (j % VR)) & 7;
}
template <class T>
__device__ __forceinline__ uint32_t tile_off(int j, int c) {
    constexpr int VR = TileCfg<T>::VR;
    return ((uint32_t)j << 7) | ((uint32_t)((c / VR) ^ tile_swz<T>(j)) << 4) | ((uint32_t)(c % VR) * (uint32_t)sizeof(T));
}

// ------------------------------------------------------------------------------------
// Plan: per (chunk, window, warp) the groups of the warp's buckets in bucket order, cut into four
// equal parts, one per octet, interleaved so that a step's words are 64 consecutive bytes.  The
// groups of a bucket that crosses a cut are added by both octets, in different steps unless the
// bucket has more groups than a part: such lists are marked BL_SLOW.  Filling groups point at the
// zero row and at a bin past the last one.  With few buckets (s * G < 256) a bucket is kept G
// times (long index modulo G picks the copy), so that the warps' shares are even; the copies are
// added when the bins are written.
// ------------------------------------------------------------------------------------
struct BlGeom {
    int nwin, sw, G, spw;  // windows, buckets per window, copies, keys (bucket copies) per warp
    int gs;                // entries per group, 4 or 1
    int64_t nchunk, cap;   // cap: words reserved per chunk, a multiple of 16
};

static bool bl_geometry(const rla_sketch *sk, BlGeom *g) {
    if (sk->nnz > BL_MAX_NNZ || sk->s > (int64_t)BL_MAX_WIN * BL_MAX_SW) return false;
    g->nwin = (int)ceil_div(sk->s, BL_MAX_SW);
    g->sw = (int)ceil_div(sk->s, g->nwin);
    g->G = 1;
    if (g->nwin == 1)
        while (g->G < 16 && g->sw * g->G < 256 && (int64_t)BL_R * sk->nnz >= 8 * (int64_t)g->sw * g->G) g->G *= 2;
    g->spw = ceil_div_i((int64_t)g->sw * g->G, BL_WARPS);
    g->nchunk = ceil_div(sk->L, BL_R);
    // Groups of four fill up with zero rows when buckets are sparse: at e = 2 they take as many
    // wavefronts per entry (3.2) as single entries, each with its own bin update.
    g->gs = (int64_t)BL_R * sk->nnz >= 2 * sk->s * g->G ? 4 : 1;
    const int64_t ne = (int64_t)BL_R * sk->nnz, keys = (int64_t)g->nwin * BL_WARPS * g->spw;
    g->cap = (ne + (g->gs - 1) * std::min(ne, keys) + 15 * BL_WARPS * g->nwin + 15) / 16 * 16 + BL_SLACK;
    return true;
}

// One CTA per chunk: a stable counting sort by (window, warp, bucket).  All threads fetch the
// entries' keys; each of H warps ranks the entries of R/H rows in increasing order against its own
// counters (ranks inside a warp access come from match_any, so the order of a bucket's entries is
// the order of the long indices); then all threads place them.  Entry while sorting: bits 0..13
// key, 14..28 rank, 31 sign.
constexpr int BL_KEY_BITS = 14;
static_assert(BL_MAX_WIN * (BL_MAX_SW + BL_WARPS) <= 1 << BL_KEY_BITS && BL_R * BL_MAX_NNZ < 1 << (31 - BL_KEY_BITS), "entry fields");
template <class T>
__global__ void __launch_bounds__(BL_BUILD_WARPS * 32) bl_build_kernel(const int32_t *bucket, const uint8_t *negative,
                                                                       int64_t L, int nnz, BlGeom g, int H, uint32_t *words,
                                                                       int2 *lists) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int K = g.nwin * BL_WARPS * g.spw, nlist = g.nwin * BL_WARPS;
    uint32_t *ent = reinterpret_cast<uint32_t *>(smem_raw);            // [R * nnz]
    uint16_t *hist = reinterpret_cast<uint16_t *>(ent + BL_R * nnz);   // [H][K] counts, then offsets inside the bucket
    uint16_t *koff = hist + H * K;                                     // [K] entries, then first group of the bucket in its list
    __shared__ int lstart[BL_MAX_WIN * BL_WARPS], lpart[BL_MAX_WIN * BL_WARPS], lslow[BL_MAX_WIN * BL_WARPS];
    __shared__ int all_words;
    constexpr int nt = BL_BUILD_WARPS * 32;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5, gsh = g.gs == 4 ? 2 : 0;
    const int64_t chunk = blockIdx.x, row0 = chunk * BL_R;
    const int rows = (int)min((int64_t)BL_R, L - row0), ne = rows * nnz, rows_w = BL_R / H;
    const int64_t base = row0 * nnz;
    uint32_t *out = words + chunk * g.cap;
    for (int i = t; i < H * K / 8; i += nt) reinterpret_cast<uint4 *>(hist)[i] = make_uint4(0, 0, 0, 0);
    for (int i = t; i < ne; i += nt) {
        const int jl = i / nnz;
        const uint32_t b = (uint32_t)__ldg(bucket + base + i);
        const int win = (int)(b / (uint32_t)g.sw);
        const int vlb = (jl & (g.G - 1)) * g.sw + (int)b - win * g.sw;
        const int list = win * BL_WARPS + (vlb & (BL_WARPS - 1));
        ent[i] = (uint32_t)(list * g.spw + vlb / BL_WARPS) | ((uint32_t)__ldg(negative + base + i) << 31);
    }
    __syncthreads();
    if (w < H) {
        uint16_t *myh = hist + w * K;
        const int hi = min((w + 1) * rows_w, rows) * nnz;
        for (int i0 = w * rows_w * nnz; i0 < hi; i0 += 32) {
            const int i = i0 + lane;
            const bool valid = i < hi;
            const uint32_t e = valid ? ent[i] : 0u;
            const int key = (int)(e & ((1u << BL_KEY_BITS) - 1u));
            const unsigned grp = __match_any_sync(FULL, valid ? key : -1 - lane);
            const int rank = __popc(grp & ((1u << lane) - 1u));
            const int before = valid ? myh[key] : 0;
            __syncwarp();
            if (valid && rank == 0) myh[key] = (uint16_t)(before + __popc(grp));
            if (valid) ent[i] = e | ((uint32_t)(before + rank) << BL_KEY_BITS);
            __syncwarp();
        }
    }
    __syncthreads();
    for (int k = t; k < K; k += nt) {  // counts -> exclusive offsets over the warps
        int run = 0;
        for (int q = 0; q < H; ++q) {
            const int c = hist[q * K + k];
            hist[q * K + k] = (uint16_t)run;
            run += c;
        }
        koff[k] = (uint16_t)run;
    }
    __syncthreads();
    {  // first group of each bucket: P lanes per list, a segment of its keys each
        const int P = g.nwin == 1 ? 16 : g.nwin == 2 ? 8 : g.nwin <= 4 ? 4 : 2;
        const int l = t / P, seg = (g.spw + P - 1) / P;
        const int k0 = l * g.spw + min(t % P * seg, g.spw), k1 = l * g.spw + min((t % P + 1) * seg, g.spw);
        int run = 0, most = 0;
        if (l < nlist)
            for (int k = k0; k < k1; ++k) {
                const int ng = (koff[k] + g.gs - 1) >> gsh;
                run += ng;
                most = max(most, ng);
            }
        int before = run;  // inclusive over the list's lanes
        for (int d = 1; d < P; d <<= 1) {
            const int v = __shfl_up_sync(FULL, before, d, P), m = __shfl_xor_sync(FULL, most, d, P);
            if (t % P >= d) before += v;
            most = max(most, m);
        }
        const int total = __shfl_sync(FULL, before, P - 1, P);
        before -= run;
        if (l < nlist) {
            for (int k = k0; k < k1; ++k) {
                const int ng = (koff[k] + g.gs - 1) >> gsh;
                koff[k] = (uint16_t)before;
                before += ng;
            }
            if (t % P == 0) {
                const int gpw = 4 >> gsh, part = ((total + 3) / 4 + gpw - 1) / gpw * gpw;
                lpart[l] = part;
                lslow[l] = most > part;
            }
        }
    }
    __syncthreads();
    if (w == 0) {  // first word of each list
        constexpr int PER = BL_MAX_WIN * BL_WARPS / 32;
        int len[PER], run = 0;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int l = lane * PER + i;
            len[i] = l < nlist ? 4 * g.gs * lpart[l] : 0;
            run += len[i];
        }
        int before = run;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int v = __shfl_up_sync(FULL, before, d);
            if (lane >= d) before += v;
        }
        if (lane == 31) all_words = before;
        before -= run;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            if (lane * PER + i < nlist) lstart[lane * PER + i] = before;
            before += len[i];
        }
    }
    __syncthreads();
    for (int l = t; l < nlist; l += nt)
        lists[chunk * nlist + l] = make_int2(lstart[l] / 16, (lpart[l] * g.gs / 4) | (lslow[l] ? BL_SLOW : 0));
    const uint32_t fill = BL_ZERO_ROW | ((uint32_t)(g.sw * g.G * (BL_PITCH / 16)) << BL_BIN_SHIFT);
    for (int i = t; i < (all_words + BL_SLACK) / 4; i += nt)
        reinterpret_cast<uint4 *>(out)[i] = make_uint4(fill, fill, fill, fill);
    __syncthreads();
    for (int i = t; i < ne; i += nt) {
        const uint32_t e = ent[i];
        const int jl = i / nnz, key = (int)(e & ((1u << BL_KEY_BITS) - 1u)), list = key / g.spw;
        const int r = hist[jl / rows_w * K + key] + (int)((e & 0x7fffffffu) >> BL_KEY_BITS);
        const int k = koff[key] + (r >> gsh), part = lpart[list];
        const int o = k / part, q = k - o * part;
        const int gpw = 4 >> gsh;  // groups per 16-byte word of an octet
        const int vlb = (key - list * g.spw) * BL_WARPS + (list & (BL_WARPS - 1));
        out[lstart[list] + (((q / gpw) * 4 + o) << 2) + (q % gpw) * g.gs + (r & (g.gs - 1))] =
            tile_off<T>(jl, 0) | ((uint32_t)(vlb * (BL_PITCH / 16)) << BL_BIN_SHIFT) | (e & 0x80000000u);
    }
}

int tile_plan_build(rla_ctx *ctx, rla_sketch *sk) {
    BlGeom g;
    sk->bl_ok = false;
    if (!bl_geometry(sk, &g)) return RLA_OK;
    const int nlist = g.nwin * BL_WARPS, K = nlist * g.spw;
    if (!sk->bl_words) RLA_CUDA_TRY(ctx, dev_alloc_t(ctx, &sk->bl_words, sizeof(uint32_t) * (size_t)(g.nchunk * g.cap)));
    if (!sk->bl_lists) RLA_CUDA_TRY(ctx, dev_alloc_t(ctx, &sk->bl_lists, sizeof(int2) * (size_t)(g.nchunk * nlist)));
    // Ranking warps: each has counters of its own for every key, which cost shared memory (CTAs per SM)
    // and time to add up, while fewer warps rank one after another.  Update of 2^20 -> s, us, with
    // 8 / 4 / 2 / 1: nnz 1, s = 1000 54 / 51 / 53 / 54, s = 4096 131 / 108 / 107 / 108, s = 8320 185 / 121 / 104 / 99;
    // nnz 8, s = 1000 279 / 279 / 283 / 301, s = 8320 418 / 332 / 331 / 359; of 10^4 -> 1000, nnz 8: 43 / 45 / 56 / 75.
    const int H = K <= 1100 ? 8 : K > 6000 && sk->nnz <= 2 ? 2 : 4;
    const size_t smem = sizeof(uint32_t) * BL_R * sk->nnz + sizeof(uint16_t) * (size_t)K * (H + 1);
    auto go = [&](auto kern) -> int {
        RLA_CUDA_TRY(ctx, set_smem_max(kern));
        kern<<<(unsigned)g.nchunk, BL_BUILD_WARPS * 32, smem, ctx->stream>>>(sk->bucket, sk->negative, sk->L, (int)sk->nnz, g, H,
                                                                             sk->bl_words, sk->bl_lists);
        return check_launch(ctx, "bl_build");
    };
    RLA_TRY(sk->p.dtype == RLA_F32 ? go(bl_build_kernel<float>) : go(bl_build_kernel<double>));
    sk->bl_ok = true;
    return RLA_OK;
}

// ------------------------------------------------------------------------------------
// Compress
// ------------------------------------------------------------------------------------
template <class T>
struct TileParams {
    const T *X;
    int64_t x_ld;  // contiguous: element (j, v) at X[j + v*x_ld]; strided: at X[v + j*x_ld]
    int64_t L, nv, s;
    const uint32_t *words;
    const int2 *lists;
    BlGeom g;
    T *Y;
    int64_t y_es, y_vs;
    T alpha, beta;
    int beta_zero;
    T *partials;  // [slot][sw][C]
    Split split;  // over (tile, window, chunk), chunk fastest
    int64_t unit;  // chunks per split unit: 1, or all of a (tile, window) when no partial sums are kept
};

// y +- x, 16 bytes per lane
__device__ __forceinline__ float4 octet_add(float4 y, float4 x, uint32_t w) {
    const float s = __uint_as_float((w & 0x80000000u) | 0x3f800000u);
    const float2 s2 = make_float2(s, s);
    const float2 lo = __ffma2_rn(make_float2(x.x, x.y), s2, make_float2(y.x, y.y));
    const float2 hi = __ffma2_rn(make_float2(x.z, x.w), s2, make_float2(y.z, y.w));
    return make_float4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ double2 octet_add(double2 y, double2 x, uint32_t w) {
    const long long m = (long long)(w & 0x80000000u) << 32;
    return make_double2(y.x + __longlong_as_double(__double_as_longlong(x.x) ^ m),
                        y.y + __longlong_as_double(__double_as_longlong(x.y) ^ m));
}
// +-x0 +-x1 +-x2 +-x3 + y, 16 bytes per lane
__device__ __forceinline__ float4 octet_sum(float4 x0, float4 x1, float4 x2, float4 x3, uint4 w, float4 y) {
    auto sg = [](uint32_t u) {
        const float f = __uint_as_float((u & 0x80000000u) | 0x3f800000u);
        return make_float2(f, f);
    };
    const float2 s0 = sg(w.x), s1 = sg(w.y), s2 = sg(w.z), s3 = sg(w.w);
    float2 lo = __fmul2_rn(make_float2(x0.x, x0.y), s0), hi = __fmul2_rn(make_float2(x0.z, x0.w), s0);
    lo = __ffma2_rn(make_float2(x1.x, x1.y), s1, lo);
    hi = __ffma2_rn(make_float2(x1.z, x1.w), s1, hi);
    lo = __ffma2_rn(make_float2(x2.x, x2.y), s2, lo);
    hi = __ffma2_rn(make_float2(x2.z, x2.w), s2, hi);
    lo = __ffma2_rn(make_float2(x3.x, x3.y), s3, lo);
    hi = __ffma2_rn(make_float2(x3.z, x3.w), s3, hi);
    lo = __fadd2_rn(lo, make_float2(y.x, y.y));
    hi = __fadd2_rn(hi, make_float2(y.z, y.w));
    return make_float4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ double2 octet_sum(double2 x0, double2 x1, double2 x2, double2 x3, uint4 w, double2 y) {
    auto sg = [](double x, uint32_t u) {
        return __longlong_as_double(__double_as_longlong(x) ^ ((long long)(u & 0x80000000u) << 32));
    };
    const double a = ((sg(x0.x, w.x) + sg(x1.x, w.y)) + sg(x2.x, w.z)) + sg(x3.x, w.w);
    const double b = ((sg(x0.y, w.x) + sg(x1.y, w.y)) + sg(x2.y, w.z)) + sg(x3.y, w.w);
    return make_double2(y.x + a, y.y + b);
}

// Loads of the next unit, issued where they stand: the compiler would move plain loads down to
// their use, behind the current unit's sums, and expose their latency.
__device__ __forceinline__ float4 ld_ahead(const float4 *a) {
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(a));
    return v;
}
__device__ __forceinline__ double2 ld_ahead(const double2 *a) {
    double2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(a));
    return v;
}
__device__ __forceinline__ float ld_ahead(const float *a) {
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(a));
    return v;
}
__device__ __forceinline__ double ld_ahead(const double *a) {
    double v;
    asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(a));
    return v;
}

// How a unit's elements are read: contiguous vectors with 16-byte aligned starts, contiguous
// vectors at any alignment (16-byte loads of the aligned windows, rows shifted), strided vectors
// with 16-byte aligned rows, strided vectors at any alignment.
enum { TILE_CONTIG = 0, TILE_SHIFT = 1, TILE_ROWS = 2, TILE_ROWS_ANY = 3 };

// STEP: items of 16 bytes per thread whose old values (beta) are read before the first one is written.
template <class T, int MODE, int GS, int STEP>
__global__ void __launch_bounds__(BL_WARPS * 32, 1) tile_compress_kernel(TileParams<T> p) {
    using V = typename TileVec<T>::type;
    constexpr int VR = TileCfg<T>::VR, C = TileCfg<T>::C;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char *bin_raw = smem_raw + BL_TILE_BYTES;
    const int t = threadIdx.x, lane = t & 31, wp = t >> 5, l8 = lane & 7;
    const uint32_t lane16 = (uint32_t)l8 << 4;
    const int64_t nchunk = p.g.nchunk;
    const int64_t u0 = p.split.start(blockIdx.x) * p.unit, u1 = p.split.start(blockIdx.x + 1) * p.unit;
    if (u0 >= u1) return;
    auto zero_bins = [&]() {
        for (int i = t; i < (p.g.sw * p.g.G + 1) * (BL_PITCH / 16); i += BL_WARPS * 32) reinterpret_cast<V *>(bin_raw)[i] = V{};
    };
    zero_bins();
    if (t < 8) reinterpret_cast<V *>(smem_raw + BL_ZERO_ROW)[t] = V{};
    // Contiguous vectors: a thread's column of the tile and its first row; a warp load covers 8
    // lanes x VR rows of 4 columns, the thread's BL_PF loads consecutive blocks of 8*VR rows.
    // Strided vectors: a warp load covers 4 rows (16-byte loads) or 32/C rows (element loads).
    // The swizzle repeats every 8*VR rows, so a thread's shared-memory addresses are one base
    // per row residue plus compile-time offsets.
    constexpr int CQ = C / 4, RW = 32 / C;
    const int my_c = (wp % CQ) * 4 + (lane >> 3), my_r = (wp / CQ) * BL_PF * 8 * VR + l8 * VR;
    const bool has_tail = MODE == TILE_SHIFT && my_r + BL_PF * 8 * VR == BL_R + 7 * VR;
    V pf[BL_PF], tail{};
    int shift = 0;  // rows by which the loaded 16-byte windows start before the thread's rows
    auto load_unit = [&](int64_t tile, int64_t chunk) {
        const int64_t j0 = chunk * BL_R, v0 = tile * C;
        if constexpr (MODE <= TILE_SHIFT) {
            const T *x = p.X + (v0 + my_c) * p.x_ld + j0;
            if (MODE == TILE_SHIFT) shift = (int)((reinterpret_cast<uintptr_t>(x) / sizeof(T)) & (VR - 1));
            // every window of the unit inside its vector: plain loads
            if (v0 + C <= p.nv && j0 + BL_R + (MODE == TILE_SHIFT ? VR : 0) <= p.L && (MODE == TILE_CONTIG || j0 > 0)) {
                const V *xv = reinterpret_cast<const V *>(x + my_r - shift);
#pragma unroll
                for (int k = 0; k < BL_PF; ++k) pf[k] = ld_ahead(xv + k * 8);
                if (has_tail) tail = ld_ahead(reinterpret_cast<const V *>(x + BL_R - shift));
                return;
            }
            const int left = v0 + my_c < p.nv ? (int)min((int64_t)BL_R, p.L - j0) : 0;
            auto load = [&](int r) {
                V y{};
                T *ye = reinterpret_cast<T *>(&y);
#pragma unroll
                for (int e = 0; e < VR; ++e)
                    if (r + e >= 0 && r + e < left) ye[e] = ld_ahead(x + r + e);
                return y;
            };
#pragma unroll
            for (int k = 0; k < BL_PF; ++k) pf[k] = load(my_r + k * 8 * VR - shift);
            if (has_tail) tail = load(BL_R - shift);
        } else if constexpr (MODE == TILE_ROWS) {
            const int r0 = wp * 4 + (lane >> 3);
            const int64_t v = v0 + l8 * VR;
            const T *x = p.X + v + (j0 + r0) * p.x_ld;
            const int64_t step = 64 * p.x_ld;
            const int left = (int)min((int64_t)BL_R, p.L - j0) - r0, nv = (int)min((int64_t)VR, p.nv - v);
            if (nv == VR) {
#pragma unroll
                for (int k = 0; k < BL_PF; ++k) pf[k] = k * 64 < left ? ld_ahead(reinterpret_cast<const V *>(x + k * step)) : V{};
            } else {
#pragma unroll
                for (int k = 0; k < BL_PF; ++k) {
                    pf[k] = V{};
                    T *ye = reinterpret_cast<T *>(&pf[k]);
#pragma unroll
                    for (int e = 0; e < VR; ++e)
                        if (k * 64 < left && e < nv) ye[e] = ld_ahead(x + k * step + e);
                }
            }
        } else {
            const int r0 = wp * RW + lane / C;
            const T *x = p.X + v0 + lane % C + (j0 + r0) * p.x_ld;
            const int64_t step = BL_WARPS * RW * p.x_ld;
            const int left = v0 + lane % C < p.nv ? (int)min((int64_t)BL_R, p.L - j0) - r0 : 0;
            T *d = reinterpret_cast<T *>(pf);
#pragma unroll
            for (int k = 0; k < BL_PF * VR; ++k) {
                d[k] = k * BL_WARPS * RW < left ? ld_ahead(x) : T(0);
                x += step;
            }
        }
    };
    auto store_unit = [&]() {
        if constexpr (MODE <= TILE_SHIFT) {
#pragma unroll
            for (int i = 0; i < VR; ++i) {
                const int r = my_r - shift + i;  // negative only in the first block
                unsigned char *d = smem_raw + r * 128 + (((my_c / VR) ^ tile_swz<T>(r & (8 * VR - 1))) << 4) +
                                   (my_c % VR) * sizeof(T);
#pragma unroll
                for (int k = 0; k < BL_PF; ++k)
                    if (MODE == TILE_CONTIG || k > 0 || r >= 0)
                        *reinterpret_cast<T *>(d + k * 8 * VR * 128) = reinterpret_cast<const T *>(&pf[k])[i];
                if (i < VR - 1 && has_tail && i < shift)
                    *reinterpret_cast<T *>(smem_raw + tile_off<T>(BL_R - shift + i, my_c)) = reinterpret_cast<const T *>(&tail)[i];
            }
        } else if constexpr (MODE == TILE_ROWS) {
            unsigned char *d = smem_raw + tile_off<T>(wp * 4 + (lane >> 3), l8 * VR);
#pragma unroll
            for (int k = 0; k < BL_PF; ++k) *reinterpret_cast<V *>(d + k * 64 * 128) = pf[k];
        } else {
            constexpr int M = sizeof(T) == 4 ? 2 : 1;  // loads after which the swizzle repeats
#pragma unroll
            for (int m = 0; m < M; ++m) {
                unsigned char *d = smem_raw + tile_off<T>((m * BL_WARPS + wp) * RW + lane / C, lane % C);
#pragma unroll
                for (int k = m; k < BL_PF * VR; k += M)
                    *reinterpret_cast<T *>(d + (k - m) * BL_WARPS * RW * 128) = reinterpret_cast<const T *>(pf)[k];
            }
        }
    };
    auto row = [&](uint32_t w) { return *reinterpret_cast<const V *>(smem_raw + ((w & BL_ROW_MASK) ^ lane16)); };
    auto bins_of = [&](uint32_t w) {
        return reinterpret_cast<V *>(bin_raw + ((w >> (BL_BIN_SHIFT - 4)) & BL_BIN_MASK) + lane16);
    };
    int64_t tile = u0 / nchunk / p.g.nwin, chunk = u0 % nchunk;
    int win = (int)(u0 / nchunk % p.g.nwin);
    load_unit(tile, chunk);
    int2 li_next = __ldg(p.lists + (chunk * p.g.nwin + win) * BL_WARPS + wp);
    for (int64_t u = u0; u < u1; ++u) {
        const int2 li = li_next;
        const int nq = li.y & (BL_SLOW - 1);
        const uint4 *lp = reinterpret_cast<const uint4 *>(p.words + chunk * p.g.cap) + li.x * 4 + (lane >> 3);
        uint4 w[BL_AHEAD];
#pragma unroll
        for (int i = 0; i < BL_AHEAD; ++i) w[i] = __ldg(lp + 4 * i);
        store_unit();
        __syncthreads();
        const int64_t tile_u = tile, chunk_u = chunk;
        const int win_u = win;
        if (u + 1 < u1) {
            if (++chunk == nchunk) {
                chunk = 0;
                if (++win == p.g.nwin) {
                    win = 0;
                    ++tile;
                }
            }
            load_unit(tile, chunk);
            li_next = __ldg(p.lists + (chunk * p.g.nwin + win) * BL_WARPS + wp);
        }
        // ---- the octet's groups; the rows of the next group are read before the current one
        // is added, so that the bin update does not hold them up ----
        if (!(li.y & BL_SLOW)) {
            V x0 = row(w[0].x), x1 = row(w[0].y), x2 = row(w[0].z), x3 = row(w[0].w);
            // words are read BL_AHEAD steps ahead (past the list: the next one's or filling, not
            // added), so that the first ones read after the next unit's elements, whose
            // arrival they would wait for, are not needed before those have come
            for (int q = 0; q < nq; q += BL_AHEAD) {
                lp += 4 * BL_AHEAD;
#pragma unroll
                for (int i = 0; i < BL_AHEAD; ++i) {
                    if (q + i >= nq) break;
                    const uint4 wc = w[i], wn = w[(i + 1) % BL_AHEAD];
                    if constexpr (GS == 4) {
                        V *bp = bins_of(wc.x);
                        V y = *bp;
                        y = octet_sum(x0, x1, x2, x3, wc, y);
                        x0 = row(wn.x);
                        x1 = row(wn.y);
                        x2 = row(wn.z);
                        x3 = row(wn.w);
                        *bp = y;
                    } else {
                        auto one = [&](V &x, uint32_t u, uint32_t un) {
                            V *bp = bins_of(u);
                            V y = *bp;
                            y = octet_add(y, x, u);
                            x = row(un);
                            *bp = y;
                        };
                        one(x0, wc.x, wn.x);
                        __syncwarp();
                        one(x1, wc.y, wn.y);
                        __syncwarp();
                        one(x2, wc.z, wn.z);
                        __syncwarp();
                        one(x3, wc.w, wn.w);
                    }
                    w[i] = __ldg(lp + 4 * i);
                    __syncwarp();  // orders these bin updates before the next step's
                }
            }
        } else {  // the octets update the bins one after another
            for (int q = 0; q < nq; ++q, lp += 4) {
                const uint4 w = __ldg(lp);
                for (int o = 0; o < 4; ++o) {
                    if ((lane >> 3) == o) {
                        if constexpr (GS == 4) {
                            V *bp = bins_of(w.x);
                            *bp = octet_sum(row(w.x), row(w.y), row(w.z), row(w.w), w, *bp);
                        } else {
                            const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                V *bp = bins_of(ws[i]);
                                *bp = octet_add(*bp, row(ws[i]), ws[i]);
                            }
                        }
                    }
                    __syncwarp();
                }
            }
        }
        __syncthreads();
        if (chunk_u + 1 < nchunk && u + 1 < u1) continue;
        // ---- last chunk of this (tile, window) in the CTA's range: write the bins ----
        const int64_t gbeg = u - chunk_u, v0 = tile_u * C;
        const int64_t lo = (int64_t)win_u * p.g.sw;
        const int cnt = (int)min((int64_t)p.g.sw, p.s - lo);
        const int nc = (int)min((int64_t)C, p.nv - v0);
        // bins of bucket b, 16 bytes from column q * VR on (lanes along b: conflict-free)
        auto bin = [&](int b, int q) {
            V a = *reinterpret_cast<const V *>(bin_raw + b * BL_PITCH + q * 16);
            for (int r = 1; r < p.g.G; ++r) {
                const V x = *reinterpret_cast<const V *>(bin_raw + (r * p.g.sw + b) * BL_PITCH + q * 16);
                T *ae = reinterpret_cast<T *>(&a);
                const T *xe = reinterpret_cast<const T *>(&x);
#pragma unroll
                for (int e = 0; e < VR; ++e) ae[e] += xe[e];
            }
            return a;
        };
        if (u0 <= gbeg && gbeg + nchunk <= u1) {
            // lanes along the dimension that is contiguous in memory
            const bool down = p.y_es == 1;
            const int items = (down ? (cnt + 31) / 32 * 32 : cnt) * 8;
            for (int i0 = t; i0 < items; i0 += BL_WARPS * 32 * STEP) {
                T old[STEP][VR];
                auto item = [&](int k, auto f) {  // f(bucket, 16 bytes of its bins, address, elements left)
                    const int i = i0 + k * BL_WARPS * 32;
                    const int b = down ? (i >> 8) * 32 + lane : i >> 3, q = down ? (i >> 5) & 7 : i & 7;
                    if (b < cnt) f(b, q, p.Y + (lo + b) * p.y_es + (v0 + q * VR) * p.y_vs, nc - q * VR);
                };
                if constexpr (STEP > 1) {
#pragma unroll
                    for (int k = 0; k < STEP; ++k)
                        item(k, [&](int, int, const T *yp, int left) {
#pragma unroll
                            for (int e = 0; e < VR; ++e)
                                if (e < left) old[k][e] = yp[e * p.y_vs];
                        });
                }
#pragma unroll
                for (int k = 0; k < STEP; ++k)
                    item(k, [&](int b, int q, T *yp, int left) {
                        if (left <= 0) return;
                        const V a = bin(b, q);
#pragma unroll
                        for (int e = 0; e < VR; ++e)
                            if (e < left) {
                                T r = p.alpha * reinterpret_cast<const T *>(&a)[e];
                                if constexpr (STEP > 1) r += p.beta * old[k][e];
                                else if (!p.beta_zero) r += p.beta * yp[e * p.y_vs];
                                yp[e * p.y_vs] = r;
                            }
                    });
            }
        } else {
            V *part = reinterpret_cast<V *>(p.partials + (int64_t)p.split.slot(blockIdx.x, gbeg) * p.g.sw * C);
            for (int i = t; i < cnt * 8; i += BL_WARPS * 32) part[i] = bin(i >> 3, i & 7);
        }
        __syncthreads();
        if (u + 1 < u1) zero_bins();
    }
}

// Adds the partial bins of the (tile, window)s shared by several CTAs, in CTA order; 256 accesses of
// E elements per CTA, TR_AHEAD partials in flight.  One element per thread spreads a few (tile,
// window)s over the GPU: a single one has up to 148 partials, whose latency is all this kernel does
// (131072 x 1 Float32 to 100 buckets, nnz 2: 45 us a call; 108 us with four elements per thread and
// four partials in flight).  16 bytes per thread otherwise: the number of CTAs, most of them with two
// partials, counts then.  by_cut: CTA column x takes the (tile, window) that is cut where worker x + 1
// starts, if that is its first cut (at most W - 1 of them are shared, whatever their number); else
// (tile, window) x.
constexpr int TR_AHEAD = 16;
template <class T, int E>
__global__ void __launch_bounds__(256) tile_reduce_kernel(TileParams<T> p, int by_cut) {
    constexpr int C = TileCfg<T>::C, NB = 256 * E / C, AHEAD = TR_AHEAD / E;  // NB: buckets per CTA
    using V = std::conditional_t<E == 1, T, typename TileVec<T>::type>;
    __shared__ T tile[NB][C + 1];
    const int64_t cut = by_cut ? p.split.start(blockIdx.x + 1) : 0;
    const int64_t grp = by_cut ? cut / p.g.nchunk : blockIdx.x, gbeg = grp * p.g.nchunk;
    if (by_cut && cut == gbeg) return;
    const int gf = p.split.owner(gbeg), gl = p.split.owner(gbeg + p.g.nchunk - 1);
    if (by_cut ? gf != (int)blockIdx.x : gf == gl) return;  // another CTA's, or written by its only worker
    const int64_t lo = (grp % p.g.nwin) * p.g.sw, v0 = (grp / p.g.nwin) * C;
    const int cnt = (int)min((int64_t)p.g.sw, p.s - lo);
    const int b0 = blockIdx.y * NB, i = threadIdx.x * E;
    if (b0 >= cnt) return;
    const int64_t ps = (int64_t)p.g.sw * C;
    if (b0 + i / C < cnt) {
        const T *part = p.partials + b0 * C + i;
        T a[E];
        *reinterpret_cast<V *>(a) = ld_ahead(reinterpret_cast<const V *>(part + p.split.slot(gf, gbeg) * ps));
        for (int g0 = gf + 1; g0 <= gl; g0 += AHEAD) {
            V v[AHEAD];
#pragma unroll
            for (int k = 0; k < AHEAD; ++k) v[k] = ld_ahead(reinterpret_cast<const V *>(part + 2 * (int64_t)min(g0 + k, gl) * ps));
#pragma unroll
            for (int k = 0; k < AHEAD; ++k)
                if (g0 + k <= gl) {
#pragma unroll
                    for (int e = 0; e < E; ++e) a[e] += reinterpret_cast<const T *>(&v[k])[e];
                }
        }
#pragma unroll
        for (int e = 0; e < E; ++e) tile[i / C][i % C + e] = a[e];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < E; ++q) {
        const int k = threadIdx.x + 256 * q;
        const int b = p.y_es == 1 ? k % NB : k / C, c = p.y_es == 1 ? k / NB : k % C;
        if (b0 + b >= cnt || v0 + c >= p.nv) continue;
        T *yp = p.Y + (lo + b0 + b) * p.y_es + (v0 + c) * p.y_vs;
        T r = p.alpha * tile[b][c];
        if (!p.beta_zero) r += p.beta * *yp;
        *yp = r;
    }
}

// Whether cutting (tile, window)s between W CTAs pays for the partial sums, against CTAs with whole
// ones.  It saves chunks on the longest CTA, each 2.7 us and 0.9 us per entry and window, and costs the
// reduction, 6.5 us and 5 us per 100000 partial bins (least squares over 1113 calls of nnz 2 to 8, s up
// to 8320, 700 to 100000 long, both types; us a call, whole / cut):
//   Float32, nnz 2: 2000 x 1000 to 1000 43 / 38; 1000 x 3000 to 1000 39 / 54; 4000 x 10000 to 2080 188 / 191;
//   100000 x 200 to 500 677 / 70.
static bool sharing_pays(const rla_sketch *sk, const BlGeom &g, int64_t groups, int64_t W) {
    const int64_t saved = ceil_div(groups, W) * g.nchunk - ceil_div(groups * g.nchunk, W);
    const double bins = (double)std::min<int64_t>(2 * W, W + groups) * g.sw;
    return saved * (2.7 + 0.9 * sk->nnz / g.nwin) > 6.5 + 5e-5 * bins;
}

template <class T>
int tile_compress(rla_ctx *ctx, const rla_sketch *sk, const T *X, int64_t x_es, int64_t x_vs, int64_t nv, T *Y,
                  int64_t y_es, int64_t y_vs, T alpha, T beta, bool beta_zero) {
    constexpr int VR = TileCfg<T>::VR, C = TileCfg<T>::C;
    BlGeom g;
    if (!sk->bl_ok || !bl_geometry(sk, &g)) return set_error(ctx, RLA_E_UNSUPPORTED, "no bucket lists for this sketch");
    const int64_t groups = ceil_div(nv, C) * g.nwin, units = groups * g.nchunk;
    int W = (int)std::min<int64_t>(ctx->sm_count, units);
    void *part = nullptr;
    const size_t part_bytes = (size_t)(2 * W) * g.sw * C * sizeof(T);
    // No partial sums when each CTA has whole (tile, window)s: in a graph capture that finds the
    // scratch too small, or has four rounds of them (a captured scratch must not be grown later).
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    RLA_CUDA_TRY(ctx, cudaStreamIsCapturing(ctx->stream, &cap));
    const bool whole = cap != cudaStreamCaptureStatusNone &&
                       (ctx->scratch.bytes < part_bytes || groups >= 4 * (int64_t)ctx->sm_count);
    const bool shared = W > 1 && g.nchunk > 1 && !whole && sharing_pays(sk, g, groups, W);
    if (shared) RLA_TRY(scratch_get(ctx, part_bytes, &part));
    else W = (int)std::min<int64_t>(ctx->sm_count, groups);
    const bool contig = x_es == 1;
    TileParams<T> p{X, contig ? x_vs : x_es, sk->L, nv, sk->s, sk->bl_words, sk->bl_lists, g, Y, y_es, y_vs,
                    alpha, beta, beta_zero, (T *)part, Split::make(shared ? units : groups, W), shared ? 1 : g.nchunk};
    const size_t smem = (size_t)BL_TILE_BYTES + (size_t)(g.sw * g.G + 1) * BL_PITCH;
    const bool aligned = (nv == 1 && contig) || p.x_ld % VR == 0;
    const bool vec = aligned && (uintptr_t)X % 16 == 0;
    auto go = [&](auto kern) -> int {
        RLA_CUDA_TRY(ctx, set_smem_max(kern));
        kern<<<W, BL_WARPS * 32, smem, ctx->stream>>>(p);
        return check_launch(ctx, "tile_compress");
    };
    auto by_mode = [&](auto gs, auto step) -> int {
        constexpr int GS = decltype(gs)::value, ST = decltype(step)::value;
        if (contig) return vec ? go(tile_compress_kernel<T, TILE_CONTIG, GS, ST>) : go(tile_compress_kernel<T, TILE_SHIFT, GS, ST>);
        return vec ? go(tile_compress_kernel<T, TILE_ROWS, GS, ST>) : go(tile_compress_kernel<T, TILE_ROWS_ANY, GS, ST>);
    };
    // With beta a tile of few chunks waits longer for the old values, one by one, than for its
    // sums (1002 x 43482 Float64 to 1002, nnz 4: 710 us a call, 527 with four at a time); their
    // registers slow down the sums of longer ones (490312 x 99 Float32 from the right, s = 3194: 345 / 422).
    using One = std::integral_constant<int, 1>;
    using Four = std::integral_constant<int, 4>;
    const bool ahead = !beta_zero && g.nchunk <= 16;
    if (g.gs == 4) RLA_TRY(ahead ? by_mode(Four(), Four()) : by_mode(Four(), One()));
    else RLA_TRY(ahead ? by_mode(One(), Four()) : by_mode(One(), One()));
    if (!shared) return RLA_OK;
    const int by_cut = groups > W - 1;
    const unsigned gx = (unsigned)(by_cut ? W - 1 : groups);
    // one element per thread while its grid is one round of CTAs (8 per SM)
    const int scalar = ceil_div_i(g.sw, 256 / C);
    if ((int64_t)gx * scalar <= (int64_t)ctx->sm_count * 8)
        tile_reduce_kernel<T, 1><<<dim3(gx, scalar), 256, 0, ctx->stream>>>(p, by_cut);
    else
        tile_reduce_kernel<T, VR><<<dim3(gx, ceil_div_i(g.sw, 256 * VR / C)), 256, 0, ctx->stream>>>(p, by_cut);
    return check_launch(ctx, "tile_reduce");
}

template int tile_compress<float>(rla_ctx *, const rla_sketch *, const float *, int64_t, int64_t, int64_t, float *, int64_t,
                                  int64_t, float, float, bool);
template int tile_compress<double>(rla_ctx *, const rla_sketch *, const double *, int64_t, int64_t, int64_t, double *,
                                   int64_t, int64_t, double, double, bool);

}  // namespace rla
