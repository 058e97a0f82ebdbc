// rla_sparse_lift.cu -- SparseSign / CountSketch expand (S'*Y, A*S' ...) on tiles of vectors.
//
// Y(j, v) = alpha * sum_e sign(j, e) * X(bucket(j, e), v) + beta * Y(j, v), j < L.  The short
// operand X (s rows) is staged once per tile of vectors in shared memory, one row per bucket, so
// that LPE lanes read an entry's values with 16-byte accesses: one conflict-free wavefront per 128
// bytes.  Each warp takes 32 long indices at a time: it packs their entries into 16-bit words,
// sums the nnz rows of four (32/LPE) long indices per step in registers, and turns the 32 x C
// block of results through shared memory into 16-byte column stores.  Bound by the row reads
// (nnz wavefronts per 128 bytes of output; shared-memory pipe 79 % busy, the output's HBM
// traffic alone would take 32 us): 131072 x 200 Float64, s = 1000, nnz = 8 in 120 us, 436 us with
// a thread per output element.  The entry loop is unrolled for the usual nnz (154 us without).
//
// LPE = 8 / 4 / 2 lanes per entry (rows of 128 / 64 / 32 bytes) for s up to 1095 / 2380 / 4309 at
// nnz = 8 (1137 / 2457 / 4437 at nnz <= 2): the widest row that fits; above, and for calls too small
// to pay for the staging (lift_pays), the thread-per-element kernel of rla_sparse.cu.
#include "rla_internal.cuh"
#include "rla_kernels.cuh"

namespace rla {

constexpr int LIFT_WARPS = 16, LIFT_MAX_NNZ = 32;  // most warps of a CTA

template <class T, int LPE>
struct LiftCfg {
    static constexpr int VR = 16 / (int)sizeof(T);  // elements per 16 bytes
    static constexpr int C = LPE * VR;              // vectors per tile
    static constexpr int PITCH = LPE * 16 + 16;     // bytes per staged row: 16-byte column writes conflict-free
    static constexpr int JS = 32 / LPE;             // long indices per step
    static constexpr int OUT = 32 * LPE * 16;       // bytes of a warp's result block
};

template <class T>
struct LiftParams {
    const T *X;
    int64_t x_es, x_vs, L, nv, s;
    const int32_t *bucket;
    const uint8_t *negative;
    int nnz, wpj;  // wpj: 16-bit words kept per long index (nnz rounded up to even)
    T *Y;
    int64_t y_es, y_vs;
    T alpha, beta;
    int beta_zero;
    int64_t nblk;  // blocks of 32 long indices
    Split split;   // over (tile, a block of 32 long indices per warp)
};

__device__ __forceinline__ void lift_add(float4 &a, float4 x, uint32_t sign) {
    const float s = __uint_as_float(sign | 0x3f800000u);
    const float2 s2 = make_float2(s, s);
    const float2 lo = __ffma2_rn(make_float2(x.x, x.y), s2, make_float2(a.x, a.y));
    const float2 hi = __ffma2_rn(make_float2(x.z, x.w), s2, make_float2(a.z, a.w));
    a = make_float4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ void lift_add(double2 &a, double2 x, uint32_t sign) {
    const long long m = (long long)sign << 32;
    a.x += __longlong_as_double(__double_as_longlong(x.x) ^ m);
    a.y += __longlong_as_double(__double_as_longlong(x.y) ^ m);
}

// Slot of 16 bytes q of row j in a warp's result block: the column reads below (8 lanes along
// j in steps of VR, 4 columns) then hit distinct banks for LPE = 8.
template <class T, int LPE>
__device__ __forceinline__ int lift_slot(int j, int q) {
    constexpr int VR = LiftCfg<T, LPE>::VR;
    return q ^ ((j / VR + (8 / VR) * (j % VR)) & (LPE - 1));
}

// NNZ: entries per long index when it is a compile-time 1, 2, 4 or 8, else 0 (p.nnz).
template <class T, int LPE, int NNZ>
__global__ void __launch_bounds__(LIFT_WARPS * 32, 1) lift_kernel(LiftParams<T> p) {
    using Cfg = LiftCfg<T, LPE>;
    using V = std::conditional_t<sizeof(T) == 4, float4, double2>;
    constexpr int VR = Cfg::VR, C = Cfg::C, JS = Cfg::JS;
    const int nnz = NNZ ? NNZ : p.nnz, wpj = NNZ ? (NNZ + 1) / 2 * 2 : p.wpj;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int t = threadIdx.x, lane = t & 31, wp = t >> 5, nt = blockDim.x, warps = nt >> 5;
    unsigned char *out = smem_raw + wp * Cfg::OUT;
    uint16_t *words = reinterpret_cast<uint16_t *>(smem_raw + warps * Cfg::OUT) + wp * 32 * wpj;
    unsigned char *xs = smem_raw + warps * (Cfg::OUT + 32 * wpj * 2);
    const int64_t u0 = p.split.start(blockIdx.x), u1 = p.split.start(blockIdx.x + 1);
    const int64_t nj = (p.nblk + warps - 1) / warps;
    int64_t have = -1;
    for (int64_t u = u0; u < u1; ++u) {
        const int64_t tile = u / nj, v0 = tile * C;
        const int nc = (int)min((int64_t)C, p.nv - v0);
        if (tile != have) {  // stage X(:, v0 .. v0 + C): row b at b * PITCH
            __syncthreads();
            have = tile;
            if (p.x_es == 1) {
                // lanes along b; VR vectors per thread make one 16-byte store
                const int ss = (int)p.s;
                for (int i = t; i < ss * LPE; i += nt) {
                    const int q = i / ss, b = i - q * ss;
                    V y{};
                    T *ye = reinterpret_cast<T *>(&y);
#pragma unroll
                    for (int e = 0; e < VR; ++e)
                        if (q * VR + e < nc) ye[e] = __ldg(p.X + b + (v0 + q * VR + e) * p.x_vs);
                    *reinterpret_cast<V *>(xs + b * Cfg::PITCH + q * 16) = y;
                }
            } else {
                for (int i = t; i < (int)p.s * C; i += nt) {
                    const int b = i / C, c = i % C;
                    *reinterpret_cast<T *>(xs + b * Cfg::PITCH + c * sizeof(T)) =
                        c < nc ? __ldg(p.X + b * p.x_es + (v0 + c) * p.x_vs) : T(0);
                }
            }
            __syncthreads();
        }
        const int64_t blk = (u - tile * nj) * warps + wp;
        if (blk >= p.nblk) continue;  // warp-uniform
        const int64_t j0 = blk * 32;
        const int cnt = (int)min((int64_t)32, p.L - j0);
        // ---- the block's entries: bucket | sign << 15, lane = long index when nnz is known ----
        if constexpr (NNZ > 0) {
            if (lane < cnt) {
                const int32_t *bp = p.bucket + (j0 + lane) * NNZ;
                const uint8_t *np = p.negative + (j0 + lane) * NNZ;
                int32_t b[NNZ];
                uint32_t n[NNZ];
                if constexpr (NNZ == 8) {
                    const int4 b0 = __ldg(reinterpret_cast<const int4 *>(bp)), b1 = __ldg(reinterpret_cast<const int4 *>(bp) + 1);
                    const uint2 m = __ldg(reinterpret_cast<const uint2 *>(np));
                    const int32_t bb[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        b[e] = bb[e];
                        n[e] = ((e < 4 ? m.x : m.y) >> (8 * (e & 3))) & 1u;
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < NNZ; ++e) {
                        b[e] = __ldg(bp + e);
                        n[e] = __ldg(np + e);
                    }
                }
                uint32_t *wo = reinterpret_cast<uint32_t *>(words + lane * wpj);
#pragma unroll
                for (int e = 0; e < NNZ; e += 2) {
                    uint32_t w = (uint32_t)b[e] | (n[e] << 15);
                    if (e + 1 < NNZ) w |= ((uint32_t)b[(e + 1) % NNZ] << 16) | (n[(e + 1) % NNZ] << 31);
                    wo[e / 2] = w;
                }
            }
        } else {
            for (int i = lane; i < cnt * nnz; i += 32) {
                const int jl = i / nnz;
                words[jl * wpj + i - jl * nnz] =
                    (uint16_t)((uint32_t)__ldg(p.bucket + j0 * nnz + i) | ((uint32_t)__ldg(p.negative + j0 * nnz + i) << 15));
            }
        }
        if (!p.beta_zero) {  // the old values of the block come into L2 during its sums
            const T *yb = p.Y + j0 * p.y_es + v0 * p.y_vs;
            if (p.y_es == 1) {
                for (int c = 0; c < nc; ++c)
                    if (lane < cnt) asm volatile("prefetch.global.L2 [%0];" ::"l"(yb + lane + c * p.y_vs));
            } else {
                for (int i = lane; i < cnt * C; i += 32)
                    if (i % C < nc) asm volatile("prefetch.global.L2 [%0];" ::"l"(yb + i / C * p.y_es + i % C * p.y_vs));
            }
        }
        __syncwarp();
        // ---- sums of JS long indices per step ----
        const int l = lane % LPE, g = lane / LPE;
        const unsigned char *xl = xs + l * 16;
        auto entry = [&](V &a, uint32_t b, uint32_t sign) {
            lift_add(a, *reinterpret_cast<const V *>(xl + b * Cfg::PITCH), sign);
        };
#pragma unroll 2
        for (int q = 0; q < LPE; ++q) {
            const int jl = q * JS + g;
            V a{};
            if (jl < cnt) {
                const uint16_t *wj = words + jl * wpj;
                auto pair = [&](uint32_t w) {
                    entry(a, w & 0x7fffu, (w << 16) & 0x80000000u);
                    entry(a, (w >> 16) & 0x7fffu, w & 0x80000000u);
                };
                if constexpr (NNZ == 8) {
                    const uint4 w = *reinterpret_cast<const uint4 *>(wj);
                    pair(w.x);
                    pair(w.y);
                    pair(w.z);
                    pair(w.w);
                } else {
                    const uint32_t *w2 = reinterpret_cast<const uint32_t *>(wj);
                    int e = 0;
#pragma unroll
                    for (; e + 2 <= nnz; e += 2) pair(w2[e >> 1]);
                    if (e < nnz) {
                        const uint32_t w = wj[e];
                        entry(a, w & 0x7fffu, (w << 16) & 0x80000000u);
                    }
                }
            }
            *reinterpret_cast<V *>(out + jl * (LPE * 16) + lift_slot<T, LPE>(jl, l) * 16) = a;
        }
        __syncwarp();
        // ---- write the 32 x C block ----
        auto get = [&](int j, int c) {
            return *reinterpret_cast<const T *>(out + j * (LPE * 16) + lift_slot<T, LPE>(j, c / VR) * 16 + (c % VR) * sizeof(T));
        };
        const bool y16 = reinterpret_cast<uintptr_t>(p.Y) % 16 == 0;
        T *yb = p.Y + j0 * p.y_es + v0 * p.y_vs;
        if (!p.beta_zero) {
            // lanes along the contiguous dimension; the old values of eight elements per lane are read
            // before the first one is written (131072 x 200 Float64 from 1000, nnz 8: 281 us a call one by
            // one, 189 now)
            constexpr int STEP = 8;
            const bool down = p.y_es == 1;
            for (int i0 = 0; i0 < (down ? C : cnt * C / 32 + 1); i0 += STEP) {
                T old[STEP];
                auto row = [&](int i) { return down ? lane : (32 * (i0 + i) + lane) / C; };
                auto col = [&](int i) { return down ? i0 + i : lane % C; };  // C divides 32
                auto on = [&](int i) { return row(i) < cnt && col(i) < nc; };
#pragma unroll
                for (int i = 0; i < STEP; ++i)
                    if (on(i)) old[i] = yb[row(i) * p.y_es + col(i) * p.y_vs];
#pragma unroll
                for (int i = 0; i < STEP; ++i)
                    if (on(i)) yb[row(i) * p.y_es + col(i) * p.y_vs] = p.alpha * get(row(i), col(i)) + p.beta * old[i];
            }
        } else if (p.y_es == 1) {
            if (cnt == 32 && p.y_vs % VR == 0 && y16) {
                // 8 lanes along j, VR rows each, of 4 columns per pass
                constexpr int RB = 32 / (8 * VR);
#pragma unroll
                for (int i = 0; i < RB * (C / 4); ++i) {
                    const int c = (i / RB) * 4 + (lane >> 3), j = ((i % RB) * 8 + (lane & 7)) * VR;
                    V y;
                    T *ye = reinterpret_cast<T *>(&y);
#pragma unroll
                    for (int e = 0; e < VR; ++e) ye[e] = p.alpha * get(j + e, c);
                    if (c < nc) *reinterpret_cast<V *>(yb + j + c * p.y_vs) = y;
                }
            } else {
                for (int c = 0; c < nc; ++c)
                    if (lane < cnt) yb[lane + c * p.y_vs] = p.alpha * get(lane, c);
            }
        } else {
            for (int i = lane; i < cnt * C; i += 32)
                if (i % C < nc) yb[i / C * p.y_es + i % C * p.y_vs] = p.alpha * get(i / C, i % C);
        }
        __syncwarp();
    }
}

// Lanes per entry whose staged rows fit next to the warps' blocks, 0 when none do.
template <class T>
static int lift_lanes(const rla_ctx *ctx, const rla_sketch *sk, size_t *smem) {
    const int wpj = ((int)sk->nnz + 1) / 2 * 2;
    if (sk->nnz > LIFT_MAX_NNZ || sk->s >= 32768) return 0;
    for (int lpe = 8; lpe >= 2; lpe /= 2) {
        *smem = (size_t)LIFT_WARPS * (32 * lpe * 16 + 32 * wpj * 2) + (size_t)sk->s * (lpe * 16 + 16);
        if (*smem <= (size_t)ctx->smem_optin - 1024) return lpe;
    }
    return 0;
}

// How a call is spread: fewer warps per CTA while that spreads a small call over more SMs (every CTA
// stages X).
struct LiftGrid {
    int64_t tiles, blocks_per_tile, units;  // vector tiles, groups of a block per warp, their product
    int warps, W;
    int64_t stagings;  // most tiles that a CTA stages
    static LiftGrid make(const rla_ctx *ctx, int64_t L, int64_t nv, int64_t C) {
        LiftGrid g;
        const int64_t nblk = ceil_div(L, 32);
        g.tiles = ceil_div(nv, C);
        g.warps = LIFT_WARPS;
        while (g.warps > 4 && g.tiles * ceil_div(nblk, g.warps) < ctx->sm_count) g.warps /= 2;
        g.blocks_per_tile = ceil_div(nblk, g.warps);
        g.units = g.tiles * g.blocks_per_tile;
        g.W = (int)std::min<int64_t>(ctx->sm_count, g.units);
        g.stagings = ceil_div(ceil_div(g.units, g.W), g.blocks_per_tile);
        return g;
    }
};

// Whether staging pays, against a thread per output element (rla_sparse.cu).  Times of a call in
// us, that kernel / this one, Float32 unless named:
//  * Column-major results of 1024 rows and more.  That kernel takes about (2 + nnz) ps more per output;
//    staging costs about 8 us at s = 1000 (8 lanes), twice that from a row-major short operand: 30000 x
//    16, nnz 8, s = 1000: 33 / 38; 131072 x 32, nnz 1: 42 / 36.  A tile of 32 (Float64: 16) vectors
//    that is mostly empty costs as much as a full one: 2^20 long indices of nnz 8, 1 vector
//    38 / 73, 4 vectors 81 / 72; nnz 1, 4 vectors 41 / 48, 8 vectors 57 / 49; nnz 3 (no unrolled
//    loop) 8 vectors 67 / 73, 16 vectors 110 / 81.  With beta the old values take this one longer: Float64
//    1000481 x 22, nnz 3 155 / 220, 131072 x 200, nnz 8 442 / 189; 4239 x 179, nnz 12: 30 / 40.
//  * Other results by the sum of what each kernel spends (below).  Row-major: that kernel's blocks
//    hold 128 vectors whatever their number is, and read a column-major operand across: 2^20 x 2,
//    nnz 8: 300 / 95; 30000 x 32, nnz 8, s = 1000: 39 / 51; 131072 x 16, nnz 1: 66 / 42; 8000 x 500, nnz 16,
//    s = 1000, column-major operand: 235 / 47.  Short columns: 50 x 100000, nnz 3 Float64 71 / 196, 200 x
//    40000, nnz 8 131 / 79.
//  * Rows off 32-byte boundaries leave neighbouring tiles parts of one sector, and the result
//    does not stay in L2 until both are written: Float64, row-major operand, odd leading dimension,
//    nnz 1, 30000 x 1000: s = 2000 160 / 296; s = 1000 with nnz 3 209 / 257, but nnz 8 272 / 243;
//    column-major operand, s = 1 149 / 224, s = 1000 197 / 187.
//  * Two lanes per entry, Float64: tiles of 4 vectors write 32-byte pieces of rows (2^20 x 64, nnz 1:
//    302 / 401), and with nnz 3 the words of 2^20 long indices are read again for every four
//    columns (2^20 x 64: 415 / 485; 131072 x 200: 226 / 178); with beta 229508 x 198, nnz 1: 304 / 379, and 29150 x
//    1119, nnz 2, row-major: 335 / 480.
template <class T>
static bool lift_pays(const rla_sketch *sk, const LiftGrid &g, int lpe, int64_t x_es, int64_t nv, int64_t y_es, bool beta) {
    if (nv < 2) return false;
    const int64_t L = sk->L, nnz = sk->nnz, staged = sk->s * lpe;
    const bool unrolled = nnz == 1 || nnz == 2 || nnz == 4 || nnz == 8, narrow64 = sizeof(T) == 8 && lpe == 2;
    const bool rows_in = x_es != 1, rows_out = y_es != 1;
    if (narrow64 && beta && nnz <= 2) return false;
    if (rows_out) {
        if (narrow64 && nv > 32 && nnz != 8 && rows_in) return false;
        if (y_es * sizeof(T) % 32 != 0 && L * nv * (int64_t)sizeof(T) > 110000000 && g.tiles > 3) {
            if (rows_in && (sizeof(T) == 8 ? lpe < 8 || nnz < 8 : lpe == 2)) return false;
            if (!rows_in && sizeof(T) == 8 && nnz == 1 && (sk->s <= 300 || lpe < 8)) return false;
        }
    } else {
        if (narrow64 && !unrolled && nnz < 8 && L >= (1 << 19)) return false;
        if (L >= 1024) {
            if (nv < (nnz >= 8 ? 4 : unrolled ? 8 : 16) || (beta && nnz < 4)) return false;
            return L * nv * (2 + nnz) >= (beta ? 2 : 1) * std::max<int64_t>(1000 * staged * (rows_in ? 2 : 1), 6000000);
        }
    }
    // us: that kernel's blocks of 128 outputs, gathered values and output bytes; here the stagings, their
    // rows (of one staging for row-major results, of all of them for short columns), bytes and values
    // (least squares over 5200 calls of nnz 1 to 16, s up to 4000, both types)
    struct Cost {
        double block, value, byte, staging, row, byte_here, value_here;
    };
    static constexpr Cost costs[2][2] = {{{10.1e-5, 1.33e-6, 0.22e-6, 2.3, 0.72e-3, 0.13e-6, 0.041e-6},
                                          {0.0, 2.52e-6, 0.31e-6, 2.3, 0.82e-3, 0.12e-6, 0.045e-6}},
                                         {{16.2e-5, 2.14e-6, 0.20e-6, 1.5, 0.92e-3, 0.33e-6, 0.043e-6},
                                          {19.9e-5, 0.56e-6, 0.28e-6, 2.0, 1.15e-3, 0.29e-6, 0.048e-6}}};
    const Cost &c = costs[rows_out][rows_in];
    const double values = (double)L * nv * nnz, bytes = (double)L * nv * sizeof(T);
    const double there = c.block * (rows_out ? L * ceil_div(nv, 128) : ceil_div(L, 128) * nv) + c.value * values + c.byte * bytes;
    const double here = c.staging * g.stagings + c.row * staged * (rows_out ? 1 : g.stagings) + c.byte_here * bytes +
                        c.value_here * values * sizeof(T);
    return there > here + (beta ? 6.0 : 1.5);  // beta: the old values add latency here
}

template <class T>
int sparse_lift(rla_ctx *ctx, const rla_sketch *sk, const T *X, int64_t x_es, int64_t x_vs, int64_t nv, T *Y,
                int64_t y_es, int64_t y_vs, T alpha, T beta, bool beta_zero, bool *taken) {
    size_t smem = 0;
    const int lpe = lift_lanes<T>(ctx, sk, &smem);
    *taken = false;
    if (!lpe) return RLA_OK;
    const LiftGrid g = LiftGrid::make(ctx, sk->L, nv, lpe * (16 / (int64_t)sizeof(T)));
    *taken = lift_pays<T>(sk, g, lpe, x_es, nv, y_es, !beta_zero);
    if (!*taken) return RLA_OK;
    LiftParams<T> p{X, x_es, x_vs, sk->L, nv, sk->s, sk->bucket, sk->negative, (int)sk->nnz, ((int)sk->nnz + 1) / 2 * 2,
                    Y, y_es, y_vs, alpha, beta, beta_zero, ceil_div(sk->L, 32), Split::make(g.units, g.W)};
    auto go = [&](auto kern) -> int {
        RLA_CUDA_TRY(ctx, set_smem_max(kern));
        kern<<<g.W, g.warps * 32, smem, ctx->stream>>>(p);
        return check_launch(ctx, "sparse_lift");
    };
    auto by_nnz = [&](auto lanes) -> int {
        constexpr int N = decltype(lanes)::value;
        switch (sk->nnz) {
            case 1: return go(lift_kernel<T, N, 1>);
            case 2: return go(lift_kernel<T, N, 2>);
            case 4: return go(lift_kernel<T, N, 4>);
            case 8: return go(lift_kernel<T, N, 8>);
            default: return go(lift_kernel<T, N, 0>);
        }
    };
    if (lpe == 8) return by_nnz(std::integral_constant<int, 8>());
    if (lpe == 4) return by_nnz(std::integral_constant<int, 4>());
    return by_nnz(std::integral_constant<int, 2>());
}

template int sparse_lift<float>(rla_ctx *, const rla_sketch *, const float *, int64_t, int64_t, int64_t, float *, int64_t,
                                int64_t, float, float, bool, bool *);
template int sparse_lift<double>(rla_ctx *, const rla_sketch *, const double *, int64_t, int64_t, int64_t, double *,
                                 int64_t, int64_t, double, double, bool, bool *);

}  // namespace rla
