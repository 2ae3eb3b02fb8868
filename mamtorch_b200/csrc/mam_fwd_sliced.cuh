// MAM forward for products with too few output tiles to fill the chip: the reduction is cut over a thread-block
// cluster, merged through distributed shared memory, and the indices are resolved in the same launch.
//
// mam_fwd_tiled_kernel gives every 64x128 tile to one CTA, which walks all of K.  A layer applied to a few tokens
// (8 x 768 x 3072: 24 tiles, seven eighths of each padding) or a small training step (256 x 512 x 256: 8 tiles)
// then occupies 8-24 of 148 SMs and its time is the length of that one serial walk: K / 32 chunks at about
// 3.4 us each, whatever M is.  Here
//  * the tile is small where M is small (8 or 32 rows), so less of it is padding;
//  * the CTAs of a cluster (up to 8) take consecutive ranges of 32-wide K chunks of one tile and meet once: each
//    leaves its running extremes (and chunk ids) in its own shared memory, and after a cluster barrier every CTA
//    reduces its share of the tile's outputs over the ranks in ascending order with strict compares, so the first
//    chunk that attains the extreme still wins;
//  * with indices, the recorded chunk of every output is rescanned right there (128 bytes of a and of W per extreme,
//    out of L2) for the first k that attains the extreme: the separate resolver launch, whose 64x128 tiles would
//    again leave most SMs idle, falls away.
// Values, indices and rounding are those of the tiled kernel: one rounded product, extremes by max / min, first k.
#pragma once
#include "mam_fwd_tiled.cuh"

namespace mamb200 {

template <int TM_, int TN_, int WM_, int WN_, int STAGES_, bool TRACK_>
struct SlicedCfg {
    static constexpr int TM = TM_, TN = TN_, WM = WM_, WN = WN_, STAGES = STAGES_;
    static constexpr bool TRACK = TRACK_;
    static constexpr int BM = WM * 4 * TM, BN = WN * 8 * TN;
    static constexpr int WARPS = WM * WN, THREADS = WARPS * 32, SLOTS = TM * TN;
    static constexpr int A_BYTES = BM * FWD_BK * 4, W_BYTES = BN * FWD_BK * 4, STAGE_BYTES = A_BYTES + W_BYTES;
    static constexpr int RING_BYTES = STAGES * STAGE_BYTES;
    static constexpr int PART_BYTES = 2 * SLOTS * THREADS * 4;      // both extremes of every output, over the ring
    static constexpr int ID_BYTES = TRACK ? 2 * SLOTS * THREADS * 2 : 0;
    static constexpr int BAR_BYTES = 2 * STAGES * 8;
    static constexpr int SMEM_BYTES = 1024 + RING_BYTES + BAR_BYTES + ID_BYTES;
    // CTAs per SM that shared memory leaves room for, with the registers to match: the 32x64 tile runs 5 (values) and 4
    // (indices) of them; one fewer costs a fifth (68x1780x2415 with indices 60 -> 76 us, 11773x62x4 values 13.5 -> 16.5)
    static constexpr int MIN_CTAS = THREADS > 128 ? 1 : TRACK ? 512 / THREADS : THREADS == 128 ? 5 : 4;
    static_assert(TM % 2 == 0, "row swizzle keys assume an even TM");
    static_assert(BM <= 256 && BN <= 256, "TMA box rows");
    static_assert(PART_BYTES <= RING_BYTES, "the partial extremes reuse the operand ring");
};

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_ranks() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t peer_smem(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ float peer_f32(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ unsigned peer_u16(uint32_t addr) {
    unsigned short v;
    asm volatile("ld.shared::cluster.u16 %0, [%1];" : "=h"(v) : "r"(addr) : "memory");
    return v;
}

// One index per lane: the first k of the 32-wide chunk `c` of this lane's output whose product a[k]*w[k] equals `v`;
// the chunk's first k if none does (every product is NaN).  The eight lanes of a quarter-warp hold eight neighbouring
// outputs of one row and work on one output at a time, each lane on four k, so that a load instruction touches
// four 128-byte lines of a and of W; a lane on its own chunk instead touches 32 (256 x 512 x 256, whole forward: 17.6
// us that way, 13.2 this way).  All sixteen loads are issued before the first compare (19.0 us one after the other).  Rows, columns and k outside are clamped for the loads and never match.  K % 4 == 0, rows
// 16-byte aligned.
__device__ __forceinline__ int first_in_chunk(const float* __restrict__ a, const float* __restrict__ w, long long m,
                                              long long n_quarter, long long M, long long N, long long K, unsigned c,
                                              float v, int lane) {
    const float* arow = a + min(m, M - 1) * K;
    float4 x[8], z[8];
    int k[8];
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        k[s] = (int)__shfl_sync(0xffffffffu, c, s, 8) * FWD_BK + 4 * (lane & 7);
        const long long kc = min((long long)k[s], K - 4);
        x[s] = __ldg(reinterpret_cast<const float4*>(arow + kc));
        z[s] = __ldg(reinterpret_cast<const float4*>(w + min(n_quarter + s, N - 1) * K + kc));
    }
    int mine = 0;
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        const float want = __shfl_sync(0xffffffffu, v, s, 8);
        int hit = 4;
        if (__fmul_rn(x[s].w, z[s].w) == want) hit = 3;
        if (__fmul_rn(x[s].z, z[s].z) == want) hit = 2;
        if (__fmul_rn(x[s].y, z[s].y) == want) hit = 1;
        if (__fmul_rn(x[s].x, z[s].x) == want) hit = 0;
        const unsigned hits = __ballot_sync(0xffffffffu, hit < 4 && k[s] < K) >> (lane & 24) & 0xffu;
        const int from = hits ? __ffs(hits) - 1 : 0;
        // without a hit lane 0 of the quarter holds the chunk's first k
        const int got = __shfl_sync(0xffffffffu, k[s] + (hits ? hit : 0), from, 8);
        if ((lane & 7) == s) mine = got;
    }
    return mine;
}

struct SlicedParams {
    const float* a;   // the operands again, for the index pass
    const float* w;
    float* y;
    int* argmax;
    int* argmin;
    long long M, K, N;
    EpilogueArgs ep;
    float one;        // 1.0f kept opaque to the compiler
    int* error;
};

// grid: tiles x cluster size, consecutive CTAs form the cluster of one tile; tiles n-fastest.
template <class Cfg>
__global__ void __launch_bounds__(Cfg::THREADS, Cfg::MIN_CTAS)
mam_fwd_sliced_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW,
                      const SlicedParams prm) {
    constexpr int TM = Cfg::TM, TN = Cfg::TN, STAGES = Cfg::STAGES, THREADS = Cfg::THREADS;
    constexpr bool TRACK = Cfg::TRACK;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + Cfg::RING_BYTES);
    uint64_t* empty_bar = full_bar + STAGES;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_rank(), ranks = cluster_ranks();
    const long long M = prm.M, K = prm.K, N = prm.N;
    const int ntn = (int)((N + Cfg::BN - 1) / Cfg::BN);
    const long long tile = blockIdx.x / ranks;
    const long long m0 = tile / ntn * Cfg::BM, n0 = tile % ntn * Cfg::BN;
    const int nk = (int)((K + FWD_BK - 1) / FWD_BK);
    const int tail_quads = (int)((K - (long long)(nk - 1) * FWD_BK) / 4);
    const int c_begin = (int)((long long)nk * rank / ranks), c_end = (int)((long long)nk * (rank + 1) / ranks);

    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], Cfg::WARPS);
        }
        mbar_fence_init();
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmW);
    }
    __syncthreads();

    auto issue = [&](int c) {   // one thread: chunk c into its stage of the ring
        const int s = (c - c_begin) % STAGES;
        mbar_expect_tx(&full_bar[s], Cfg::STAGE_BYTES);
        unsigned char* dst = smem + s * Cfg::STAGE_BYTES;
        tma_load_2d(dst, &tmA, &full_bar[s], c * FWD_BK, (int)m0);
        tma_load_2d(dst + Cfg::A_BYTES, &tmW, &full_bar[s], c * FWD_BK, (int)n0);
    };
    int issued = 0;   // copies of chunks, counted by the thread that issues them
    if (tid == 0)
        for (int c = c_begin; c < c_end && c < c_begin + STAGES; ++c, ++issued) issue(c);

    const int wm = warp / Cfg::WN, wn = warp % Cfg::WN, lane_m = lane >> 3, lane_n = lane & 7;
    const int a_first = wm * 4 * TM + lane_m, w_first = wn * 8 * TN + lane_n;
    const uint32_t smem_base = smem_u32(smem);
    const uint32_t a_row0 = (uint32_t)a_first * 128u, w_row0 = (uint32_t)Cfg::A_BYTES + (uint32_t)w_first * 128u;
    const uint32_t a_key = (uint32_t)lane_m << 4, w_key = (uint32_t)lane_n << 4;
    const uint32_t id_addr = smem_base + Cfg::RING_BYTES + Cfg::BAR_BYTES + (uint32_t)tid * 2u;

    float vmax[TM][TN], vmin[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            vmax[i][j] = -INFINITY;
            vmin[i][j] = INFINITY;
        }
    if constexpr (TRACK) {
#pragma unroll
        for (int s = 0; s < 2 * Cfg::SLOTS; ++s) sts16_s(id_addr + s * THREADS * 2, (unsigned)c_begin);
    }

    // After a wait that gave up nothing more is waited for, released or issued (by the lane concerned; a stage is released
    // by lanes that saw its copy land, and the issuing thread saw it released): the loop runs out on what the ring
    // holds, and the CTA comes to the cluster barriers with its copies waited for below.
    bool ok = true;
    for (int c = c_begin; c < c_end; ++c) {
        const int it = c - c_begin, s = it % STAGES;
        ok = ok && mbar_wait_bounded(&full_bar[s], (uint32_t)(it / STAGES) & 1u);
        const uint32_t ap = smem_base + (uint32_t)(s * Cfg::STAGE_BYTES) + a_row0;
        const uint32_t wp = smem_base + (uint32_t)(s * Cfg::STAGE_BYTES) + w_row0;
        float lmax[TRACK ? TM : 1][TRACK ? TN : 1], lmin[TRACK ? TM : 1][TRACK ? TN : 1];
        auto quad = [&](const uint32_t qoff, const bool first) {
            const uint32_t xa0 = ap | (qoff ^ a_key), xa1 = xa0 ^ 64u, xw = wp | (qoff ^ w_key);
            ulonglong2 av[TM];
            static_for<0, TM>([&](auto ic) {
                constexpr int i = decltype(ic)::value;
                av[i] = lds128_at<i * 512>((i & 1) ? xa1 : xa0);
            });
            static_for<0, TN>([&](auto jc) {
                constexpr int j = decltype(jc)::value;
                const ulonglong2 wv = lds128_at<j * 1024>(xw);
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    float p0, p1, p2, p3;
                    unpack2(mul2(av[i].x, wv.x), p0, p1);
                    unpack2(mul2(av[i].y, wv.y), p2, p3);
                    if constexpr (TRACK) {
                        lmax[i][j] = first ? fmaxf(p0, p1) : fmax3(lmax[i][j], p0, p1);
                        lmin[i][j] = first ? fminf(p0, p1) : fmin3(lmin[i][j], p0, p1);
                        lmax[i][j] = fmax3(lmax[i][j], p2, p3);
                        lmin[i][j] = fmin3(lmin[i][j], p2, p3);
                    } else {
                        vmax[i][j] = fmax3(fmax3(vmax[i][j], p0, p1), p2, p3);
                        vmin[i][j] = fmin3(fmin3(vmin[i][j], p0, p1), p2, p3);
                    }
                }
            });
        };
        const uint32_t qend = (uint32_t)((c + 1 < nk) ? FWD_BK / 4 : tail_quads) << 4;
        quad(0u, true);
#pragma unroll 1
        for (uint32_t qoff = 16u; qoff < qend; qoff += 16u) quad(qoff, false);
        __syncwarp();
        if (lane == 0 && ok) mbar_arrive(&empty_bar[s]);
        if (tid == 0 && ok && c + STAGES < c_end) {   // refill the stage once every warp has left it
            ok = mbar_wait_bounded(&empty_bar[s], (uint32_t)(it / STAGES) & 1u);
            if (ok) {
                issue(c + STAGES);
                ++issued;
            }
        }
        __syncwarp();
        if constexpr (TRACK) {
            // merge of the chunk's extremes as in the tiled kernel: the value moves by a multiply with an opaque
            // 1.0, off the ALU pipe
            const unsigned short kid = (unsigned short)c;
            static_for<0, TM * TN>([&](auto slot) {
                constexpr int S = decltype(slot)::value, i = S / TN, j = S % TN;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.gt.f32 p, %1, %0;\n\t"
                    "@p mul.rn.f32 %0, %1, %2;\n\t"
                    "@p st.shared.u16 [%3+%5], %4;\n\t}"
                    : "+f"(vmax[i][j])
                    : "f"(lmax[i][j]), "f"(prm.one), "r"(id_addr), "h"(kid), "n"((S * 2 + 0) * THREADS * 2)
                    : "memory");
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.lt.f32 p, %1, %0;\n\t"
                    "@p mul.rn.f32 %0, %1, %2;\n\t"
                    "@p st.shared.u16 [%3+%5], %4;\n\t}"
                    : "+f"(vmin[i][j])
                    : "f"(lmin[i][j]), "f"(prm.one), "r"(id_addr), "h"(kid), "n"((S * 2 + 1) * THREADS * 2)
                    : "memory");
            });
        }
    }

    // ---- meet: extremes into the ring, then reduce over the ranks.  Every copy into the ring has landed and been read --
    // or a wait gave up: then the flag is set, the last copy of each stage is waited for once more (no CTA leaves with
    // copies in flight) and the ring is left alone; what the peers read from it is memory of this CTA all the same.
    const bool failed = __syncthreads_or(!ok);
    if (failed && tid == 0) {
        atomicExch(prm.error, 1);
        for (int it = max(0, issued - STAGES); it < issued; ++it)
            mbar_wait_bounded(&full_bar[it % STAGES], (uint32_t)(it / STAGES) & 1u);
    }
    float* part = reinterpret_cast<float*>(smem) + tid;     // [2 * slot + side][thread]
    if (!failed) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                part[(2 * (i * TN + j) + 0) * THREADS] = vmax[i][j];
                part[(2 * (i * TN + j) + 1) * THREADS] = vmin[i][j];
            }
    }
    __syncwarp();
    cluster_barrier();
    const uint32_t part_addr = smem_u32(part);
    for (uint32_t slot = rank; slot < (uint32_t)Cfg::SLOTS; slot += ranks) {
        const long long m = m0 + a_first + 4 * (int)(slot / TN), n = n0 + w_first + 8 * (int)(slot % TN);
        const bool mine = m < M && n < N;
        float hi = -INFINITY, lo = INFINITY;
        unsigned chi = 0, clo = 0;
        for (uint32_t r = 0; r < ranks; ++r) {
            const uint32_t pa = peer_smem(part_addr + 2 * slot * THREADS * 4, r);
            const float h = peer_f32(pa), l = peer_f32(pa + THREADS * 4);
            if constexpr (TRACK) {
                const uint32_t ia = peer_smem(id_addr + 2 * slot * THREADS * 2, r);
                if (h > hi) chi = peer_u16(ia);
                if (l < lo) clo = peer_u16(ia + THREADS * 2);
            }
            hi = fmaxf(hi, h);
            lo = fminf(lo, l);
        }
        if (mine) prm.y[m * N + n] = mam_epilogue(hi, lo, prm.ep, m, n, N);
        if constexpr (TRACK) {
            const long long nq = n - lane_n;   // the quarter-warp's first column
            __syncwarp();
            const int imax = first_in_chunk(prm.a, prm.w, m, nq, M, N, K, chi, hi, lane);
            const int imin = first_in_chunk(prm.a, prm.w, m, nq, M, N, K, clo, lo, lane);
            if (mine) {
                // an extreme that never left its start (products all NaN or on the wrong infinity) keeps k = 0, as
                // strict compares leave it (the any-shape kernel)
                prm.argmax[m * N + n] = hi > -INFINITY ? imax : 0;
                prm.argmin[m * N + n] = lo < INFINITY ? imin : 0;
            }
        }
    }
    __syncwarp();
    cluster_barrier();   // no CTA leaves while a peer still reads its shared memory
}

}  // namespace mamb200
