// qr_apply_cosets.cu -- compensated complex64 y = H psi for operators of
// several strings per x group (Jordan-Wigner sums, spin chains).
//
// The state is cut into tiles of 4,096 amplitudes; output tile q meets partner
// tile q ^ (x >> 12) for every x group (row semantics of
// qrusty/src/accel.rs:171-210).  A producer warp streams the partner tiles, two
// per ring slot, by 1-D TMA bulk copies; 16 consumer warps hold 8 rows per
// thread; the producer's idle warps build the next tile's factor tables (the
// tile's sign and parities applied to each sub-group's four factors), so the
// consumers pass no CTA barrier.
//
// Partner loads are shared.  A thread's 8 rows are a coset of the even-weight
// subsets of row bits 8-11 (t, with bit 8 flipped for odd popc(m), + 512 m), so
// x groups that differ by such a subset read the same 8 amplitudes: the four
// hops from an outer bit to bits 8-11 take one set of loads, and a
// Jordan-Wigner sum on n = 26 qubits 254 sets instead of 326.  With rows t +
// 512 m, m the bits 9-11, it would be 277.  Bit 8's pairing also leaves every
// hop that spans bits 8-11 without a sign pattern over m.  A hop's factor
// depends on m through one of the four bits: its two sub-groups F, G are one
// merged table entry (F + G, F - G), and a complete set of four such hops (a
// quad) runs without a dispatch.
//
// What bounds it (Jordan-Wigner n = 26): 254 sets of loads x 18 shared-memory
// wavefronts per warp (0.53 of the time), packed FMAs and parities at 0.5 of
// the issue slots, the latency of 45 blocks of two single-sub-group tiles, and
// beside them 57 GB of partner tiles per product from L2.  Per sub-group and
// tile (16 warps, n = 22 probes): lone 340 cycles, in a quad 360, by dispatch
// 730, against 446-538, 570-850 and the same before.
//
// Measured (us, before -> after; before: rows t + 512 m, partner tiles in
// pairs, the last warp out of a slot refilling it): Jordan-Wigner n = 26,
// 10,000 terms 9,340 -> 7,240; n = 20, 4,000 103 -> 84; chain n = 22 110 -> 93,
// n = 24 464 -> 390.  Relative error at n = 26 2.1e-7 -> 1.7e-7 (a fold every 8
// blocks instead of 16).
#include "qr_common.cuh"
#include "qr_device.cuh"

namespace qr {

namespace {

constexpr uint32_t kCThreads = 512, kCWarps = kCThreads / 32;
constexpr uint32_t kCBlockThreads = kCThreads + 128;  // and a producer warpgroup (one warp works)
constexpr uint32_t kCTileBytes = 4096 * 8, kCSlotBytes = 2 * kCTileBytes;
constexpr uint32_t kCMaxSlots = 3;
constexpr uint32_t kCFold = 8;  // blocks per compensated fold

constexpr bool odd3(int v) { return ((v ^ (v >> 1) ^ (v >> 2)) & 1) != 0; }

// The eight rows of thread t are t' + 512 m, t' = t with bit 8 flipped for odd
// popc(m); psi at those rows XOR a coset's offset.
__device__ __forceinline__ void coset_load(float2 (&p)[8], const unsigned char *sm, uint32_t base,
                                           uint32_t w) {
    const uint32_t b0 = base ^ (w & 0x8ff8u), b1 = b0 ^ 2048u;
#pragma unroll
    for (int m = 0; m < 8; ++m)
        p[m] = *reinterpret_cast<const float2 *>(sm + (odd3(m) ? b1 : b0) + ((uint32_t)m << 12));
}

// A sub-group's table entry and sign for this thread
template <bool TV>
__device__ __forceinline__ float2 coset_entry(uint32_t &sg, const float2 *tab, uint4 d, uint32_t g,
                                              uint32_t t) {
    if constexpr (TV) {
        const uint32_t u = ((uint32_t)__popc(t & d.z) & 1u) | (((uint32_t)__popc(t & d.w) & 1u) << 1);
        sg = (uint32_t)__popc(t & d.y) << 31;
        return tab[g * 4 + u];
    } else {
        sg = 0;
        return tab[g * 4];
    }
}
__device__ __forceinline__ float2 dup(float v, uint32_t sg) {
    const float f = __uint_as_float(__float_as_uint(v) ^ sg);
    return make_float2(f, f);
}

__device__ __forceinline__ float2 neg2(float2 v) { return __fmul2_rn(v, make_float2(-1.f, -1.f)); }

// A += re D p, B += im D p, y = A + i B; register index m meets p[m ^ XM] with
// the sign (-1)^popc(m & ZM)
template <int XM, int ZM>
__device__ __forceinline__ void coset_fma(float2 (&A)[8], float2 (&B)[8], const float2 (&p)[8],
                                          float2 fr, float2 fi) {
    float2 nr = fr, ni = fi;
    if constexpr (ZM != 0) {
        nr = neg2(fr);
        ni = neg2(fi);
    }
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        const bool n = odd3(m & ZM);
        A[m] = __ffma2_rn(n ? nr : fr, p[m ^ XM], A[m]);
        B[m] = __ffma2_rn(n ? ni : fi, p[m ^ XM], B[m]);
    }
}

// Two sub-groups F, G of one x group whose sign patterns are ZM and ZM ^ DL:
// one factor per register index, (-1)^popc(m & ZM) (F + (-1)^popc(m & DL) G),
// with p = F + G, m = F - G
template <int XM, int ZM, int DL>
__device__ __forceinline__ void coset_fma2(float2 (&A)[8], float2 (&B)[8], const float2 (&p)[8],
                                           float2 pr, float2 pi, float2 mr, float2 mi) {
    float2 npr = pr, npi = pi, nmr = mr, nmi = mi;
    if constexpr (ZM != 0) {
        npr = neg2(pr);
        npi = neg2(pi);
        nmr = neg2(mr);
        nmi = neg2(mi);
    }
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        const bool n = odd3(m & ZM), d = odd3(m & DL);
        A[m] = __ffma2_rn(n ? (d ? nmr : npr) : (d ? mr : pr), p[m ^ XM], A[m]);
        B[m] = __ffma2_rn(n ? (d ? nmi : npi) : (d ? mi : pi), p[m ^ XM], B[m]);
    }
}

// keys: XM | ZM << 3 (0 ... 63), or 64 + (F | ZM << 2) of a merged pair with
// XM = 0, 1, 2, 4 for F = 0 ... 3 and DL = 7, 1, 2, 4.  (Twelve bodies with the
// sign patterns at run time were 5 % slower on chains, equal on
// Jordan-Wigner sums.)
__device__ __forceinline__ void coset_dispatch(uint32_t key, float2 (&A)[8], float2 (&B)[8],
                                               const float2 (&p)[8], float4 T, uint32_t sg) {
    const float2 fr = dup(T.x, sg), fi = dup(T.y, sg), gr = dup(T.z, sg), gi = dup(T.w, sg);
#define QR_C1(k) \
    case k: coset_fma<(k & 7), (k >> 3)>(A, B, p, fr, fi); break;
#define QR_C8(k) QR_C1(k) QR_C1(k + 1) QR_C1(k + 2) QR_C1(k + 3) QR_C1(k + 4) QR_C1(k + 5) \
    QR_C1(k + 6) QR_C1(k + 7)
#define QR_F1(k)                                                                            \
    case 64 + k:                                                                            \
        coset_fma2<((k & 3) == 0 ? 0 : 1 << ((k & 3) - 1)), (k >> 2),                       \
                   ((k & 3) == 0 ? 7 : 1 << ((k & 3) - 1))>(A, B, p, fr, fi, gr, gi);       \
        break;
#define QR_F8(k) QR_F1(k) QR_F1(k + 1) QR_F1(k + 2) QR_F1(k + 3) QR_F1(k + 4) QR_F1(k + 5) \
    QR_F1(k + 6) QR_F1(k + 7)
    switch (key) {
        QR_C8(0) QR_C8(8) QR_C8(16) QR_C8(24) QR_C8(32) QR_C8(40) QR_C8(48) QR_C8(56)
        QR_F8(0) QR_F8(8) QR_F8(16) QR_F8(24)
        default: break;
    }
#undef QR_F8
#undef QR_F1
#undef QR_C8
#undef QR_C1
}

// Lone sub-groups [g, end) of key 0, one's partner loads and table entry in
// flight while the other's products are formed
template <bool TV>
__device__ __forceinline__ void coset_lone(float2 (&A)[8], float2 (&B)[8], const unsigned char *sm,
                                           uint32_t base, const float2 *tab, const uint4 *td,
                                           uint32_t g, uint32_t end, uint32_t t) {
#pragma unroll 2
    for (; g < end; ++g) {
        float2 p[8];
        uint32_t sg;
        const uint4 d = td[g];
        coset_load(p, sm, base, d.x);
        const float2 T = coset_entry<TV>(sg, tab, d, g, t);
        coset_fma<0, 0>(A, B, p, dup(T.x, sg), dup(T.y, sg));
    }
}

// Entry of a merged pair: (F + G, F - G), and the thread's sign
__device__ __forceinline__ float4 coset_entry2(uint32_t &sg, const float2 *tab, uint4 d, uint32_t g,
                                               uint32_t t) {
    const uint32_t u = ((uint32_t)__popc(t & d.z) & 1u) | (((uint32_t)__popc(t & d.w) & 1u) << 1);
    sg = (uint32_t)__popc(t & d.y) << 31;
    return reinterpret_cast<const float4 *>(tab + g * 4)[u];
}

template <int XM, int ZM, int DL>
__device__ __forceinline__ void coset_quarter(float2 (&A)[8], float2 (&B)[8], const float2 (&p)[8],
                                              const float2 *tab, uint4 d, uint32_t g, uint32_t t) {
    uint32_t sg;
    const float4 T = coset_entry2(sg, tab, d, g, t);
    coset_fma2<XM, ZM, DL>(A, B, p, dup(T.x, sg), dup(T.y, sg), dup(T.z, sg), dup(T.w, sg));
}

// A coset of four merged pairs, x = o + e_8 ... o + e_11 for one outer bit o,
// with the sign patterns of a Jordan-Wigner hop: one set of partner loads and
// no dispatch for eight sub-groups
__device__ __forceinline__ void coset_quad(float2 (&A)[8], float2 (&B)[8], const unsigned char *sm,
                                           uint32_t base, const float2 *tab, const uint4 *td,
                                           uint32_t g, uint32_t t) {
    float2 p[8];
    const uint4 d0 = td[g], d1 = td[g + 2];
    coset_load(p, sm, base, d0.x);
    coset_quarter<0, 0, 7>(A, B, p, tab, d0, g, t);
    const uint4 d2 = td[g + 4];
    coset_quarter<1, 7, 1>(A, B, p, tab, d1, g + 2, t);
    const uint4 d3 = td[g + 6];
    coset_quarter<2, 6, 2>(A, B, p, tab, d2, g + 4, t);
    coset_quarter<4, 4, 4>(A, B, p, tab, d3, g + 6, t);
}

// The block's two tiles with one uniform sub-group each, neither permuted
__device__ __forceinline__ void coset_cheap(float2 (&A)[8], float2 (&B)[8], const unsigned char *sm,
                                            uint32_t base, const float2 *tab, uint32_t g) {
    const float2 Ta = tab[g * 4], Tb = tab[g * 4 + 4];
    float2 p[8];
    coset_load(p, sm, base, 0);
    coset_fma<0, 0>(A, B, p, make_float2(Ta.x, Ta.x), make_float2(Ta.y, Ta.y));
    coset_load(p, sm, base, 0x8000u);
    coset_fma<0, 0>(A, B, p, make_float2(Tb.x, Tb.x), make_float2(Tb.y, Tb.y));
}

template <bool WIDE>
__device__ __forceinline__ uint32_t tile_parity(uint64_t q, uint64_t m) {
    if constexpr (WIDE) return (uint32_t)__popcll(q & m) & 1u;
    else return (uint32_t)__popc((uint32_t)q & (uint32_t)m) & 1u;
}

}  // namespace

template <bool WIDE>
__global__ void __launch_bounds__(kCBlockThreads, 1) apply_c64c_cosets(const ApplyArgs a,
                                                                       uint32_t slots,
                                                                       uint32_t ntab) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint64_t full[kCMaxSlots], empty[kCMaxSlots], tab_full[2], tab_empty[2];
    __shared__ uint32_t s_abort_;
    volatile uint32_t *s_abort = &s_abort_;
    uint4 *s_blk = reinterpret_cast<uint4 *>(smem_raw + (size_t)slots * kCSlotBytes);
    uint4 *s_td = s_blk + a.ncblk;
    float2 *s_tabs = reinterpret_cast<float2 *>(s_td + a.ncsub);
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    for (uint32_t i = t; i < a.ncblk; i += kCBlockThreads) s_blk[i] = a.cblk[i];
    for (uint32_t i = t; i < a.ncsub; i += kCBlockThreads) s_td[i] = a.ctdesc[i];
    if (t == 0) {
        for (uint32_t s = 0; s < slots; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kCWarps);
        }
        for (uint32_t k = 0; k < 2; ++k) {
            mbar_init(&tab_full[k], 3);
            mbar_init(&tab_empty[k], kCWarps);
        }
        s_abort_ = 0;
        mbar_fence_init();
    }
    __syncthreads();

    if (warp >= kCWarps) {
        // producer: the partner tiles of each block, a ring ahead
        asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
        if (warp == kCWarps && lane == 0) {
            uint32_t s = 0, round = 0, last_round[kCMaxSlots], issued = 0;
            bool ok = true;
            int64_t step = 0;  // test hook: ring step of CTA 0
            for (uint64_t item = blockIdx.x; item < a.nitems && ok; item += gridDim.x) {
                const uint64_t st = item / a.ntiles, q = item - st * a.ntiles;
                const float2 *src = static_cast<const float2 *>(a.psi) + st * a.N;
                for (uint32_t b = 0; b < a.ncblk; ++b, ++step) {
                    const uint4 bl = s_blk[b];
                    if (round > 0 && !mbar_wait_bounded(&empty[s], (round - 1) & 1u, a.wait_ns)) {
                        atomicExch(a.err, kErrMbarTimeout);
                        *s_abort = 1;
                    }
                    if (*s_abort != 0) {
                        ok = false;
                        break;
                    }
                    if (blockIdx.x != 0 || step != a.withhold) {
                        const bool two = bl.y != 0xffffffffu;
                        unsigned char *dst = smem_raw + (size_t)s * kCSlotBytes;
                        mbar_expect_tx(&full[s], two ? 2u * kCTileBytes : kCTileBytes);
                        bulk_g2s(dst, src + ((q ^ bl.x) << 12), kCTileBytes, &full[s]);
                        if (two)
                            bulk_g2s(dst + kCTileBytes, src + ((q ^ bl.y) << 12), kCTileBytes,
                                     &full[s]);
                        issued |= 1u << s;
                        last_round[s] = round;
                    }
                    if (++s == slots) {
                        s = 0;
                        ++round;
                    }
                }
            }
            // no copy is in flight when the CTA exits, also when the consumers'
            // wait expires after the last one was issued
            for (uint32_t k = 0; k < slots; ++k)
                if (issued >> k & 1u) mbar_wait_bounded(&full[k], last_round[k] & 1u, kWaitLimitNs);
        } else if (warp > kCWarps) {
            // the other three warps: factor tables of the next tile, in turn
            // into two buffers
            uint32_t buf = 0, round = 0;
            for (uint64_t item = blockIdx.x; item < a.nitems; item += gridDim.x) {
                const uint64_t q = item % a.ntiles;
                float2 *s_tab = s_tabs + (size_t)buf * a.ncsub * 4u;
                if (round > 0 && *s_abort == 0 &&
                    !mbar_wait_bounded(&tab_empty[buf], (round - 1u) & 1u, a.wait_ns)) {
                    atomicExch(a.err, kErrMbarTimeout);
                    *s_abort = 1;
                }
                if (*s_abort != 0) break;
                for (uint32_t g = t - (kCThreads + 32u); g < a.ncsub; g += 96u) {
                    const TileDataC64 &d = a.ctdata[g];
                    const uint32_t uq =
                        tile_parity<WIDE>(q, d.b0h) | (tile_parity<WIDE>(q, d.b1h) << 1);
                    const uint32_t sq = tile_parity<WIDE>(q, d.z0h);
                    const uint32_t role = (uint32_t)d.role;
                    if (role == 0) {
#pragma unroll
                        for (uint32_t u = 0; u < 4; ++u) {
                            const float2 v = d.T[u ^ uq];
                            s_tab[g * 4 + u] = make_float2(flip(v.x, sq), flip(v.y, sq));
                        }
                    } else if (role != kMergedSecond) {
                        // the two slots of a merged pair hold (F + G, F - G): one
                        // common basis, or (kMergedSign) u = parities against one
                        // basis vector and against the difference of the signs
                        const TileDataC64 &e = a.ctdata[g + 1];
                        const uint32_t ue =
                            tile_parity<WIDE>(q, e.b0h) | (tile_parity<WIDE>(q, e.b1h) << 1);
                        const uint32_t se = tile_parity<WIDE>(q, e.z0h);
                        const uint32_t low = role == kMergedSign ? 1u : 3u;
#pragma unroll
                        for (uint32_t u = 0; u < 4; ++u) {
                            const float2 v = d.T[(u ^ uq) & low], w = e.T[(u ^ ue) & low];
                            const uint32_t sw = role == kMergedSign ? se ^ (u >> 1) : se;
                            const float2 f = make_float2(flip(v.x, sq), flip(v.y, sq));
                            const float2 h = make_float2(flip(w.x, sw), flip(w.y, sw));
                            const float2 pl = __fadd2_rn(f, h), mi = sub2_rn(f, h);
                            reinterpret_cast<float4 *>(s_tab + g * 4)[u] =
                                make_float4(pl.x, pl.y, mi.x, mi.y);
                        }
                    }
                }
                __syncwarp();
                if (lane == 0)
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(
                                     saddr(&tab_full[buf]))
                                 : "memory");
                if (++buf == ntab) {
                    buf = 0;
                    ++round;
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
        float2 A[8], B[8], hi[8], p[8];
        uint32_t s = 0, par = 0, buf = 0, tpar = 0;
        const uint32_t t8 = t << 3;
        for (uint64_t item = blockIdx.x; item < a.nitems; item += gridDim.x) {
            const uint64_t st = item / a.ntiles, q = item - st * a.ntiles;
#pragma unroll
            for (int m = 0; m < 8; ++m) A[m] = B[m] = hi[m] = make_float2(0.f, 0.f);
            // the tile's factor tables, built while the last tile was computed
            const float2 *s_tab = s_tabs + (size_t)buf * a.ncsub * 4u;
            if (*s_abort == 0 && !mbar_wait_bounded(&tab_full[buf], tpar, a.wait_ns) && lane == 0) {
                atomicExch(a.err, kErrMbarTimeout);
                *s_abort = 1;
            }
            for (uint32_t b = 0; b < a.ncblk; ++b) {
                // an expired wait sets the abort flag; from then on every
                // warp skips waits and work but still passes every barrier
                bool skip = false;
                if (!__all_sync(0xffffffffu, mbar_try_wait(&full[s], par))) {
                    skip = *s_abort != 0;
                    if (!skip && !mbar_wait_bounded(&full[s], par, a.wait_ns)) {
                        if (lane == 0) {
                            atomicExch(a.err, kErrMbarTimeout);
                            *s_abort = 1;
                        }
                        skip = true;
                    }
                    skip = __any_sync(0xffffffffu, skip);
                }
                if (!skip) {
                    const uint4 bl = s_blk[b];
                    const uint32_t base = s * kCSlotBytes + t8;
                    uint32_t g = bl.z & 1023u;
                    if (bl.z >> 31) {  // the diagonal, on tile 0 of the block
                        const float2 *dg = static_cast<const float2 *>(a.diag) + (q << 12);
                        coset_load(p, smem_raw, base, 0);
#pragma unroll
                        for (int m = 0; m < 8; ++m) {
                            const float2 d = dg[(t ^ (odd3(m) ? 256u : 0u)) + 512u * m];
                            A[m] = __ffma2_rn(make_float2(d.x, d.x), p[m], A[m]);
                            B[m] = __ffma2_rn(make_float2(d.y, d.y), p[m], B[m]);
                        }
                    }
                    // lone sub-groups of key 0: the factor the same for every
                    // thread, then by thread; hops into the coset's bits
                    if ((bl.z >> 30) & 1u) {
                        coset_cheap(A, B, smem_raw, base, s_tab, g);
                    } else {
                        uint32_t end = g + ((bl.z >> 10) & 1023u);
                        coset_lone<false>(A, B, smem_raw, base, s_tab, s_td, g, end, t);
                        g = end;
                        end = g + (bl.w & 1023u);
                        coset_lone<true>(A, B, smem_raw, base, s_tab, s_td, g, end, t);
                        g = end;
                        end = g + 8u * ((bl.w >> 10) & 63u);
                        for (; g < end; g += 8)
                            coset_quad(A, B, smem_raw, base, s_tab, s_td, g, t);
                        // the others, sharing partner loads within a coset
                        end = g + (bl.w >> 16);
                        while (g < end) {
                            const uint4 d = s_td[g];
                            const uint32_t key = d.x >> 17 & 127u;
                            if (d.x & 0x10000u) coset_load(p, smem_raw, base, d.x);
                            uint32_t sg;
                            float4 T;
                            if (d.x >> 24) {  // merged pair
                                T = coset_entry2(sg, s_tab, d, g, t);
                            } else {
                                const float2 F = coset_entry<true>(sg, s_tab, d, g, t);
                                T = make_float4(F.x, F.y, F.x, F.y);
                            }
                            g += key >= 64u ? 2u : 1u;
                            coset_dispatch(key, A, B, p, T, sg);
                        }
                    }
                }
                // y = A + iB is folded into hi with an error-free two-sum, whose
                // error opens the next window (Kahan)
                if (b + 1 == a.ncblk || (b % kCFold) == kCFold - 1) {
#pragma unroll
                    for (int m = 0; m < 8; ++m) {
                        const float2 yv =
                            make_float2(__fsub_rn(A[m].x, B[m].y), __fadd_rn(A[m].y, B[m].x));
                        A[m] = two_sum_carry2(hi[m], yv);
                        B[m] = make_float2(0.f, 0.f);
                    }
                }
                __syncwarp();
                if (lane == 0)
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(saddr(&empty[s]))
                                 : "memory");
                if (++s == slots) {
                    s = 0;
                    par ^= 1u;
                }
            }
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(
                                 saddr(&tab_empty[buf]))
                             : "memory");
            if (++buf == ntab) {
                buf = 0;
                tpar ^= 1u;
            }
            float2 *yo = static_cast<float2 *>(a.y) + st * a.N + (q << 12);
            const float2 *vo = a.v ? static_cast<const float2 *>(a.v) + st * a.N + (q << 12) : nullptr;
#pragma unroll
            for (int m = 0; m < 8; ++m) {
                const uint32_t rl = (t ^ (odd3(m) ? 256u : 0u)) + 512u * m;
                float2 o = make_float2(__fadd_rn(hi[m].x, A[m].x), __fadd_rn(hi[m].y, A[m].y));
                if (vo)  // fused y = alpha (H psi) + beta v, in FP32
                    o = cx_axpby((float)a.ar, (float)a.ai, o, (float)a.br, (float)a.bi, vo[rl]);
                yo[rl] = o;
            }
        }
    }
    __syncthreads();
}

size_t coset_smem_bytes(uint32_t nsub, uint32_t nblk, uint32_t slots, uint32_t ntab) {
    return (size_t)slots * kCSlotBytes + (size_t)nblk * 16u + (size_t)nsub * (16u + ntab * 32u);
}

// Three ring slots and two tables where they fit (Jordan-Wigner n = 26: 431
// sub-groups, 232 KB), else one table (built between two tiles), else two slots.
cudaError_t launch_c64c_cosets(const ApplyArgs &a, int nsm, cudaStream_t st) {
    uint32_t slots = 3, ntab = 2;
    if (coset_smem_bytes(a.ncsub, a.ncblk, 3, 2) > kCosetSmem) ntab = 1;
    if (coset_smem_bytes(a.ncsub, a.ncblk, 3, 1) > kCosetSmem) {
        slots = 2;
        ntab = coset_smem_bytes(a.ncsub, a.ncblk, 2, 2) > kCosetSmem ? 1 : 2;
    }
    const size_t smem = coset_smem_bytes(a.ncsub, a.ncblk, slots, ntab);
    if (smem > kCosetSmem) return cudaErrorInvalidValue;
    auto kern = (a.n > 32 || a.wide) ? apply_c64c_cosets<true> : apply_c64c_cosets<false>;
    const cudaError_t e = ensure_dyn_smem(reinterpret_cast<const void *>(kern), smem);
    if (e != cudaSuccess) return e;
    const uint64_t grid = a.nitems < (uint64_t)nsm ? a.nitems : (uint64_t)nsm;
    if (grid == 0) return cudaSuccess;
    kern<<<(unsigned)grid, kCBlockThreads, smem, st>>>(a, slots, ntab);
    count_launch();
    return cudaGetLastError();
}

}  // namespace qr
