// qr_apply_strings.cu -- compensated complex64 y = H psi for operators whose
// x groups hold about one Pauli string each (random-letter sums).
//
// Row r of the product sums s_k(r) c'_k psi[r ^ x_k] over the merged strings k,
// s_k(r) = (-1)^popc(r & z_k) (qrusty/src/accel.rs:171-210).  The state is cut
// into tiles of 4,096 amplitudes; a block is one or two partner tiles (tile ^
// (x >> 12)) with the strings that read them, and both travel through a
// shared-memory ring by 1-D TMA bulk copies: the tiles of psi, and 16 bytes
// per string {partner offset | sign bits, z, re, im}.  Nothing about a string
// depends on the output tile but one popc, so there is no per-tile table and
// no CTA barrier.  A producer warp fills the ring; 16 consumer warps hold 8
// rows per thread (bits 0, 10 and 11 of the row are register bits, so one
// 16-byte shared load brings two of a string's 8 partners) and take the
// strings in turn: 4 loads, 8 sign XORs, 16 FMAs, since a string's
// coefficient is real or imaginary (one with both parts takes 32).  At the
// end of a block, once the window holds 24 strings (278 at most, where blocks
// are full), the sums are folded into a compensated pair (Kahan: the error opens
// the next window).
//
// What bounds it: shared-memory wavefronts, 18 per warp and string (16 of
// them partner amplitudes), 91 % busy (ncu, n = 18, 2,000 strings).  Hence
// 16-byte entries with the signs as bits (32-byte ones with float signs were
// 8 % slower), loaded once per string with its partners prefetched one string
// ahead, and no dispatch over sign patterns: the table kernel's runs of equal
// pattern hold one or two strings of such operators, and its jump per run and
// second FMA per amplitude cost more than the XORs.  512 x 112 + 128 x 24
// registers (setmaxnreg) of the 640 x 96 launched.
//
// Few tiles: below 2^19 amplitudes per state a tile's blocks are split over a
// cluster of up to 8 CTAs, whose compensated sums meet through distributed
// shared memory in rank order.
//
// Measured (us, before -> after; before: the per-tile table kernels): n = 16,
// 1,000 strings, 3 states 212 -> 88; n = 18, 2,000 463 -> 186; n = 20, 2,000 1,231
// -> 741; n = 22, 500 1,770 -> 903.  Relative error of a random-letter product
// 1.0-1.5e-7 with windows of few strings (was 1.3-3.0), 2.4-2.9e-7 with full
// blocks (n = 14, 9,000 strings, n = 19, 10,000; was 4.2-8.0).
#include <map>
#include <mutex>
#include <utility>

#include "qr_common.cuh"
#include "qr_device.cuh"

namespace qr {

namespace {

constexpr uint32_t kSWarps = kStrThreads / 32;          // consumer warps
constexpr uint32_t kSBlockThreads = kStrThreads + 128;  // and a producer warpgroup (one warp works)
constexpr uint32_t kSTileBytes = 4096 * 8;
constexpr uint32_t kSEntBytes = (kStrEntCap + 1) * 16;  // header and entries of a block
constexpr uint32_t kSMaxStages = 4;
constexpr float kFltMax = 3.402823466e38f;
constexpr uint32_t kSFold = 24;  // strings per compensated fold, at least (23 + kStrEntCap at most)

// partner amplitudes of one string: p[j] holds register indices 2 j, 2 j + 1
__device__ __forceinline__ void str_load(float4 (&p)[4], const unsigned char *sm, uint32_t base,
                                         uint32_t w) {
    const uint32_t off = base ^ (w & 0xfff0u);
#pragma unroll
    for (int j = 0; j < 4; ++j)
        p[j] = *reinterpret_cast<const float4 *>(sm + (off ^ ((uint32_t)j << 13)));
}

// y += f p (IM: y += i f p) with f[m] the signed factor of register index m;
// SW: the string's x swaps the two amplitudes of a pair
template <bool IM, bool SW>
__device__ __forceinline__ void str_fma(float2 (&y)[8], const float4 (&p)[4], const float (&f)[8]) {
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        const float4 v = p[m >> 1];
        const float pr = ((m & 1) != 0) != SW ? v.z : v.x, pi = ((m & 1) != 0) != SW ? v.w : v.y;
        if (IM) {
            y[m].x = fmaf(-f[m], pi, y[m].x);
            y[m].y = fmaf(f[m], pr, y[m].y);
        } else {
            y[m].x = fmaf(f[m], pr, y[m].x);
            y[m].y = fmaf(f[m], pi, y[m].y);
        }
    }
}

template <bool WIDE>
__device__ __forceinline__ void str_mac(float2 (&y)[8], const float4 (&p)[4], uint4 e, uint32_t r0,
                                        uint32_t rhi) {
    uint32_t s = (uint32_t)__popc(r0 & e.y);
    if constexpr (WIDE) s += (uint32_t)__popc(rhi & e.x);
    const bool im = __uint_as_float(e.w) != 0.f;
    // + 2^31 flips the sign bit, so an odd parity negates
    uint32_t g[8];
    g[0] = (im ? e.w : e.z) + (s << 31);
    const uint32_t M = 0x80000000u, k1 = e.x << 15, k2 = e.x << 14, k4 = e.x << 13;
    g[1] = g[0] ^ (k1 & M);
    g[2] = g[0] ^ (k2 & M);
    g[3] = g[1] ^ (k2 & M);
#pragma unroll
    for (int m = 0; m < 4; ++m) g[m + 4] = g[m] ^ (k4 & M);
    float f[8];
#pragma unroll
    for (int m = 0; m < 8; ++m) f[m] = __uint_as_float(g[m]);
    const bool sw = (e.x & 1u) != 0;
    if (!im) {
        if (sw) str_fma<false, true>(y, p, f);
        else str_fma<false, false>(y, p, f);
        return;
    }
    if (sw) str_fma<true, true>(y, p, f);
    else str_fma<true, false>(y, p, f);
    if (__uint_as_float(e.z) != 0.f) {  // real and imaginary part
#pragma unroll
        for (int m = 0; m < 8; ++m) f[m] = __uint_as_float(__float_as_uint(f[m]) ^ e.w ^ e.z);
        if (sw) str_fma<false, true>(y, p, f);
        else str_fma<false, false>(y, p, f);
    }
}

__device__ __forceinline__ bool finite_f(float v) { return fabsf(v) <= kFltMax; }

// Of the rows `left` (a mask of register indices; row: the first one's), those
// with an infinite or NaN partner in blocks [b0, b1).  A string's zero part forms
// no product, so such a row may have one finite part where 0 * inf, with every
// product formed, makes both NaN.  Asked at each fold of its blocks, so that the
// rows of a state full of them take no longer than the bounded waits allow.
__device__ __forceinline__ uint32_t str_nonfinite(uint32_t left, const uint4 *sblk, uint32_t b0,
                                                 uint32_t b1, const uint4 *ent, const float2 *psi,
                                                 uint64_t row) {
    uint32_t bad = 0;
    for (uint32_t b = b0; b < b1 && left != 0; ++b) {
        const uint4 bl = sblk[b];
        for (uint32_t i = 1; i <= bl.w && left != 0; ++i) {
            const uint32_t e = ent[bl.z + i].x;
            const uint64_t x = (uint64_t)((e >> 15) & 1u ? bl.y : bl.x) << 12 | (e & 1u) |
                               ((e >> 4) & 511u) << 1 | ((e >> 13) & 3u) << 10;
            for (uint32_t r = left; r != 0; r &= r - 1u) {
                const uint32_t m = (uint32_t)__ffs((int)r) - 1u;
                const float2 p = psi[row ^ x ^ ((m & 1u) | (m >> 1) << 10)];
                if (!(finite_f(p.x) && finite_f(p.y))) bad |= 1u << m;
            }
            left &= ~bad;
        }
    }
    return bad;
}

// The same as a call: in line it costs the single kernel 2 %; the batch kernel
// takes it in line, a call costs that one 8 %.
__device__ __noinline__ uint32_t str_nonfinite_call(uint32_t left, const uint4 *sblk, uint32_t b0,
                                                   uint32_t b1, const uint4 *ent,
                                                   const float2 *psi, uint64_t row) {
    return str_nonfinite(left, sblk, b0, b1, ent, psi, row);
}

// Fold the window's sums y into hi; the error opens the next window.  nonfinite:
// asks str_nonfinite for the window's blocks.
template <typename F>
__device__ __forceinline__ void str_fold(float2 (&y)[8], float2 (&hi)[8], F &&nonfinite) {
    // 0 * y: NaN once a part is infinite or NaN
    const float2 z2 = make_float2(0.f, 0.f);
    float2 q[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) q[m] = __ffma2_rn(y[m], z2, __fmul2_rn(y[m + 4], z2));
    q[0] = __fadd2_rn(__fadd2_rn(q[0], q[1]), __fadd2_rn(q[2], q[3]));
    if (__any_sync(0xffffffffu, q[0].x + q[0].y != 0.f)) {
        uint32_t left = 0;
#pragma unroll
        for (int m = 0; m < 8; ++m)
            left |= (finite_f(y[m].x) != finite_f(y[m].y) ? 1u : 0u) << m;
        const uint32_t bad = nonfinite(left);
        const float nan = __uint_as_float(0x7fc00000u);
#pragma unroll
        for (int m = 0; m < 8; ++m)
            if (bad >> m & 1u) y[m] = make_float2(nan, nan);
    }
#pragma unroll
    for (int m = 0; m < 8; ++m) y[m] = two_sum_carry2(hi[m], y[m]);
}

// A row's value: an infinite sum is NaN (its compensation is)
__device__ __forceinline__ float2 str_value(float2 h, float2 l) {
    const float nan = __uint_as_float(0x7fc00000u);
    const float2 o = make_float2(__fadd_rn(h.x, l.x), __fadd_rn(h.y, l.y));
    return make_float2(finite_f(o.x) ? o.x : nan, finite_f(o.y) ? o.y : nan);
}

// One block of the ring: the diagonal where it is flagged, then the strings in
// turn, one's partner loads in flight while the other's products are formed.
// Returns their number.
template <bool WIDE>
__device__ __forceinline__ uint32_t str_block(float2 (&y)[8], const unsigned char *sm,
                                              const uint4 *E, uint32_t base, const float4 *dg,
                                              uint32_t t, uint32_t r0, uint32_t rhi) {
    float4 pa[4], pb[4];
    const uint2 head = *reinterpret_cast<const uint2 *>(E);
    const uint32_t ne = head.x;
    if (head.y != 0) {
        str_load(pa, sm, base, 0);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 d = dg[t + 512u * (uint32_t)j], p = pa[j];
            float2 &u = y[2 * j], &v = y[2 * j + 1];
            u.x = fmaf(d.x, p.x, fmaf(-d.y, p.y, u.x));
            u.y = fmaf(d.x, p.y, fmaf(d.y, p.x, u.y));
            v.x = fmaf(d.z, p.z, fmaf(-d.w, p.w, v.x));
            v.y = fmaf(d.z, p.w, fmaf(d.w, p.z, v.y));
        }
    }
    uint32_t i = 1;
    uint4 ea = E[1], eb;
    if (ne > 0) str_load(pa, sm, base, ea.x);
    for (; i + 1 < ne; i += 2) {
        eb = E[i + 1];
        str_load(pb, sm, base, eb.x);
        str_mac<WIDE>(y, pa, ea, r0, rhi);
        ea = E[i + 2];
        str_load(pa, sm, base, ea.x);
        str_mac<WIDE>(y, pb, eb, r0, rhi);
    }
    if (i < ne) {
        eb = E[i + 1];
        str_load(pb, sm, base, eb.x);
        str_mac<WIDE>(y, pa, ea, r0, rhi);
        str_mac<WIDE>(y, pb, eb, r0, rhi);
    } else if (i == ne) {
        str_mac<WIDE>(y, pa, ea, r0, rhi);
    }
    return ne;
}

__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void arrive_cluster(uint32_t addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
__device__ __forceinline__ void arrive_local(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(saddr(bar)) : "memory");
}
__device__ __forceinline__ bool try_wait_cluster(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(saddr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool wait_cluster(uint64_t *bar, uint32_t parity, uint64_t limit_ns) {
    if (try_wait_cluster(bar, parity)) return true;
    const uint64_t t0 = gtimer_ns();
    while (!try_wait_cluster(bar, parity))
        if (gtimer_ns() - t0 > limit_ns) return false;
    return true;
}
__device__ __forceinline__ float4 ld_cluster(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(addr)
                 : "memory");
    return v;
}

}  // namespace

template <bool WIDE>
__global__ void __launch_bounds__(kSBlockThreads, 1) apply_c64c_strings(const ApplyArgs a,
                                                                        uint32_t stages,
                                                                        uint32_t ks, uint32_t tpb) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint64_t full[kSMaxStages], empty[kSMaxStages], xfull, xfree;
    __shared__ uint32_t s_abort_;
    volatile uint32_t *s_abort = &s_abort_;
    const uint32_t slot = tpb * kSTileBytes;  // partner tiles of a block
    unsigned char *s_ent = smem_raw + (size_t)stages * slot;
    float4 *xbuf = reinterpret_cast<float4 *>(s_ent + (size_t)stages * kSEntBytes);
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint32_t rank = ks > 1 ? blockIdx.x % ks : 0u;
    const uint32_t cl = blockIdx.x / ks, ncl = gridDim.x / ks;
    const uint32_t b0 = a.part[rank], b1 = a.part[rank + 1];
    if (t == 0) {
        for (uint32_t s = 0; s < stages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kSWarps);
        }
        mbar_init(&xfull, ks * kSWarps);
        mbar_init(&xfree, ks * kSWarps);
        s_abort_ = 0;
        mbar_fence_init();
    }
    __syncthreads();
    if (ks > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }

    if (warp >= kSWarps) {
        // producer: partner tile and entry list of each block, a ring ahead
        asm volatile("setmaxnreg.dec.sync.aligned.u32 24;");
        if (warp == kSWarps && lane == 0) {
            uint32_t s = 0, round = 0, last_round[kSMaxStages];
            uint32_t issued = 0;  // stages with a copy
            bool ok = true;
            uint64_t step = 0;    // test hook: steps of cluster 0, all ranks, in block order
            for (uint64_t item = cl; item < a.nitems && ok; item += ncl, step += a.nsblk) {
                const uint64_t st = item / a.ntiles, q = item - st * a.ntiles;
                const float2 *src = static_cast<const float2 *>(a.psi) + st * a.N;
                uint4 nx = b0 < b1 ? a.sblk[b0] : make_uint4(0u, 0u, 0u, 0u);
                for (uint32_t b = b0; b < b1; ++b) {
                    const uint4 bl = nx;
                    if (b + 1 < b1) nx = a.sblk[b + 1];
                    if (round > 0 && !mbar_wait_bounded(&empty[s], (round - 1) & 1u, a.wait_ns)) {
                        atomicExch(a.err, kErrMbarTimeout);
                        *s_abort = 1;
                    }
                    if (*s_abort != 0) {
                        ok = false;
                        break;
                    }
                    if (cl != 0 || (int64_t)(step + b) != a.withhold) {
                        const uint32_t eb = (bl.w + 1u) * 16u;
                        const bool two = bl.y != 0xffffffffu;
                        mbar_expect_tx(&full[s], (two ? 2u : 1u) * kSTileBytes + eb);
                        unsigned char *dst = smem_raw + (size_t)s * slot;
                        bulk_g2s(dst, src + ((q ^ bl.x) << 12), kSTileBytes, &full[s]);
                        if (two)
                            bulk_g2s(dst + kSTileBytes, src + ((q ^ bl.y) << 12), kSTileBytes,
                                     &full[s]);
                        bulk_g2s(s_ent + (size_t)s * kSEntBytes, a.ent + bl.z, eb,
                                 &full[s]);
                        issued |= 1u << s;
                        last_round[s] = round;
                    }
                    if (++s == stages) {
                        s = 0;
                        ++round;
                    }
                }
            }
            // no copy is in flight when the CTA exits, also when the consumers'
            // wait expires after the last one was issued
            for (uint32_t k = 0; k < stages; ++k)
                if (issued >> k & 1u) mbar_wait_bounded(&full[k], last_round[k] & 1u, kWaitLimitNs);
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
        float2 y[8], hi[8];
        uint32_t s = 0, par = 0, it = 0;
        const uint32_t t16 = t << 4;
        for (uint64_t item = cl; item < a.nitems; item += ncl, ++it) {
            const uint64_t st = item / a.ntiles, q = item - st * a.ntiles;
            const uint32_t r0 = (uint32_t)(q << 12) | t << 1;
            const uint32_t rhi = WIDE ? (uint32_t)(q >> 20) << 24 : 0u;
            uint32_t win = 0, wb = b0;  // the window's strings and first block
            auto fold = [&](uint32_t end) {
                str_fold(y, hi, [&](uint32_t left) {
                    return str_nonfinite_call(left, a.sblk, wb, end, a.ent,
                                         static_cast<const float2 *>(a.psi) + st * a.N,
                                         (q << 12) | (t << 1));
                });
            };
#pragma unroll
            for (int m = 0; m < 8; ++m) y[m] = hi[m] = make_float2(0.f, 0.f);
            for (uint32_t b = b0; b < b1; ++b) {
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
                    const uint4 *E = reinterpret_cast<const uint4 *>(s_ent + (size_t)s * kSEntBytes);
                    win += str_block<WIDE>(y, smem_raw, E, s * slot + t16,
                                           static_cast<const float4 *>(a.diag) + (q << 11), t, r0,
                                           rhi);
                    if (win >= kSFold) {
                        fold(b + 1);
                        win = 0;
                        wb = b + 1;
                    }
                }
                __syncwarp();
                if (lane == 0) arrive_local(&empty[s]);
                if (++s == stages) {
                    s = 0;
                    par ^= 1u;
                }
            }
            fold(b1);

            float2 *yo = static_cast<float2 *>(a.y) + st * a.N + (q << 12);
            const float2 *vo = a.v ? static_cast<const float2 *>(a.v) + st * a.N + (q << 12) : nullptr;
            auto finish = [&](uint32_t rl, float2 o) {
                if (vo)  // fused y = alpha (H psi) + beta v, in FP32
                    o = cx_axpby((float)a.ar, (float)a.ai, o, (float)a.br, (float)a.bi, vo[rl]);
                yo[rl] = o;
            };
            auto row_of = [&](uint32_t m) { return 2u * t + (m & 1u) + 1024u * (m >> 1); };
            if (ks == 1) {
#pragma unroll
                for (int m = 0; m < 8; ++m) finish(row_of((uint32_t)m), str_value(hi[m], y[m]));
            } else {
                // the ranks' sums meet in shared memory: rank r adds rows
                // of register index m = r, r + ks, ... of every rank, in rank order
                auto wait_x = [&](uint64_t *bar, uint32_t parity) {
                    bool bad = *s_abort != 0;
                    if (!bad && !wait_cluster(bar, parity, a.wait_ns)) {
                        if (lane == 0) {
                            atomicExch(a.err, kErrMbarTimeout);
                            *s_abort = 1;
                        }
                        bad = true;
                    }
                    return __any_sync(0xffffffffu, bad);
                };
                bool bad = it > 0 && wait_x(&xfree, (it - 1) & 1u);
#pragma unroll
                for (int m = 0; m < 8; ++m)
                    xbuf[m * 512 + t] = make_float4(hi[m].x, hi[m].y, y[m].x, y[m].y);
                __syncwarp();
                if (lane < ks) {
                    asm volatile("fence.acq_rel.cluster;" ::: "memory");
                    arrive_cluster(mapa(saddr(&xfull), lane));
                }
                bad = wait_x(&xfull, it & 1u) || bad;
                if (!bad) {
                    for (uint32_t m = rank; m < 8; m += ks) {
                        const uint32_t at = saddr(xbuf + m * 512 + t);
                        float4 v = ld_cluster(mapa(at, 0));
                        float2 h = make_float2(v.x, v.y), l = make_float2(v.z, v.w);
                        for (uint32_t r = 1; r < ks; ++r) {
                            v = ld_cluster(mapa(at, r));
                            const float2 e = two_sum_carry2(h, make_float2(v.x, v.y));
                            l = __fadd2_rn(l, __fadd2_rn(e, make_float2(v.z, v.w)));
                        }
                        finish(row_of(m), str_value(h, l));
                    }
                }
                __syncwarp();
                if (lane < ks) {
                    asm volatile("fence.acq_rel.cluster;" ::: "memory");
                    arrive_cluster(mapa(saddr(&xfree), lane));
                }
            }
        }
    }
    __syncthreads();
    if (ks > 1) {  // a peer may still read this CTA's sums or arrive on its barriers
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

// An expired wait of the batch: its own error word and, as which items are lost
// is not known, that of every operator in the work list
__device__ __forceinline__ void str_batch_late(const StrBatchArgs &a) {
    atomicExch(a.err, kErrMbarTimeout);
    for (uint32_t i = 0; i < a.nops; ++i)
        if (a.ops[i].err != nullptr) atomicExch(a.ops[i].err, kErrMbarTimeout);
}

// Many operators, states and tiles in one launch: the same ring and inner loop,
// a CTA per SM taking the next (operator, state, tile) item, largest first,
// from a counter as it gets free.  What an operator's own launch leaves idle
// is the SMs its tiles do not cover (four states of 2^17 amplitudes are 128
// tiles on 152 SMs; smaller ones are split over clusters, with a round of
// exchange per tile) and its start and end; the ring runs on from item to
// item.  24 operators of 10 to 17 qubits, 4 states: 1,335 us (1,428 with the
// small ones in the table kernel and a launch per large one).  A string and
// tile cost 390 clocks of an SM, as in a full launch of one operator, of which
// the shared-memory wavefronts are 288.  A block's item travels with it: {operator, state, tile, first | last
// << 1 | end << 2}.
__global__ void __launch_bounds__(kSBlockThreads, 1) apply_c64c_strings_batch(const StrBatchArgs a) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint64_t full[kSMaxStages], empty[kSMaxStages];
    __shared__ uint4 s_meta[kSMaxStages];
    __shared__ uint32_t s_abort_;
    volatile uint32_t *s_abort = &s_abort_;
    constexpr uint32_t kEnd = 4u;
    unsigned char *s_ent = smem_raw + (size_t)kSMaxStages * kSTileBytes;
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t == 0) {
        for (uint32_t s = 0; s < kSMaxStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kSWarps);
        }
        s_abort_ = 0;
        mbar_fence_init();
    }
    __syncthreads();

    if (warp >= kSWarps) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 24;");
        if (warp == kSWarps && lane == 0) {
            uint32_t s = 0, round = 0, issued = 0, last_round[kSMaxStages];
            bool ok = true;
            // the stage is free, or the kernel gives up
            auto take = [&]() {
                if (round > 0 && !mbar_wait_bounded(&empty[s], (round - 1) & 1u, a.wait_ns)) {
                    str_batch_late(a);
                    *s_abort = 1;
                }
                ok = *s_abort == 0;
                return ok;
            };
            auto next = [&]() {
                if (++s == kSMaxStages) {
                    s = 0;
                    ++round;
                }
            };
            uint32_t i = atomicAdd(a.counter, 1u);
            int64_t step = blockIdx.x == 0 ? 0 : -1;  // test hook: ring step of CTA 0
            while (ok && i < a.nitems) {
                const uint32_t ahead = atomicAdd(a.counter, 1u);
                const BatchItem it = a.items[i];
                const StrOp op = a.ops[it.op];
                const float2 *src = a.psi[it.op] + (uint64_t)it.state * op.N;
                for (uint32_t b = 0; b < op.nblk && take(); ++b, next()) {
                    if (step >= 0 && step++ == a.withhold) continue;
                    const uint4 bl = op.sblk[b];
                    const uint32_t eb = (bl.w + 1u) * 16u;
                    s_meta[s] = make_uint4(it.op, it.state, it.tile,
                                           (b == 0 ? 1u : 0u) | (b + 1 == op.nblk ? 2u : 0u));
                    mbar_expect_tx(&full[s], kSTileBytes + eb);
                    bulk_g2s(smem_raw + (size_t)s * kSTileBytes,
                             src + ((uint64_t)(it.tile ^ bl.x) << 12), kSTileBytes, &full[s]);
                    bulk_g2s(s_ent + (size_t)s * kSEntBytes, op.ent + bl.z, eb, &full[s]);
                    issued |= 1u << s;
                    last_round[s] = round;
                }
                i = ahead;
            }
            if (ok && take()) {
                s_meta[s] = make_uint4(0u, 0u, 0u, kEnd);
                arrive_local(&full[s]);
                issued |= 1u << s;  // the stage's last phase is this one
                last_round[s] = round;
            }
            // no copy is in flight when the CTA exits, also when the consumers'
            // wait expires after the last one was issued
            for (uint32_t k = 0; k < kSMaxStages; ++k)
                if (issued >> k & 1u) mbar_wait_bounded(&full[k], last_round[k] & 1u, kWaitLimitNs);
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
        float2 y[8], hi[8];
        uint32_t s = 0, par = 0, win = 0;
        uint32_t b = 0, wb = 0;  // the item's block, the window's first
        for (;;) {
            // an expired wait sets the abort flag; every warp then leaves
            bool skip = false;
            if (!__all_sync(0xffffffffu, mbar_try_wait(&full[s], par))) {
                skip = *s_abort != 0;
                if (!skip && !mbar_wait_bounded(&full[s], par, a.wait_ns)) {
                    if (lane == 0) {
                        str_batch_late(a);
                        *s_abort = 1;
                    }
                    skip = true;
                }
                skip = __any_sync(0xffffffffu, skip);
            }
            if (skip) break;
            const uint4 me = s_meta[s];
            if (me.w & kEnd) break;
            if (me.w & 1u) {
                win = b = wb = 0;
#pragma unroll
                for (int m = 0; m < 8; ++m) y[m] = hi[m] = make_float2(0.f, 0.f);
            }
            win += str_block<false>(
                y, smem_raw, reinterpret_cast<const uint4 *>(s_ent + (size_t)s * kSEntBytes),
                s * kSTileBytes + (t << 4),
                reinterpret_cast<const float4 *>(a.ops[me.x].diag) + ((uint64_t)me.z << 11), t,
                me.z << 12 | t << 1, 0u);
            ++b;
            const bool last = (me.w & 2u) != 0;
            if (win >= kSFold || last) {
                str_fold(y, hi, [&](uint32_t left) {
                    const StrOp &op = a.ops[me.x];
                    return str_nonfinite(left, op.sblk, wb, b, op.ent,
                                         a.psi[me.x] + (uint64_t)me.y * op.N,
                                         (uint64_t)me.z << 12 | t << 1);
                });
                win = 0;
                wb = b;
            }
            __syncwarp();
            if (lane == 0) arrive_local(&empty[s]);
            if (++s == kSMaxStages) {
                s = 0;
                par ^= 1u;
            }
            if (!last) continue;
            float2 *yo = a.y[me.x] + (uint64_t)me.y * a.ops[me.x].N + ((uint64_t)me.z << 12);
#pragma unroll
            for (int m = 0; m < 8; ++m)
                yo[2u * t + (m & 1u) + 1024u * (m >> 1)] = str_value(hi[m], y[m]);
        }
    }
    __syncthreads();
}

cudaError_t launch_strings_batch(const StrBatchArgs &a, uint32_t ctas, cudaStream_t st) {
    const size_t sm = (size_t)kSMaxStages * (kSTileBytes + kSEntBytes);
    cudaError_t e = ensure_dyn_smem(reinterpret_cast<const void *>(apply_c64c_strings_batch), sm);
    if (e != cudaSuccess) return e;
    const uint32_t grid = a.nitems < ctas ? a.nitems : ctas;
    if (grid == 0) return cudaSuccess;
    apply_c64c_strings_batch<<<grid, kSBlockThreads, sm, st>>>(a);
    count_launch();
    return cudaGetLastError();
}

// Clusters of ks CTAs that run at once (a GPC's SMs need not be a multiple of
// ks): asked once per device, kernel and ks.
static cudaError_t resident_clusters(const cudaLaunchConfig_t *cfg, const void *kern, uint32_t ks,
                                     int *out) {
    static std::mutex mu;
    static std::map<std::pair<std::pair<int, const void *>, uint32_t>, int> known;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(mu);
    const auto key = std::make_pair(std::make_pair(dev, kern), ks);
    const auto it = known.find(key);
    if (it != known.end()) {
        *out = it->second;
        return cudaSuccess;
    }
    int n = (int)cfg->gridDim.x;
    if (ks > 1) {
        e = cudaOccupancyMaxActiveClusters(&n, kern, cfg);
        if (e != cudaSuccess) return e;
    }
    if (n < 1) n = 1;
    known[key] = n;
    *out = n;
    return cudaSuccess;
}

cudaError_t launch_c64c_strings(const ApplyArgs &a_in, const StrSplit &sp, uint64_t call_items,
                                int nsm, cudaStream_t st) {
    ApplyArgs a = a_in;
    a.nsblk = sp.nblk;
    auto kern = (a.n > 32 || a.wide) ? apply_c64c_strings<true> : apply_c64c_strings<false>;
    const uint32_t stages = sp.tpb > 1 ? 3u : 4u;
    const size_t ring = (size_t)stages * (sp.tpb * kSTileBytes + kSEntBytes), xbytes = 65536;
    const size_t most = ring + (sp.tpb > 1 ? 0u : xbytes);
    if (most > 227u * 1024u) return cudaErrorInvalidValue;
    cudaError_t e = ensure_dyn_smem(reinterpret_cast<const void *>(kern), most);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3(kSBlockThreads);
    cfg.stream = st;
    cfg.attrs = at;
    // The split that needs the least time: rounds of resident clusters times
    // the strings of one CTA and its blocks (two strings each), with 16 more
    // for the exchange of the sums.  Measured, n = 16, 1,000 strings, split in
    // 1 / 2 / 4 / 5 / 8: one state 169 / 93 / 52 / 44 / 60 us (15 clusters of
    // 8 run at once, so 16 tiles take two rounds), three states 169 / 93 / 99
    // / 81 / 117, eight 170 / 181 / 194 / 195 / 257.
    uint32_t ks = 1;
    uint64_t ncl = 0, best = ~0ull;
    for (uint32_t k = 1; k <= (sp.tpb > 1 ? 1u : kStrMaxSplit); ++k) {
        if (k > 1 && sp.nstr < 8u * k) break;
        at[0].val.clusterDim.x = k;
        cfg.numAttrs = k > 1 ? 1 : 0;
        cfg.dynamicSmemBytes = ring + (k > 1 ? xbytes : 0u);
        cfg.gridDim = dim3((unsigned)nsm / k * k);
        int res = 0;
        e = resident_clusters(&cfg, reinterpret_cast<const void *>(kern), k, &res);
        if (e != cudaSuccess) return e;
        const uint64_t rounds = (call_items + (uint64_t)res - 1) / (uint64_t)res;
        const uint64_t cost = rounds * ((sp.nstr + 2ull * sp.nblk) / k + (k > 1 ? 16u : 0u));
        if (cost < best) {
            best = cost;
            ks = k;
            ncl = (uint64_t)res;
        }
    }
    if (ncl > a.nitems) ncl = a.nitems;
    if (ncl == 0) return cudaSuccess;
    for (uint32_t r = 0; r <= ks; ++r) a.part[r] = sp.part[ks - 1][r];
    at[0].val.clusterDim.x = ks;
    cfg.numAttrs = ks > 1 ? 1 : 0;
    cfg.dynamicSmemBytes = ring + (ks > 1 ? xbytes : 0u);
    cfg.gridDim = dim3((unsigned)(ncl * ks));
    e = cudaLaunchKernelEx(&cfg, kern, a, stages, ks, sp.tpb);
    if (e != cudaSuccess) return e;
    count_launch();
    return cudaGetLastError();
}

}  // namespace qr
