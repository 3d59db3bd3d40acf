// qr_csr.cu -- CSR assembly of a Pauli sum and CSR * vector on sm_103a.
//
// csr_fill replaces qrusty's rowwise builder (qrusty/src/accel.rs:171-210
// make_row, :267-336 make_unsafe_vectors_chunked).  Row r of the matrix has
// exactly G entries, one per distinct x mask: column r ^ x_g, value the sum
// of +-c'_k over the terms of group g in input order (a left fold starting
// from the first term, as make_row's fold does), explicit zeros kept.
//
// Column order without sorting: with the groups' x masks sorted ascending,
// the rank of r ^ x_g among {r ^ x_h} is
//     pos_r(g) = g + sum_{b : bit b of r set} sigma_{g,b},
// where sigma_{g,b} = +S (x_g has 0 at b) or -S (x_g has 1 at b) and S is
// the size of g's sibling subtree at bit b of the binary trie of the x
// masks (nonzero only at the trie's branching bits).  qr_group.cu computes
// the sigmas; each thread places one (row, group) entry directly.
//
// Values without a per-row fold: a group's value in row r depends on r only
// through the parities of r against the group's z masks, i.e. against z0 and
// a GF(2) basis beta_1..beta_d of the differences z_k ^ z0.  For d <= 4
// the group's +-c'_k are folded in input order once per class (2^(d+1)
// classes) -- the same additions in the same order as make_row, hence the
// same bits -- and the kernel reads the row's class from that table.
#include "qr_common.cuh"
#include "qr_device.cuh"

namespace qr {

__global__ void __launch_bounds__(256) csr_indptr_kernel(uint64_t N, uint64_t G,
                                                         uint64_t *indptr) {
    for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r <= N;
         r += (uint64_t)gridDim.x * blockDim.x)
        indptr[r] = r * G;
}

// Row bits as a 32-bit word when n <= 32 (half the integer work), else 64.
template <bool WIDE> struct RowT { using T = uint32_t; };
template <> struct RowT<true> { using T = uint64_t; };

template <typename W>
__device__ __forceinline__ uint32_t parity(W v) {
    if constexpr (sizeof(W) == 8) return (uint32_t)__popcll(v) & 1u;
    else return (uint32_t)__popc(v) & 1u;
}
template <typename W>
__device__ __forceinline__ int lowbit(W v) {
    if constexpr (sizeof(W) == 8) return __ffsll((long long)v) - 1;
    else return __ffs((int)v) - 1;
}

// sum of sigma_b over the set bits b of m (sig: the group's row of the table)
template <typename W>
__device__ __forceinline__ int32_t sigma_sum(W m, const int32_t *sig) {
    int32_t s = 0;
    for (; m; m &= m - 1) s += sig[lowbit(m)];
    return s;
}

__device__ __forceinline__ void csr_store(const CsrArgs &a, uint64_t rr, int32_t pos, uint64_t col,
                                          double2 v) {
    if (pos < 0 || (uint64_t)pos >= a.G) {  // cannot happen for a valid trie table
        atomicExch(a.err, kErrCsrPos);
        return;
    }
    const uint64_t o = rr * a.G + (uint64_t)pos;
    a.indices[o] = col;
    reinterpret_cast<double2 *>(a.data)[o] = v;
}

// Class of row r for group d: bit 0 = parity(r & z0), bit j+1 = parity(r & beta_j).
template <typename W>
__device__ __forceinline__ uint32_t csr_class(const CsrGroup &d, W r) {
    uint32_t c = parity<W>(r & (W)d.z0);
#pragma unroll
    for (int j = 0; j < kCsrMaxRank; ++j)
        if ((uint32_t)j < d.d) c |= parity<W>(r & (W)d.beta[j]) << (j + 1);
    return c;
}

constexpr int kCsrThreads = 256;
constexpr uint32_t kCsrSmemSig = 12288;  // sigma entries staged in shared memory (48 KB)
constexpr size_t kCsrLutBytes = 16u * 1024u;
constexpr uint32_t kCsrSmemCtab = 2048;  // class-table entries staged in shared memory (32 KB)

// Low-bit width of the per-group position lookup table: G x (2^L + 1)
// 32-bit entries (rows padded by one word so lanes on consecutive groups hit
// distinct banks) within 16 KB.  L <= 8, so 256-row launches stay aligned.
__host__ __device__ inline int csr_lut_bits(uint32_t G) {
    int L = 8;
    while (L > 1 && (size_t)G * ((1u << L) + 1) * 4u > kCsrLutBytes) --L;
    return L;
}

// Class-table groups.  G <= 256: blocks take chunks of 2^L rows; in a chunk,
// thread t owns group g = t % G of rows t / G, t / G + 256 / G, ..., so its
// descriptor and position mask stay in registers; the position terms of the
// row bits above the chunk are summed once per chunk and the low L bits come
// from a shared-memory table built per block.  G > 256: one row per pass,
// threads stride the groups.  Fold-mode groups are left to csr_fold_kernel,
// so no lane of a warp waits on another's long fold.
template <bool WIDE>
__global__ void __launch_bounds__(kCsrThreads) csr_fill_kernel(const CsrArgs a) {
    using W = typename RowT<WIDE>::T;
    extern __shared__ int32_t s_dyn[];
    const uint32_t G = (uint32_t)a.G;
    if (G <= (uint32_t)kCsrThreads) {
        const int L = csr_lut_bits(G);
        const uint32_t lsz = (1u << L) + 1;  // padded row
        for (uint32_t i = threadIdx.x; i < G * lsz; i += kCsrThreads) {
            const uint32_t g = i / lsz, v = i - g * lsz;
            const W pm = (W)a.pmask[g] & (((W)1 << L) - 1) & (W)v;
            s_dyn[i] = v < (1u << L) ? sigma_sum<W>(pm, a.sig + (size_t)g * (uint32_t)a.n) : 0;
        }
        // class tables next to the position table when they fit
        double2 *s_ctab = reinterpret_cast<double2 *>(s_dyn + ((G * lsz + 3u) & ~3u));
        const bool ctab_smem = a.nctab <= kCsrSmemCtab;
        if (ctab_smem)
            for (uint32_t i = threadIdx.x; i < a.nctab; i += kCsrThreads) s_ctab[i] = a.ctab[i];
        __syncthreads();
        const uint32_t rpp = kCsrThreads / G;
        const uint32_t t = threadIdx.x;
        if (t >= rpp * G) return;  // no barrier follows
        const uint32_t rs = t / G, g = t - rs * G;
        const CsrGroup d = a.grp[g];
        if (d.d == kCsrFold) return;
        const W xg = (W)a.gx[g], pm = (W)a.pmask[g];
        const W lomask = ((W)1 << L) - 1;
        const int32_t *sg = a.sig + (size_t)g * (uint32_t)a.n;
        const int32_t *lut = s_dyn + g * lsz;
        const uint64_t nchunk = (a.nrows + lomask) >> L;
        // the class table is read through a pointer of known state space
        // (shared or global), so the loads are LDS / LDG, not generic
        auto rows = [&](const double2 *tab) {
            for (uint64_t ch = blockIdx.x; ch < nchunk; ch += gridDim.x) {
                const uint64_t rr0 = ch << L;
                const W base = (W)(a.row0 + rr0);
                const int32_t phi = (int32_t)g + sigma_sum<W>(base & pm & ~lomask, sg);
                const uint64_t rend = min(rr0 + ((uint64_t)1 << L), a.nrows);
                // two rows per step: their table reads are in flight together
                for (uint64_t rr = rr0 + rs; rr < rend; rr += 2 * (uint64_t)rpp) {
                    const uint64_t rr2 = rr + rpp;
                    const W r = (W)(a.row0 + rr), r2 = (W)(a.row0 + rr2);
                    const bool two = rr2 < rend;
                    const double2 v1 = tab[csr_class<W>(d, r)];
                    const double2 v2 = two ? tab[csr_class<W>(d, r2)] : v1;
                    csr_store(a, rr, phi + lut[(uint32_t)(r & lomask)], (uint64_t)(r ^ xg), v1);
                    if (two)
                        csr_store(a, rr2, phi + lut[(uint32_t)(r2 & lomask)], (uint64_t)(r2 ^ xg),
                                  v2);
                }
            }
        };
        if (ctab_smem) rows(s_ctab + d.tab);
        else rows(a.ctab + d.tab);
    } else {
        const uint64_t nsig = (uint64_t)G * (uint32_t)a.n;
        const bool staged = nsig <= kCsrSmemSig;
        if (staged)
            for (uint32_t i = threadIdx.x; i < nsig; i += kCsrThreads) s_dyn[i] = a.sig[i];
        __syncthreads();
        const int32_t *sig = staged ? s_dyn : a.sig;
        for (uint64_t rr = blockIdx.x; rr < a.nrows; rr += gridDim.x) {
            const W r = (W)(a.row0 + rr);
            for (uint32_t g = threadIdx.x; g < G; g += kCsrThreads) {
                const CsrGroup d = a.grp[g];
                if (d.d == kCsrFold) continue;
                const int32_t pos = (int32_t)g + sigma_sum<W>(r & (W)a.pmask[g],
                                                              sig + (size_t)g * (uint32_t)a.n);
                csr_store(a, rr, pos, (uint64_t)(r ^ (W)a.gx[g]),
                          a.ctab[d.tab + csr_class<W>(d, r)]);
            }
        }
    }
}

// Fold-mode groups (z span wider than kCsrMaxRank): one thread per row, all
// lanes of a warp on the same group, the group's +-c'_k folded in input-term
// order from the first term (make_row's fold), terms read warp-uniformly.
// The leading terms up to a bounded z-span rank (kCsrPrefixRank) come from a
// per-class fold of them (same additions, same order); the rest are added
// per row.  A part (re or im) whose every coefficient is +-0 takes no FP64
// additions: under round-to-nearest a sum of signed zeros is -0 exactly when
// every addend is -0, so the fold's result is -0 iff each +-c'_k part is -0.
template <bool RZ, bool IZ>
__device__ __forceinline__ double2 csr_fold_row(const CsrArgs &a, uint64_t r, const CsrGroup &d,
                                                uint32_t f) {
    const uint64_t *tz = a.tz;
    const double *tc = a.tc;
    double vr = 0.0, vi = 0.0;
    uint32_t nr = 1u, ni = 1u;  // every addend so far -0 (zero parts)
    uint32_t k = d.k0;
    const uint32_t m = d.pre & 0xffffffu;
    if (m != 0) {
        // the fold of the leading m terms, looked up by the row's sign class
        const uint32_t dp = d.pre >> 24;
        const uint64_t *pb = a.pbeta + (size_t)f * kCsrPrefixRank;
        uint32_t c = (uint32_t)__popcll(r & d.z0) & 1u;
        for (uint32_t j = 0; j < dp; ++j) c |= ((uint32_t)__popcll(r & pb[j]) & 1u) << (j + 1);
        const double2 v = a.ptab[d.tab + c];
        vr = v.x;
        vi = v.y;
        nr = (uint32_t)signbit(v.x);
        ni = (uint32_t)signbit(v.y);
        k += m;
    }
    for (; k < d.k1; ++k) {
        // sign applied to the bit pattern: no floating-point negation
        const uint64_t sb = (uint64_t)(__popcll(r & tz[k]) & 1) << 63;
        if constexpr (RZ) {
            nr &= (uint32_t)(sb >> 63) ^ (uint32_t)signbit(tc[2 * k]);
        } else {
            const double cr = __longlong_as_double(__double_as_longlong(tc[2 * k]) ^ (long long)sb);
            vr = k == d.k0 ? cr : __dadd_rn(vr, cr);
        }
        if constexpr (IZ) {
            ni &= (uint32_t)(sb >> 63) ^ (uint32_t)signbit(tc[2 * k + 1]);
        } else {
            const double ci =
                __longlong_as_double(__double_as_longlong(tc[2 * k + 1]) ^ (long long)sb);
            vi = k == d.k0 ? ci : __dadd_rn(vi, ci);
        }
    }
    if constexpr (RZ) vr = nr ? -0.0 : 0.0;
    if constexpr (IZ) vi = ni ? -0.0 : 0.0;
    return make_double2(vr, vi);
}

__device__ __forceinline__ double2 csr_fold_entry(const CsrArgs &a, uint64_t r, const CsrGroup &d,
                                                  uint32_t f) {
    switch (d.zparts & 3u) {  // warp-uniform
        case 1: return csr_fold_row<true, false>(a, r, d, f);
        case 2: return csr_fold_row<false, true>(a, r, d, f);
        case 3: return csr_fold_row<true, true>(a, r, d, f);
        default: return csr_fold_row<false, false>(a, r, d, f);
    }
}

// ------------------------------------------------------------ staged fill
// Rows are assembled in shared memory and leave the SM as contiguous TMA
// bulk stores (cp.async.bulk shared -> global): a warp's entries of one row
// land at permuted positions, which as direct global stores become many
// partial-line L2 writes.  Three staging buffers of R rows: one barrier per
// stage, and a buffer's bulk store has a whole stage to finish reading it.
// Eight warps assemble class-table entries; a ninth issues the bulk stores
// and folds the entries of a short fold-mode group (csr_inline_fold).  Other
// folds are computed first by csr_fold_kernel<true> into a row-major value
// buffer and placed from there: their serial chains would hold the block at
// the barrier, and stored in place after the fill each entry becomes a DRAM
// read-modify-write of a line the bulk store has already evicted (cheaper than
// the placing for one group of many rows: qr_csr_build).  Without a
// value buffer they are left unset and stored afterwards by
// csr_fold_kernel<false>.  Which of these a launch needs is a template
// argument: the code of all three in one body costs 10 %.
//
// Bound by the write stream (2.11 GB at chain n = 21, 42 groups: 271 us at
// the rate of a device fill), so the order of the writes counts: blocks that
// stride or halve the rows by a fixed rule finish unevenly and reach
// 6.6 TB/s with any stage size, blocks that take the next piece of rows as
// they get free 7.7.  Hence one block per unit of about 128 KB, and a resident
// block goes on with the next unit that has not started
// (clusterlaunchcontrol), which keeps its tables.  What is left above the
// write stream's time is a stage's barrier, stores and bookkeeping: chain
// n = 21 takes 330 us (two-buffer stages over fixed strides, per-chunk sums
// in every thread and a fold kernel before it: 487), random strings n = 16,
// 200 groups, 55 us (67).
constexpr uint32_t kCsrBufs = 3;  // staging buffers
constexpr int kCsrStageThreads = kCsrThreads + 32;
constexpr size_t kCsrStageBytes = 16896u;  // one buffer, at most: R rows x G x (8 + 16) bytes
constexpr size_t kCsrUnitBytes = 131072u;   // output of one unit, about
constexpr size_t kCsrLowBytes = 9u * 1024u, kCsrTableBytes = 26u * 1024u;
constexpr int kCsrChunkBits = 6;        // chunk rows of the inline fold: two per lane of its warp
constexpr uint32_t kCsrRingItems = 256;  // value-buffer entries of a chunk kept ahead, at most
constexpr uint32_t kCsrInlineRem = 64;  // its terms past the prefix, at most

// Chunk and stage of the staged fill.  A chunk is 2^L rows.  What a row's bits
// add to a group's position and class comes from tables of one 16-bit word
// per (group, bits): position term (11 bits, signed) and class term (5 bits),
// rows padded to an odd number of 32-bit words; one table for the low L bits
// and `up` tables for U bits each above them (bits above those are summed per
// chunk).  For the inline fold the same split holds the parities that pick
// prefix class and term signs.  The tables depend on masks only and are
// written once per operator (csr_tables_kernel).  A stage holds R rows (even,
// so that bulk stores are whole 16-byte units), the chunk in equal parts.
struct CsrStage {
    int L, U, up;
    uint32_t R, lsz, usz;  // lsz, usz: 16-bit words of a group's table row
    uint32_t ups, ups_sz;  // first upper table, words of one
    uint32_t cls, sgn, bytes;  // byte offsets of the inline folds' classes and signs; table bytes
    // byte offsets in shared memory (class table: 0 where it stays in global memory)
    uint32_t ctab, tc, bufs, buf_bytes, fold, fphi, fval, total;
    bool ring;  // value-buffer entries pass through shared memory
};
__host__ __device__ inline uint32_t csr_align(size_t b, uint32_t to) {
    return ((uint32_t)b + to - 1u) & ~(to - 1u);
}
__host__ __device__ inline CsrStage csr_stage(uint32_t G, int n, uint32_t nctab, uint32_t nfv) {
    CsrStage s;
    // 64 rows where they fill a stage, else 256; 512 for one group of many rows (one
    // string, n = 20: 19 us with 256, 15 so; n = 6 6.6 and 8.6)
    s.L = (size_t)G * 24u << kCsrChunkBits >= kCsrStageBytes ? kCsrChunkBits
          : G == 1 && n >= 18                                ? 9
                                                             : 8;
    while (s.L > 1 && (size_t)G * ((1u << s.L) + 2) * 2u > kCsrLowBytes) --s.L;
    s.U = s.L > 1 ? s.L - 1 : 1;
    s.lsz = (1u << s.L) + 2;
    s.usz = (1u << s.U) + 2;
    s.ups = csr_align((size_t)G * s.lsz, 8);
    s.ups_sz = csr_align((size_t)G * s.usz, 8);
    s.up = 0;
    while (s.L + s.up * s.U < n &&
           ((size_t)s.ups + (size_t)(s.up + 1) * s.ups_sz) * 2u <= kCsrTableBytes)
        ++s.up;
    const uint32_t words = (1u << s.L) + (uint32_t)s.up * (1u << s.U);
    s.cls = (s.ups + (uint32_t)s.up * s.ups_sz) * 2u;
    s.sgn = csr_align(s.cls + words * 2u, 16);
    s.bytes = csr_align(s.sgn + words * 8u, 16);
    const uint32_t rows = 1u << s.L;
    uint32_t most = (uint32_t)(kCsrStageBytes / ((size_t)G * 24u)) & ~1u;
    if (most < 2) most = 2;
    const uint32_t parts = (rows + most - 1) / most;
    s.R = ((rows + parts - 1) / parts + 1u) & ~1u;
    const bool ct = nctab <= kCsrSmemCtab;
    s.ctab = ct ? s.bytes : 0u;
    s.tc = s.bytes + (ct ? nctab * (uint32_t)sizeof(double2) : 0u);
    s.bufs = csr_align(s.tc + kCsrInlineRem * sizeof(double2), 128);
    s.buf_bytes = csr_align((size_t)s.R * G * 24u, 128);
    // value buffer: the groups' x and index, and for two chunks their position
    // terms and values
    s.fold = s.bufs + kCsrBufs * s.buf_bytes;
    s.fphi = s.fold + nfv * 12u;
    s.fval = csr_align(s.fphi + 2u * nfv * sizeof(int32_t), 16);
    s.ring = nfv > 0 && (nfv << s.L) <= kCsrRingItems;
    s.total = s.fval + (s.ring ? 2u * (nfv << s.L) * (uint32_t)sizeof(double2) : 0u);
    return s;
}
// Chunks of one unit: about kCsrUnitBytes of output, fewer where the rows
// would leave SMs idle.
__host__ __device__ inline uint32_t csr_unit_chunks(uint32_t G, int L, uint64_t nchunk, int nsm) {
    uint64_t q = kCsrUnitBytes / (((size_t)G * 24u) << L);
    if (q > nchunk / (2u * (uint32_t)nsm)) q = nchunk / (2u * (uint32_t)nsm);
    return q < 1 ? 1u : (uint32_t)q;
}

// A fold-mode group inside the staged fill: one warp per CTA folds a chunk's
// rows, two per lane, in about 130 clocks a term past the prefix; the block's
// share of the write stream takes about (G << L) * 2.8 clocks a chunk.  Folded
// here while the fold is a third of that at most (chain n = 21, 9 terms and
// 2,688 entries a chunk: 338 us against 370 through the value buffer; an
// operator of 94 groups, 26 terms and chunks of 16 rows: 195 against 158;
// both with prefixes of rank 10).  One group (the
// diagonal of a spin chain); all row bits have to be in the tables.
bool csr_inline_fold(uint64_t G, int n, uint32_t nfold, uint32_t fold_rem) {
    if (G > (uint64_t)kCsrThreads || nfold != 1 || fold_rem > kCsrInlineRem) return false;
    const CsrStage s = csr_stage((uint32_t)G, n, 0, 0);
    return s.L <= kCsrChunkBits && s.L + s.up * s.U >= n &&
           fold_rem * 128u <= (uint32_t)G << s.L;
}
size_t csr_tables_bytes(uint64_t G, int n) {
    return G <= (uint64_t)kCsrThreads ? csr_stage((uint32_t)G, n, 0, 0).bytes : 0;
}

__global__ void __launch_bounds__(kCsrThreads) csr_tables_kernel(const CsrArgs a) {
    const uint32_t G = (uint32_t)a.G;
    const CsrStage cs = csr_stage(G, a.n, a.nctab, 0);
    uint16_t *const w16 = const_cast<uint16_t *>(a.tables);
    const uint32_t nlow = G << cs.L, nup = G << cs.U, ntab = nlow + (uint32_t)cs.up * nup;
    const uint32_t per = (1u << cs.L) + (uint32_t)cs.up * (1u << cs.U);
    const uint32_t step = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < ntab + (a.inline_fold ? per : 0u);
         i += step) {
        if (i < ntab) {
            const uint32_t lev = i < nlow ? 0u : 1u + (i - nlow) / nup;
            const uint32_t j = lev ? (i - nlow) % nup : i;
            const int b = lev ? cs.U : cs.L;
            const uint32_t g = j >> b, v = j & ((1u << b) - 1u);
            const uint64_t z = (uint64_t)v << (lev ? cs.L + (int)(lev - 1u) * cs.U : 0);
            const CsrGroup dg = a.grp[g];
            uint32_t w = (uint32_t)sigma_sum<uint64_t>(z & a.pmask[g],
                                                       a.sig + (size_t)g * (uint32_t)a.n) & 0x7ffu;
            if (dg.d != kCsrFold) w |= csr_class<uint64_t>(dg, z) << 11;
            w16[lev ? cs.ups + (lev - 1u) * cs.ups_sz + g * cs.usz + v : g * cs.lsz + v] =
                (uint16_t)w;
        } else {
            const uint32_t j = i - ntab;
            const uint32_t lo = 1u << cs.L;
            const uint32_t lev = j < lo ? 0u : 1u + (j - lo) / (1u << cs.U);
            const uint32_t v = lev ? (j - lo) & ((1u << cs.U) - 1u) : j;
            const uint64_t z = (uint64_t)v << (lev ? cs.L + (int)(lev - 1u) * cs.U : 0);
            const CsrGroup d = a.grp[a.fold[0]];
            const uint32_t m = d.pre & 0xffffffu, dp = d.pre >> 24;
            uint32_t c = parity<uint64_t>(z & d.z0);
            for (uint32_t q = 0; q < dp; ++q) c |= parity<uint64_t>(z & a.pbeta[q]) << (q + 1);
            uint64_t sg = 0;
            for (uint32_t q = 0; d.k0 + m + q < d.k1; ++q)
                sg |= (uint64_t)parity<uint64_t>(z & a.tz[d.k0 + m + q]) << q;
            w16[cs.cls / 2u + j] = (uint16_t)c;
            reinterpret_cast<uint64_t *>(w16 + cs.sgn / 2u)[j] = sg;
        }
    }
}

cudaError_t launch_csr_tables(const CsrArgs &a, cudaStream_t st) {
    if (a.G > (uint64_t)kCsrThreads) return cudaSuccess;
    const CsrStage cs = csr_stage((uint32_t)a.G, a.n, a.nctab, 0);
    cudaError_t e = cudaMemsetAsync(const_cast<uint16_t *>(a.tables), 0, cs.bytes, st);
    if (e != cudaSuccess) return e;
    const uint32_t n = ((uint32_t)a.G << cs.L) + (uint32_t)cs.up * ((uint32_t)a.G << cs.U);
    csr_tables_kernel<<<(n + kCsrThreads - 1) / kCsrThreads, kCsrThreads, 0, st>>>(a);
    count_launch();
    return cudaGetLastError();
}

__device__ __forceinline__ void csr_bulk_s2g(void *dst, const void *src, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
                 "r"(saddr(src)), "r"(bytes)
                 : "memory");
}
// Ask for the next block of the grid that has not started; the answer (16
// bytes) arrives on the barrier.
__device__ __forceinline__ void next_block_ask(void *resp, uint64_t *bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], 16;" ::"r"(saddr(bar))
                 : "memory");
    asm volatile(
        "clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 "
        "[%0], [%1];" ::"r"(saddr(resp)),
        "r"(saddr(bar))
        : "memory");
}
// Block index of the answer, or kCsrNoUnit.
constexpr uint32_t kCsrNoUnit = 0xffffffffu;
__device__ __forceinline__ uint32_t next_block_answer(const void *resp) {
    uint32_t x;
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b128 v;\n\tld.shared.b128 v, [%1];\n\t"
        "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, v;\n\t"
        "mov.u32 %0, 0xffffffff;\n\t"
        "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %0, v;\n\t}"
        : "=r"(x)
        : "r"(saddr(resp))
        : "memory");
    return x;
}
__device__ __forceinline__ uint32_t hi_word(double v) { return (uint32_t)__double2hiint(v); }
// term << 31 of a sign mask onto a value
__device__ __forceinline__ double sign_by(double v, uint32_t bit) {
    return __hiloint2double((int)(hi_word(v) ^ (bit << 31)), __double2loint(v));
}

// The inline fold's group.
struct FoldDesc {
    uint64_t x;
    uint32_t g, tab, m, rem, zparts;
};
// The terms after the prefix folded onto the values of a lane's two rows
// (csr_fold_row's additions and signs of zero), together: a dependent addition
// takes about 100 clocks.
template <bool RE, bool IM>
__device__ __forceinline__ void fold_rest(const FoldDesc &fd, const double2 *tc,
                                          const uint64_t (&sg)[2], double2 (&v)[2]) {
    constexpr uint32_t K = 2;
    const bool pre = fd.m != 0;
    uint32_t nr[K], ni[K];
#pragma unroll
    for (uint32_t i = 0; i < K; ++i) {
        nr[i] = pre ? hi_word(v[i].x) >> 31 : 1u;
        ni[i] = pre ? hi_word(v[i].y) >> 31 : 1u;
    }
    for (uint32_t j = 0; j < fd.rem; ++j) {
        const double2 c = tc[j];
#pragma unroll
        for (uint32_t i = 0; i < K; ++i) {
            const uint32_t s1 = (uint32_t)(sg[i] >> j) & 1u;
            const double cr = sign_by(c.x, s1), ci = sign_by(c.y, s1);
            if constexpr (RE) v[i].x = pre || j ? __dadd_rn(v[i].x, cr) : cr;
            else nr[i] &= hi_word(cr) >> 31;
            if constexpr (IM) v[i].y = pre || j ? __dadd_rn(v[i].y, ci) : ci;
            else ni[i] &= hi_word(ci) >> 31;
        }
    }
#pragma unroll
    for (uint32_t i = 0; i < K; ++i) {
        if constexpr (!RE) v[i].x = nr[i] ? -0.0 : 0.0;
        if constexpr (!IM) v[i].y = ni[i] ? -0.0 : 0.0;
    }
}

// FOLD: 0 no fold-mode group placed, 1 one folded here, 2 from the value buffer
template <bool WIDE, int FOLD>
__global__ void __launch_bounds__(kCsrStageThreads, 3) csr_fill_staged_kernel(const CsrArgs a,
                                                                              uint32_t q) {
    using W = typename RowT<WIDE>::T;
    extern __shared__ __align__(128) int32_t s_dyn[];
    __shared__ __align__(16) uint4 s_resp;
    __shared__ __align__(8) uint64_t s_bar;
    __shared__ FoldDesc s_fold;
    __shared__ __align__(16) double2 s_fval[2][1 << kCsrChunkBits];
    __shared__ uint32_t s_next[2];  // next unit, by the parity of this block's units
    unsigned char *const s_base = reinterpret_cast<unsigned char *>(s_dyn);
    const uint32_t G = (uint32_t)a.G;
    const uint32_t nfv = FOLD == 2 ? a.nfold : 0u;
    constexpr bool inl = FOLD == 1;
    const CsrStage cs = csr_stage(G, a.n, a.nctab, nfv);
    const int L = cs.L, U = cs.U;
    const uint32_t lsz = cs.lsz;
    const uint32_t t = threadIdx.x;
    const bool helper = t >= (uint32_t)kCsrThreads;  // the ninth warp
    const W lomask = ((W)1 << L) - 1;
    const uint64_t nchunk = (a.nrows + lomask) >> L;
    {
        const uint4 *src = reinterpret_cast<const uint4 *>(a.tables);
        uint4 *dst = reinterpret_cast<uint4 *>(s_base);
        for (uint32_t i = t; i < cs.bytes / 16u; i += kCsrStageThreads) dst[i] = src[i];
    }
    const uint16_t *s_lut = reinterpret_cast<const uint16_t *>(s_base);
    const bool ctab_smem = cs.ctab != 0;
    double2 *s_ctab = reinterpret_cast<double2 *>(s_base + cs.ctab);
    if (ctab_smem)
        for (uint32_t i = t; i < a.nctab; i += kCsrStageThreads) s_ctab[i] = a.ctab[i];
    double2 *s_tc = reinterpret_cast<double2 *>(s_base + cs.tc);
    if (inl) {
        const CsrGroup &df = a.grp[a.fold[0]];
        const uint32_t m = df.pre & 0xffffffu, k = df.k0 + m, rem = df.k1 - k;
        if (t == 0) s_fold = {a.gx[a.fold[0]], a.fold[0], df.tab, m, rem, df.zparts & 3u};
        for (uint32_t i = t; i < rem && i < kCsrInlineRem; i += kCsrStageThreads)
            s_tc[i] = make_double2(a.tc[2 * (size_t)(k + i)], a.tc[2 * (size_t)(k + i) + 1]);
    }
    // groups of the value buffer
    uint64_t *s_fx = reinterpret_cast<uint64_t *>(s_base + cs.fold);
    uint32_t *s_fg = reinterpret_cast<uint32_t *>(s_fx + nfv);
    for (uint32_t f = t; f < nfv; f += kCsrStageThreads) {
        s_fg[f] = a.fold[f];
        s_fx[f] = a.gx[a.fold[f]];
    }
    if (t == (uint32_t)kCsrThreads) {
        mbar_init(&s_bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    const uint32_t R = cs.R;
    const uint32_t rpp = kCsrThreads / G;
    const uint32_t rs = t / G, g = t - rs * G;
    CsrGroup d{};
    W xg = 0;
    bool active = false;
    if (t < rpp * G) {  // idle threads still take every barrier
        d = a.grp[g];
        active = d.d != kCsrFold;
        xg = (W)a.gx[g];
    }
    const uint16_t *lut = s_lut + (active ? g : 0u) * lsz;
    const double2 *tab = (ctab_smem ? s_ctab : a.ctab) + d.tab;
    // Groups of span rank 0 and 1 (2 and 4 classes) keep their values in
    // registers: the entries of classes 0 and 2, and for each part whether
    // the class with bit 0 set (every term's sign flipped) has it negated
    // (not so where the sum cancels to zero).  Lanes reading the table at
    // their rows' classes conflict on its banks.
    double2 e0 = make_double2(0.0, 0.0), e1 = e0;
    uint32_t neg = 0;  // bits 0, 1: parts of e0; bits 2, 3: of e1
    bool held = active && d.d <= 1;
    if (held) {
        e0 = tab[0];
        e1 = d.d ? tab[2] : e0;
        const double2 f0 = tab[1], f1 = d.d ? tab[3] : f0;
        auto flip_of = [&](double p, double r, uint32_t bit) {
            const uint64_t x = (uint64_t)(__double_as_longlong(p) ^ __double_as_longlong(r));
            if (x == 1ull << 63) neg |= 1u << bit;
            else if (x != 0) held = false;
        };
        flip_of(e0.x, f0.x, 0);
        flip_of(e0.y, f0.y, 1);
        flip_of(e1.x, f1.x, 2);
        flip_of(e1.y, f1.y, 3);
    }
    auto pos_of = [](uint32_t w) { return (int32_t)(w << 21) >> 21; };
    // position (from gq on) and class terms of a chunk's high bits
    auto high_terms = [&](uint32_t gq, W hi, bool fold, int32_t *ph, uint32_t *cl) {
        int32_t p = (int32_t)gq;
        uint32_t c = 0;
        const uint16_t *row = s_lut + cs.ups + gq * cs.usz;
        W rest = hi >> L;
        for (int l = 0; l < cs.up; ++l, row += cs.ups_sz) {
            const uint32_t w = row[(uint32_t)rest & ((1u << U) - 1u)];
            p += pos_of(w);
            c ^= w >> 11;
            rest >>= U;
        }
        if (rest) {  // bits above the tables
            const W top = rest << (L + cs.up * U);
            p += sigma_sum<W>(top & (W)a.pmask[gq], a.sig + (size_t)gq * (uint32_t)a.n);
            if (!fold) c ^= csr_class<W>(a.grp[gq], top);
        }
        *ph = p;
        *cl = c;
    };
    uint32_t b = 0;  // staging buffer
    uint32_t par = 0, ask = 0;
    uint32_t unit = blockIdx.x;
    int32_t phi = 0;
    uint32_t cls = 0;
    auto answer = [&]() {
        if (mbar_wait_bounded(&s_bar, ask, kWaitLimitNs)) return next_block_answer(&s_resp);
        atomicExch(a.err, kErrMbarTimeout);
        return kCsrNoUnit;
    };
    // Inline fold, a chunk ahead of the stages: at a chunk's first stage the
    // helper's lanes read the next chunk's prefix values (on their way while
    // the stages pass), at its last stage they add the other terms and leave
    // the values in shared memory, by the parity of this block's chunks.
    const uint32_t lane = t & 31u;
    const uint16_t *s_cls = reinterpret_cast<const uint16_t *>(s_base + cs.cls);
    const uint64_t *s_sgn = reinterpret_cast<const uint64_t *>(s_base + cs.sgn);
    double2 it_v[2];   // rows lane and lane + 32 of the next chunk
    uint64_t it_s[2];
    auto fold_fetch = [&](uint64_t ch) {
        W rest = (W)(a.row0 + (ch << L)) >> L;
        uint32_t c = 0;
        uint64_t sg = 0;
        for (uint32_t j = 1u << L, l = 0; l < (uint32_t)cs.up; ++l, j += 1u << U, rest >>= U) {
            const uint32_t i = j + ((uint32_t)rest & ((1u << U) - 1u));
            c ^= s_cls[i];
            sg ^= s_sgn[i];
        }
#pragma unroll
        for (uint32_t i = 0; i < 2; ++i) {
            const uint32_t rl = (lane + 32u * i) & ((1u << L) - 1u);
            it_s[i] = sg ^ s_sgn[rl];
            it_v[i] = s_fold.m ? a.ptab[s_fold.tab + (c ^ s_cls[rl])] : make_double2(0.0, 0.0);
        }
    };
    auto fold_finish = [&](uint32_t to) {
        switch (s_fold.zparts) {
            case 1: fold_rest<false, true>(s_fold, s_tc, it_s, it_v); break;
            case 2: fold_rest<true, false>(s_fold, s_tc, it_s, it_v); break;
            case 3: fold_rest<false, false>(s_fold, s_tc, it_s, it_v); break;
            default: fold_rest<true, true>(s_fold, s_tc, it_s, it_v); break;
        }
        s_fval[to][lane] = it_v[0];
        s_fval[to][lane + 32u] = it_v[1];
        __syncwarp();
    };
    // Value buffer, a chunk ahead as well: position terms of the groups'
    // entries, and the values on their way to shared memory (from DRAM, the
    // fill's write stream having evicted them from L2).
    int32_t *s_fphi = reinterpret_cast<int32_t *>(s_base + cs.fphi);
    double2 *s_fv = reinterpret_cast<double2 *>(s_base + cs.fval);
    auto buffer_ahead = [&](uint64_t ch, uint32_t to) {
        const uint64_t rr0 = ch << L;
        const uint32_t rows = (uint32_t)min((uint64_t)1 << L, a.nrows - rr0);
        for (uint32_t f = lane; f < nfv; f += 32) {
            uint32_t cl;
            high_terms(s_fg[f], (W)(a.row0 + rr0), true, &s_fphi[to * nfv + f], &cl);
        }
        if (!cs.ring) return;
        for (uint32_t i = lane; i < nfv << L; i += 32) {
            const uint32_t f = i >> L, rl = i & ((1u << L) - 1u);
            if (rl < rows)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                                 saddr(s_fv + (to * nfv << L) + i)),
                             "l"(a.fvals + (size_t)f * a.nrows + rr0 + rl)
                             : "memory");
        }
    };
    if (helper && nfv > 0) {
        buffer_ahead((uint64_t)unit * q, 0);
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    // the unit after this block's first: asked for now, and each later one
    // while the unit before the last known is filled
    uint32_t after = kCsrNoUnit;
    if (t == (uint32_t)kCsrThreads) {
        next_block_ask(&s_resp, &s_bar);
        s_next[1] = answer();
    }
    if (helper && inl) {
        fold_fetch((uint64_t)unit * q);
        fold_finish(0);
    }
    __syncthreads();
    after = s_next[1];
    ask = 1;
    uint32_t cpar = 0;  // parity of this block's chunks
    while (unit != kCsrNoUnit) {
        if (t == (uint32_t)kCsrThreads && after != kCsrNoUnit) {
            // the last answer has been read: its buffer goes back to the async proxy
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            next_block_ask(&s_resp, &s_bar);
        }
        const uint64_t ch1 = min((uint64_t)(unit + 1ull) * q, nchunk);
        for (uint64_t ch = (uint64_t)unit * q; ch < ch1; ++ch) {
            const uint64_t rr0 = ch << L;
            const uint32_t crows = (uint32_t)min((uint64_t)1 << L, a.nrows - rr0);
            const W hi = (W)(a.row0 + rr0);
            if (active) high_terms(g, hi, false, &phi, &cls);
            for (uint32_t low = 0; low < crows; low += R) {
                const uint32_t rows = min(R, crows - low);
                const W r0 = hi + low;
                unsigned char *buf = s_base + cs.bufs + b * cs.buf_bytes;
                uint64_t *s_idx = reinterpret_cast<uint64_t *>(buf);
                double2 *s_val = reinterpret_cast<double2 *>(buf + R * G * 8u);
                auto put = [&](uint32_t rl, int32_t pos, W x, double2 v) {
                    if ((uint32_t)pos >= G) {  // cannot happen for a valid trie table
                        atomicExch(a.err, kErrCsrPos);
                        return;
                    }
                    s_idx[rl * G + (uint32_t)pos] = (uint64_t)((r0 + rl) ^ x);
                    s_val[rl * G + (uint32_t)pos] = v;
                };
                if (active) {
#pragma unroll 2
                    for (uint32_t rl = rs; rl < rows; rl += rpp) {
                        const uint32_t w = lut[low + rl];
                        const uint32_t c = cls ^ (w >> 11);
                        double2 v;
                        if (held) {
                            v = c & 2u ? e1 : e0;
                            const uint32_t m = neg >> (c & 2u);
                            v.x = sign_by(v.x, m & c);
                            v.y = sign_by(v.y, (m >> 1) & c);
                        } else {
                            v = ctab_smem ? s_ctab[d.tab + c] : tab[c];
                        }
                        put(rl, phi + pos_of(w), xg, v);
                    }
                }
                // entries of the value buffer
                if (nfv > 0 && !helper) {
                    const uint32_t nitem = nfv * rows;
                    for (uint32_t i = (uint32_t)kCsrThreads - 1u - t; i < nitem; i += kCsrThreads) {
                        const uint32_t f = i / rows, rl = i - f * rows;
                        const double2 v = cs.ring
                                              ? s_fv[((cpar * nfv + f) << L) + low + rl]
                                              : a.fvals[(size_t)f * a.nrows + rr0 + low + rl];
                        put(rl, s_fphi[cpar * nfv + f] + pos_of(s_lut[s_fg[f] * lsz + low + rl]),
                            (W)s_fx[f], v);
                    }
                }
                const bool last = low + R >= crows;  // the chunk's last stage
                const uint64_t chn = ch + 1 < ch1 ? ch + 1 : (uint64_t)after * q;
                const bool more = ch + 1 < ch1 || after != kCsrNoUnit;
                if (helper && nfv > 0) {
                    if (low == 0 && more) buffer_ahead(chn, cpar ^ 1u);
                    if (last) asm volatile("cp.async.wait_all;" ::: "memory");
                }
                if (helper && inl) {
                    if (low == 0 && more) fold_fetch(chn);
                    if (low == 0) high_terms(s_fold.g, hi, true, &phi, &cls);
                    for (uint32_t rl = lane; rl < rows; rl += 32)
                        put(rl, phi + pos_of(s_lut[s_fold.g * lsz + low + rl]), (W)s_fold.x,
                            s_fval[cpar][low + rl]);
                    if (last && more) fold_finish(cpar ^ 1u);
                }
                if (last && ch + 1 == ch1 && t == (uint32_t)kCsrThreads)
                    s_next[par] = after != kCsrNoUnit ? answer() : kCsrNoUnit;
                __syncthreads();
                if (t == (uint32_t)kCsrThreads) {
                    // the block's shared writes, ordered before this by the
                    // barrier, made visible to the bulk copies (one fence
                    // instead of every thread's: 5 % of the whole)
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    const uint64_t o = (rr0 + low) * G;
                    csr_bulk_s2g(a.indices + o, s_idx, rows * G * 8u);
                    csr_bulk_s2g(a.data + 2 * o, s_val, rows * G * 16u);
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    // the previous stage's buffer is read: stage k + 2 takes it, past
                    // the next barrier, at which this thread arrives after this wait
                    asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                }
                b = b + 1 == kCsrBufs ? 0u : b + 1;
            }
            cpar ^= 1u;
        }
        unit = after;
        after = s_next[par];  // written before the last barrier; the other half is written next
        par ^= 1u;
        ask ^= 1u;
    }
    if (t == (uint32_t)kCsrThreads) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// VALS: write the values row-major per fold group into a.fvals (coalesced),
// for the staged fill to place; otherwise store the entries in place.
template <bool VALS>
__global__ void __launch_bounds__(kCsrThreads) csr_fold_kernel(const CsrArgs a) {
    for (uint32_t f = blockIdx.y; f < a.nfold; f += gridDim.y) {
        const uint32_t g = a.fold[f];
        const CsrGroup d = a.grp[g];
        const uint64_t xg = a.gx[g], pm = a.pmask[g];
        const int32_t *sg = a.sig + (size_t)g * (uint32_t)a.n;
        for (uint64_t rr = blockIdx.x * (uint64_t)kCsrThreads + threadIdx.x; rr < a.nrows;
             rr += (uint64_t)gridDim.x * kCsrThreads) {
            const uint64_t r = a.row0 + rr;
            const double2 v = csr_fold_entry(a, r, d, f);
            if constexpr (VALS)
                a.fvals[(size_t)f * a.nrows + rr] = v;
            else
                csr_store(a, rr, (int32_t)g + sigma_sum<uint64_t>(r & pm, sg), r ^ xg, v);
        }
    }
}

// fold-mode groups, after the fill kernel on the same stream
static cudaError_t launch_csr_fold(const CsrArgs &a, int nsm, cudaStream_t st) {
    if (a.nfold == 0) return cudaSuccess;
    uint64_t gx = (a.nrows + kCsrThreads - 1) / kCsrThreads;
    const uint32_t gy = a.nfold < 65535u ? a.nfold : 65535u;
    uint64_t cap = ((uint64_t)nsm * 8 + gy - 1) / gy;
    if (cap < 1) cap = 1;
    if (gx > cap) gx = cap;
    if (a.fvals)
        csr_fold_kernel<true><<<dim3((unsigned)gx, gy), kCsrThreads, 0, st>>>(a);
    else
        csr_fold_kernel<false><<<dim3((unsigned)gx, gy), kCsrThreads, 0, st>>>(a);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_csr_fill(const CsrArgs &a, int nsm, cudaStream_t st) {
    if (a.row0 == 0 && a.indptr != nullptr) {
        uint64_t g = (a.N + 1 + 255) / 256;
        if (g > (uint64_t)nsm * 8) g = (uint64_t)nsm * 8;
        csr_indptr_kernel<<<(unsigned)g, 256, 0, st>>>(a.N, a.G, a.indptr);
        count_launch();
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    if (a.nrows == 0 || a.G == 0) return cudaSuccess;
    size_t smem;
    uint64_t g;
    const bool aligned = ((uintptr_t)a.indices % 16u) == 0 && ((uintptr_t)a.data % 16u) == 0;
    if (a.G <= (uint64_t)kCsrThreads) {
        const int L = csr_lut_bits((uint32_t)a.G);
        g = (a.nrows + (1u << L) - 1) >> L;
        smem = (((size_t)a.G * ((1u << L) + 1) + 3u) & ~(size_t)3u) * sizeof(int32_t);
        if (a.nctab <= kCsrSmemCtab) smem += (size_t)a.nctab * sizeof(double2);
        // staged path: every bulk store a whole number of 16-byte units
        // (even row counts) from 16-byte aligned outputs
        if (aligned && L >= 1 && a.nrows % 2 == 0) {
            const CsrStage cs = csr_stage((uint32_t)a.G, a.n, a.nctab, a.fvals ? a.nfold : 0u);
            const uint64_t nchunk = (a.nrows + (1u << cs.L) - 1) >> cs.L;
            const uint32_t q = csr_unit_chunks((uint32_t)a.G, cs.L, nchunk, nsm);
            g = (nchunk + q - 1) / q;
            if (g > 0x7fffffffull) return cudaErrorInvalidValue;
            const size_t sm = cs.total;
            const bool wide = a.n > 32 || a.wide;
            auto kern = a.inline_fold ? (wide ? csr_fill_staged_kernel<true, 1> : csr_fill_staged_kernel<false, 1>)
                        : a.fvals && a.nfold
                            ? (wide ? csr_fill_staged_kernel<true, 2> : csr_fill_staged_kernel<false, 2>)
                            : (wide ? csr_fill_staged_kernel<true, 0> : csr_fill_staged_kernel<false, 0>);
            cudaError_t e0 =
                cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
            if (e0 != cudaSuccess) return e0;
            if (a.fvals) {  // fold values first; the staged pass places them
                cudaError_t e = launch_csr_fold(a, nsm, st);
                if (e != cudaSuccess) return e;
            }
            kern<<<(unsigned)g, kCsrStageThreads, sm, st>>>(a, q);
            count_launch();
            cudaError_t e = cudaGetLastError();
            if (e != cudaSuccess || a.fvals || a.inline_fold) return e;
            return launch_csr_fold(a, nsm, st);
        }
    } else {
        g = a.nrows;
        const uint64_t nsig = a.G * (uint64_t)a.n;
        smem = nsig <= kCsrSmemSig ? (size_t)nsig * sizeof(int32_t) : 0;
    }
    auto kern = (a.n > 32 || a.wide) ? csr_fill_kernel<true> : csr_fill_kernel<false>;
    cudaError_t e0 = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)(kCsrLutBytes + kCsrSmemCtab * sizeof(double2)) + 64);
    if (e0 != cudaSuccess) return e0;
    // one wave of resident blocks striding the row chunks (no partial second wave)
    int per_sm = 0;
    e0 = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kCsrThreads, smem);
    if (e0 != cudaSuccess) return e0;
    if (per_sm < 1) per_sm = 1;
    if (g > (uint64_t)nsm * per_sm) g = (uint64_t)nsm * per_sm;
    kern<<<(unsigned)g, kCsrThreads, smem, st>>>(a);
    count_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    CsrArgs b = a;
    b.fvals = nullptr;  // direct path: fold entries stored in place
    return launch_csr_fold(b, nsm, st);
}

// y = A v, complex128.  Replaces spmat_dot_densevec (qrusty/src/accel.rs:338-370).
// S lanes per row, U entries per lane in flight with the step's tail
// predicated; the lanes' sums meet in a butterfly.  What bounds it: the
// matrix, read once (24 bytes per entry: 78 % of the measured HBM copy rate
// on the chains n = 20 and 22), with the FP64 pipe next (two multiply-adds
// per real entry, the lanes' sum: 0.7 of the time).  Hence one accumulator per
// part, a sum in which half of the lanes take each part (n = 20: 180 us, 191
// with both parts in every lane) and few lanes per row, and 4 CTAs of 256 threads per
// SM (64 registers) rather than deeper steps: chain n = 22, 44 entries a row,
// steps of 2 / 3 / 4 / 5 / 6 entries 1,090 / 1,030 / 979 / 890 / 839 us (all
// four multiply-adds, 11 entries in flight: 1,436).
// Partial sum of row [j0, j1) over this lane's entries.
template <int S, int U>
__device__ __forceinline__ double2 spmv_lane(uint64_t j0, uint64_t j1, uint64_t ncols,
                                             const uint64_t *__restrict__ indices,
                                             const double2 *__restrict__ data,
                                             const double2 *__restrict__ v) {
    double sr = 0.0, si = 0.0;
    for (uint64_t j = j0 + (threadIdx.x & (S - 1)); j < j1; j += (uint64_t)U * S) {
        uint64_t c[U];
        double2 d[U], x[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {  // the matrix streams once: evict-first loads
            const bool ok = j + (uint64_t)u * S < j1;
            c[u] = ok ? __ldcs(indices + j + u * S) : ncols;
            d[u] = ok ? __ldcs(data + j + u * S) : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            x[u] = c[u] < ncols ? __ldg(v + c[u]) : make_double2(0.0, 0.0);
        // real (or imaginary) entries take 2 of the 4 multiply-adds, where the
        // gathered value is not infinite or NaN
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (c[u] >= ncols) continue;  // out-of-range columns (and the tail) are skipped
            const bool fin = max(exp_bits(x[u].x), exp_bits(x[u].y)) != 0x7ff00000u;
            if (fin && mag_bits(d[u].y) == 0) {
                sr = fma(d[u].x, x[u].x, sr);
                si = fma(d[u].x, x[u].y, si);
            } else if (fin && mag_bits(d[u].x) == 0) {
                sr = fma(-d[u].y, x[u].y, sr);
                si = fma(d[u].y, x[u].x, si);
            } else {
                sr = fma(d[u].x, x[u].x, fma(-d[u].y, x[u].y, sr));
                si = fma(d[u].x, x[u].y, fma(d[u].y, x[u].x, si));
            }
        }
    }
    return make_double2(sr, si);
}

template <int S, int U>
__device__ __forceinline__ void spmv_rows(uint64_t nrows, uint64_t ncols,
                                          const uint64_t *__restrict__ indptr,
                                          const uint64_t *__restrict__ indices,
                                          const double2 *__restrict__ data,
                                          const double2 *__restrict__ v, double2 *__restrict__ y) {
    const uint32_t sl = threadIdx.x & (S - 1);
    const uint64_t groups = (uint64_t)gridDim.x * (blockDim.x / S);
    for (uint64_t r = blockIdx.x * (uint64_t)(blockDim.x / S) + (threadIdx.x / S); r < nrows;
         r += groups) {
        const double2 q = spmv_lane<S, U>(indptr[r], indptr[r + 1], ncols, indices, data, v);
        const uint32_t mask = ((1u << S) - 1u) << (threadIdx.x & 31u & ~(S - 1u));
        // halves of the row's lanes take a part each (one addition a step, not two)
        const bool im = (sl & (S / 2)) != 0;
        double p = (im ? q.y : q.x) + __shfl_xor_sync(mask, im ? q.x : q.y, S / 2, S);
#pragma unroll
        for (int o = S / 4; o > 0; o >>= 1) p += __shfl_xor_sync(mask, p, o, S);
        if ((sl & (S / 2 - 1)) == 0) reinterpret_cast<double *>(y + r)[im ? 1 : 0] = p;
    }
}

// The same for matrices that hold more than real entries: the lanes of a warp
// take their steps together, and a step whose entries are all real takes two
// multiply-adds per entry, any other all four without a branch per entry
// (300,000 rows of 40 complex entries: 151 us with spmv_rows, 95 so).
template <int S, int U>
__device__ __forceinline__ void spmv_rows_mixed(uint64_t nrows, uint64_t ncols,
                                                const uint64_t *__restrict__ indptr,
                                                const uint64_t *__restrict__ indices,
                                                const double2 *__restrict__ data,
                                                const double2 *__restrict__ v,
                                                double2 *__restrict__ y) {
    constexpr uint32_t W = 32 / S;  // rows of a warp
    const uint32_t sl = threadIdx.x & (S - 1), wr = (threadIdx.x & 31u) / S;
    const uint64_t stride = (uint64_t)gridDim.x * (blockDim.x / 32) * W;
    for (uint64_t b = (blockIdx.x * (uint64_t)(blockDim.x / 32) + threadIdx.x / 32) * W; b < nrows;
         b += stride) {
        const uint64_t r = b + wr;
        const bool in = r < nrows;
        const uint64_t j0 = in ? indptr[r] : 0, j1 = in ? indptr[r + 1] : 0;
        double sr = 0.0, si = 0.0;
        for (uint64_t j = j0 + sl; __any_sync(0xffffffffu, j < j1); j += (uint64_t)U * S) {
            uint64_t c[U];
            double2 d[U], x[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const bool ok = j + (uint64_t)u * S < j1;
                c[u] = ok ? __ldcs(indices + j + u * S) : ncols;
                d[u] = ok ? __ldcs(data + j + u * S) : make_double2(0.0, 0.0);
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                x[u] = c[u] < ncols ? __ldg(v + c[u]) : make_double2(0.0, 0.0);
            bool real = true;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                // out-of-range columns (and the tail) are skipped
                if (c[u] >= ncols) d[u] = make_double2(0.0, 0.0);
                real = real && max(exp_bits(x[u].x), exp_bits(x[u].y)) != 0x7ff00000u &&
                       mag_bits(d[u].y) == 0;
            }
            if (__all_sync(0xffffffffu, real)) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    sr = fma(d[u].x, x[u].x, sr);
                    si = fma(d[u].x, x[u].y, si);
                }
            } else {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    sr = fma(d[u].x, x[u].x, fma(-d[u].y, x[u].y, sr));
                    si = fma(d[u].x, x[u].y, fma(d[u].y, x[u].x, si));
                }
            }
        }
        const bool im = (sl & (S / 2)) != 0;
        double p = (im ? si : sr) + __shfl_xor_sync(0xffffffffu, im ? sr : si, S / 2, S);
#pragma unroll
        for (int o = S / 4; o > 0; o >>= 1) p += __shfl_xor_sync(0xffffffffu, p, o, S);
        if (in && (sl & (S / 2 - 1)) == 0) reinterpret_cast<double *>(y + r)[im ? 1 : 0] = p;
    }
}

constexpr int kSpmvMaxStep = 6;  // entries per lane in flight, at most

// The step depth is chosen from the first row's length, so that equal steps
// cover it (every row of a Pauli-sum CSR holds G entries; any CSR is handled
// at any depth), and the loop from that row's entries, 32 at most: any loop
// gives the same sums, real matrices are 5-12 % faster in spmv_rows.
template <int S>
__global__ void __launch_bounds__(256, 4) csr_spmv_kernel(uint64_t nrows, uint64_t ncols,
                                                          const uint64_t *__restrict__ indptr,
                                                          const uint64_t *__restrict__ indices,
                                                          const double2 *__restrict__ data,
                                                          const double2 *__restrict__ v,
                                                          double2 *__restrict__ y) {
    const uint64_t e = indptr[0] + (threadIdx.x & 31u);
    const bool mixed =
        __any_sync(0xffffffffu, e < indptr[1] && mag_bits(__ldg(data + e).y) != 0);
    const uint64_t want = (indptr[1] - indptr[0] + S - 1) / S;
    const uint64_t steps = (want + kSpmvMaxStep - 1) / kSpmvMaxStep;
    const int u = want < 1 ? 1 : (int)((want + steps - 1) / steps);
#define QR_SPMV_CASES(F)                                                                     \
    switch (u) {                                                                             \
        case 1: F<S, 1>(nrows, ncols, indptr, indices, data, v, y); break;                   \
        case 2: F<S, 2>(nrows, ncols, indptr, indices, data, v, y); break;                   \
        case 3: F<S, 3>(nrows, ncols, indptr, indices, data, v, y); break;                   \
        case 4: F<S, 4>(nrows, ncols, indptr, indices, data, v, y); break;                   \
        case 5: F<S, 5>(nrows, ncols, indptr, indices, data, v, y); break;                   \
        default: F<S, kSpmvMaxStep>(nrows, ncols, indptr, indices, data, v, y); break;       \
    }
    if (mixed) {
        QR_SPMV_CASES(spmv_rows_mixed)
    } else {
        QR_SPMV_CASES(spmv_rows)
    }
#undef QR_SPMV_CASES
}

cudaError_t launch_csr_spmv(uint64_t nrows, uint64_t ncols, const uint64_t *indptr,
                            const uint64_t *indices, const double *data, const double *v,
                            double *y, int nsm, cudaStream_t st) {
    if (nrows == 0) return cudaSuccess;
    // no host read of nnz or row lengths: the call stays asynchronous.
    // Sixteen lanes per row while the rows are too few to fill the SMs (2^12
    // rows of 176 entries: 14.5 us against 20.8 with four); four from 2^14
    // rows on, where a wider butterfly's additions cost more than it brings
    // (2^14 rows of 92: 26.8 against 29.0; 2^20 of 40: 188 against 439)
    const int lanes = nrows < (1ull << 14) ? 16 : 4;
    const uint64_t rows_per_block = 256 / (uint64_t)lanes;
    uint64_t g = (nrows + rows_per_block - 1) / rows_per_block;
    if (g > (uint64_t)nsm * 16) g = (uint64_t)nsm * 16;
    auto kern = lanes == 16 ? csr_spmv_kernel<16> : csr_spmv_kernel<4>;
    kern<<<(unsigned)g, 256, 0, st>>>(nrows, ncols, indptr, indices,
                                      reinterpret_cast<const double2 *>(data),
                                      reinterpret_cast<const double2 *>(v),
                                      reinterpret_cast<double2 *>(y));
    count_launch();
    return cudaGetLastError();
}

}  // namespace qr
