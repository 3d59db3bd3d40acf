// qr_host.cu -- C ABI of libqrusty_gpu (declared in include/qrusty_gpu.h).
//
// Host half of the GB300 Pauli-operator hot path: validates the terms,
// computes c'_k in FP64, groups the terms by x mask, prepares the CSR and
// apply tables, owns the operator's device memory and launches the kernels
// of qr_csr.cu / qr_apply.cu.  No CPU fallback exists: every numeric result
// is computed on the GPU.
//
// Compiled with -ffp-contract=off: c'_k = m(phase) * c_k must round exactly
// as num-complex's (ar*br - ai*bi, ar*bi + ai*br) does in qrusty's
// make_params (qrusty/src/accel.rs:141-157).
#include <algorithm>
#include <atomic>
#include <cstdarg>
#include <cstddef>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "../../include/qrusty_gpu.h"
#include "qr_common.cuh"

namespace qr {

static std::atomic<uint64_t> g_launches{0};
void count_launch(uint64_t k) { g_launches.fetch_add(k, std::memory_order_relaxed); }

cudaError_t ensure_dyn_smem(const void *fn, size_t bytes) {
    static std::mutex mu;
    static std::map<std::pair<int, const void *>, size_t> set;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(mu);
    auto key = std::make_pair(dev, fn);
    auto it = set.find(key);
    if (it != set.end() && it->second >= bytes) return cudaSuccess;
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) set[key] = bytes;
    return e;
}

static thread_local std::string g_err;

static int fail(int code, const char *fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    g_err = buf;
    return code;
}
static int cuda_fail(cudaError_t e, const char *what) {
    return fail(QR_ECUDA, "%s: %s", what, cudaGetErrorString(e));
}
int set_error(int code, const char *msg) { return fail(code, "%s", msg); }

#define QR_CUDA(call, what)                          \
    do {                                             \
        cudaError_t e_ = (call);                     \
        if (e_ != cudaSuccess) return cuda_fail(e_, what); \
    } while (0)

struct cd {
    double re, im;
};

// Device buffer with RAII release.
// Device buffer that keeps its allocation when refilled with no more bytes
// than it holds (plan rebuilds after a coefficient update reuse it instead of
// a cudaFree / cudaMalloc pair, which would synchronise the device).
struct DevBuf {
    void *p = nullptr;
    size_t bytes = 0, cap = 0;
    DevBuf() = default;
    DevBuf(const DevBuf &) = delete;
    DevBuf &operator=(const DevBuf &) = delete;
    ~DevBuf() { release(); }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        bytes = cap = 0;
    }
    cudaError_t alloc(size_t b) {
        if (b == 0) b = 16;
        if (p && b <= cap) {
            bytes = b;
            return cudaSuccess;
        }
        release();
        cudaError_t e = cudaMalloc(&p, b);
        if (e == cudaSuccess) bytes = cap = b;
        else p = nullptr;
        return e;
    }
    template <typename T>
    cudaError_t upload(const std::vector<T> &v) {
        cudaError_t e = alloc(v.size() * sizeof(T));
        if (e != cudaSuccess) return e;
        if (!v.empty()) e = cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
        return e;
    }
    template <typename T>
    T *as() const { return static_cast<T *>(p); }
};

struct Plan {
    bool built = false;
    int b = 0, tb = 0, threads = 0, amps = 0;
    uint32_t nblocks = 0;
    uint64_t nfat = 0;
    int diag_block = -1;
    bool has_diag = false;
    DevBuf blk_hi, diag;
    // qr_apply_rows.cu: complex128, and complex64 calls of few rows.  A
    // complex64 plan holds this form beside its tile form (strings, cosets or
    // per-tile tables) where both can be reached: a call of any number of
    // states finds its tables built and every coefficient update reaches them
    bool rows = false;
    uint32_t nrgroups = 0;
    size_t rtables = 0;  // byte offset of the factor tables behind the descriptors in groups
    DevBuf groups, fat_z, fat_c;
    // compensated-c64 kernel tables
    uint32_t nsub = 0, nruns = 0, nchunks = 0;
    DevBuf tdesc, tdata, blk_r0, run_g0, run_key, chunks;
    // string plans: see ApplyArgs; str.part[k - 1] are the parts of a split in k
    bool strings = false;
    StrSplit str;
    bool cosets = false;  // qr_apply_cosets.cu
    uint32_t ncblk = 0, ncsub = 0;
    DevBuf cblk, ctdesc, ctdata;
    DevBuf ent, sblk;
    // what the plan was built for, and its coefficient program: the slots
    // that qr_op_set_coeffs_device recomputes on the device, with the
    // diagonal's term list kept so that diag_wht can run again
    int dtype = 0, adjoint = 0;
    uint32_t nslots = 0;
    int ebits = 0;  // log2 of the entries of the program's widest slot
    DevBuf prog;            // its slots, their members and coordinates
    size_t prog_mem = 0, prog_coord = 0;  // byte offsets of those
    DevBuf dg;              // coefficients, z masks, bins' low masks and offsets, in turn
    size_t dg_tz = 0, dg_bz = 0, dg_boff = 0;
    uint32_t dg_nbins = 0;
    int dg_db = 0;
};

}  // namespace qr

using namespace qr;

struct qr_op {
    int n = 0;
    uint64_t N = 0, T = 0;
    int device = 0;
    int nsm = 0;
    // input terms on the device: masks, phases and the last coefficients
    // (input order); every table below is derived from them on the device
    DevBuf d_x, d_z, d_ph, d_coef;
    // grouping on the device (qr_group.cu): CSR order and the ascending x
    // groups, the merged strings (FP64 simplification, first-occurrence
    // order) with each one's input terms, the apply plan's x-groups
    uint64_t G = 0, M = 0, Ga = 0;
    DevBuf d_order, d_tz, d_gx, d_goff, d_mmap, d_mm_off, d_mm_terms, d_mx, d_mz, d_madj;
    DevBuf d_ag_off, d_ag_mem, d_mc;
    // host copies of the grouping, read by the apply plan builder and the
    // operator diagonal; mc is refetched from d_mc while host_coef_stale
    std::vector<uint64_t> gx, mx, mz;
    std::vector<uint32_t> goff, ag_off, ag_mem;
    std::vector<cd> mc;
    bool host_coef_stale = false;
    // CSR tables, built on the device on first use; their coefficient parts
    // follow every coefficient update on the device
    bool csr_ready = false;
    uint32_t nfold = 0, nctab = 0, fold_rem = 0;
    size_t csr_tables = 0;  // byte offset of the staged fill's tables in d_sig
    DevBuf d_tc, d_pmask, d_sig, d_grp, d_coord, d_ctab, d_fold, d_pbeta, d_ptab, d_fv;
    // term-gradient strings (see GradPlanArgs) per dtype, built on first use
    struct GradPlan {
        bool ready = false;
        uint32_t ndirect = 0, nbatch = 0, nwht = 0, nwbatch = 0;
        DevBuf x, z, perm, bat, wz, wperm, wbat;
    } tg[2];
    DevBuf expect_y;                    // H psi buffer of qr_expect
    Plan plans[2][2];  // [dtype][adjoint]
    Plan bplans[13];   // compensated-c64 plans with an explicit tile width (batched launches)
    DevBuf d_err;
    // host-call staging
    cudaStream_t hstream = nullptr;
    cudaStream_t cstream = nullptr;  // host-call copies of states 1.. (overlap)
    cudaEvent_t cev = nullptr;
    DevBuf stage_in, stage_out;
    // bumped by every host coefficient update: a qr_batch built on this
    // operator compares it with the value it recorded and rebuilds when they
    // differ (device updates rewrite the built tables in place instead)
    uint64_t coef_gen = 0;
    // test hooks (qr_op_set_test_hooks): mbarrier wait bound (0 = default),
    // withheld ring step (-1 = none), 64-bit row words forced
    uint64_t test_wait_ns = 0;
    int64_t test_withhold = -1;
    int test_wide = 0;
};

namespace {

struct Span {
    std::vector<uint64_t> basis;
    std::vector<uint64_t> coord;  // per term
    bool overflow = false;
    size_t used = 0;  // leading terms whose coordinates are set (all, without overflow)
};
Span gf2_span(const std::vector<uint64_t> &zs, size_t dmax);

// ---------------------------------------------------------------- coefficients
// After a device coefficient update the host copy of the merged coefficients
// is older than d_mc: fetch it (synchronous) before a plan is built.
int sync_host_coeffs(qr_op *op) {
    if (!op->host_coef_stale) return QR_OK;
    // the update ran on the caller's stream, which may not be ordered with
    // the legacy stream: wait for the device
    QR_CUDA(cudaDeviceSynchronize(), "fetch merged coefficients: sync");
    op->mc.resize(op->M);
    QR_CUDA(cudaMemcpy(op->mc.data(), op->d_mc.p, op->M * sizeof(cd), cudaMemcpyDeviceToHost),
            "fetch merged coefficients");
    op->host_coef_stale = false;
    return QR_OK;
}

// Coefficient-dependent CSR tables from d_coef, on stream st.
int refresh_csr_values(qr_op *op, cudaStream_t st) {
    QR_CUDA(csr_values(op->G, op->T, op->d_order.as<uint32_t>(), op->d_coef.as<double2>(),
                       op->d_ph.as<uint8_t>(), op->d_tc.as<double2>(), op->d_grp.as<CsrGroup>(),
                       op->d_coord.as<uint16_t>(), op->d_ctab.as<double2>(),
                       op->d_ptab.as<double2>(), op->nfold > 0, st),
            "CSR coefficient tables");
    return QR_OK;
}

// The operator's CSR tables as kernel arguments (no rows, no outputs yet).
CsrArgs csr_args(qr_op *op) {
    CsrArgs a{};
    a.N = op->N;
    a.G = op->G;
    a.gx = op->d_gx.as<uint64_t>();
    a.n = op->n;
    a.grp = op->d_grp.as<CsrGroup>();
    a.pmask = op->d_pmask.as<uint64_t>();
    a.sig = op->d_sig.as<int32_t>();
    a.tables = reinterpret_cast<const uint16_t *>(op->d_sig.as<unsigned char>() + op->csr_tables);
    a.fold = op->d_fold.as<uint32_t>();
    a.nfold = op->nfold;
    a.ctab = op->d_ctab.as<double2>();
    a.pbeta = op->d_pbeta.as<uint64_t>();
    a.ptab = op->d_ptab.as<double2>();
    a.nctab = op->nctab;
    a.tz = op->d_tz.as<uint64_t>();
    a.tc = op->d_tc.as<double>();
    a.err = op->d_err.as<int>();
    a.wide = op->test_wide;
    a.inline_fold = csr_inline_fold(op->G, op->n, op->nfold, op->fold_rem) ? 1 : 0;
    return a;
}

// CSR tables on the device, once per operator (qr_group.cu): the position
// trie, group spans and descriptors, then the coefficient parts.
int upload_csr_tables(qr_op *op) {
    if (op->csr_ready) return QR_OK;
    // d_coef may have been written on another stream
    QR_CUDA(cudaDeviceSynchronize(), "CSR tables: sync");
    const uint64_t G = op->G, T = op->T;
    QR_CUDA(op->d_pmask.alloc(G * sizeof(uint64_t)), "alloc position masks");
    // position terms by bit, then the staged fill's tables (16-byte aligned)
    op->csr_tables = (G * op->n * sizeof(int32_t) + 15u) & ~(size_t)15u;
    QR_CUDA(op->d_sig.alloc(op->csr_tables + csr_tables_bytes(G, op->n)), "alloc position tables");
    QR_CUDA(op->d_grp.alloc(G * sizeof(CsrGroup)), "alloc group descriptors");
    QR_CUDA(op->d_coord.alloc(T * sizeof(uint16_t)), "alloc span coordinates");
    QR_CUDA(op->d_fold.alloc(G * sizeof(uint32_t)), "alloc fold groups");
    QR_CUDA(op->d_pbeta.alloc(G * kCsrPrefixRank * sizeof(uint64_t)), "alloc prefix bases");
    QR_CUDA(op->d_tc.alloc(T * sizeof(cd)), "alloc CSR coefficients");
    CsrStructOut o{op->d_pmask.as<uint64_t>(), op->d_sig.as<int32_t>(), op->d_grp.as<CsrGroup>(),
                   op->d_coord.as<uint16_t>(), op->d_fold.as<uint32_t>(),
                   op->d_pbeta.as<uint64_t>()};
    CsrStructCounts cnt;
    QR_CUDA(csr_structure(op->n, G, op->d_gx.as<uint64_t>(), op->d_goff.as<uint32_t>(),
                          op->d_tz.as<uint64_t>(), o, &cnt, nullptr),
            "CSR tables");
    if (cnt.nctab > 0xffffffffull || cnt.nptab > 0xffffffffull)
        return fail(QR_EINVAL, "qr_csr_build: class tables too large");
    QR_CUDA(op->d_ctab.alloc(cnt.nctab * sizeof(cd)), "alloc class tables");
    QR_CUDA(op->d_ptab.alloc(cnt.nptab * sizeof(cd)), "alloc prefix tables");
    op->nctab = (uint32_t)cnt.nctab;
    op->nfold = cnt.nfold;
    op->fold_rem = cnt.fold_rem;
    QR_CUDA(launch_csr_tables(csr_args(op), nullptr), "CSR row-bit tables");
    int rc = refresh_csr_values(op, nullptr);
    if (rc) return rc;
    QR_CUDA(cudaStreamSynchronize(nullptr), "CSR tables: sync");
    op->csr_ready = true;
    return QR_OK;
}

// GF(2) span of the z differences of one group: basis (pivot = msb, unique)
// and the coordinates of every term's difference in that basis.
Span gf2_span(const std::vector<uint64_t> &zs, size_t dmax) {
    Span sp;
    const uint64_t z0 = zs[0];
    sp.coord.resize(zs.size());
    uint8_t ord[64];  // basis indices by descending pivot; the basis itself in order of insertion
    for (size_t k = 0; k < zs.size(); ++k) {
        uint64_t v = zs[k] ^ z0;
        uint64_t c = 0;
        for (size_t j = 0; j < sp.basis.size(); ++j) {
            const size_t i = ord[j];
            const uint64_t bv = sp.basis[i];
            const int piv = 63 - __builtin_clzll(bv);
            if ((v >> piv) & 1ull) {
                v ^= bv;
                c |= 1ull << i;
            }
        }
        if (v != 0) {
            if (sp.basis.size() >= dmax) {
                sp.overflow = true;
                sp.used = k;
                return sp;
            }
            size_t j = sp.basis.size();
            c |= 1ull << j;
            for (; j > 0 && sp.basis[ord[j - 1]] < v; --j) ord[j] = ord[j - 1];
            ord[j] = (uint8_t)sp.basis.size();
            sp.basis.push_back(v);
        }
        sp.coord[k] = c;
    }
    sp.used = zs.size();
    return sp;
}

// One sub-group of a per-tile-table plan: merged strings sharing x and z on
// the register bits, their z differences of rank <= 2, with their FP64 table.
struct SubGroup {
    uint64_t hi = 0;       // partner-tile XOR (x >> b)
    uint32_t lo = 0;       // x & (tile - 1)
    uint32_t zm = 0;       // z bits on the register bits
    uint64_t z0 = 0;
    uint64_t b0 = 0, b1 = 0;
    uint32_t d = 0;        // rank
    cd table[4];           // 2^d entries
    // merged strings of the sub-group in fold order, each with its coordinate
    // in the span basis (table entry u adds it with sign (-1)^popc(u & coord))
    std::vector<uint32_t> mem;
    std::vector<uint8_t> coord;
};

// Group descriptors and tables of a rows plan (qr_apply_rows.cu), x groups by
// x >> 12 in first-occurrence order.  A z span of rank > 4 is folded term by
// term per row in complex128; in complex64 the group is split until every
// piece has rank <= 4, so that all factors are FP64 sums rounded once.
template <typename Real, typename AddSlot>
int build_rows(qr_op *op, Plan &pl, const std::vector<cd> &c, const std::vector<uint64_t> &gxs,
               const std::vector<std::vector<size_t>> &members, bool skip_zero,
               AddSlot &&add_slot) {
    constexpr bool f32 = sizeof(Real) == 4;
    std::vector<size_t> ord(gxs.size());
    for (size_t g = 0; g < ord.size(); ++g) ord[g] = g;
    std::stable_sort(ord.begin(), ord.end(),
                     [&](size_t a, size_t b) { return (gxs[a] >> 12) < (gxs[b] >> 12); });
    std::vector<GroupDesc> descs;
    std::vector<Cplx<Real>> tab, fc;
    std::vector<uint64_t> fz;
    // strings of the descriptors in turn and their coordinates, for the
    // coefficient program
    std::vector<uint32_t> mem, first;
    std::vector<uint8_t> coord;
    auto masks = [&](const std::vector<size_t> &part) {
        std::vector<uint64_t> zs;
        zs.reserve(part.size());
        for (size_t k : part) zs.push_back(op->mz[k]);
        return zs;
    };
    auto cplx = [](cd v) { return Cplx<Real>{(Real)v.re, (Real)v.im}; };
    auto push = [&](uint64_t x, const std::vector<size_t> &part, const Span &sp, bool fat) {
        GroupDesc d;
        memset(&d, 0, sizeof(d));
        d.z0 = op->mz[part[0]];
        d.x = x;
        first.push_back((uint32_t)mem.size());
        for (size_t kk = 0; kk < part.size(); ++kk) {
            mem.push_back((uint32_t)part[kk]);
            coord.push_back(fat || sp.coord.empty() ? 0 : (uint8_t)sp.coord[kk]);
        }
        if (fat) {
            d.d = kFat;
            d.off = (uint32_t)fz.size();
            d.cnt = (uint32_t)part.size();
            for (size_t k : part) {
                fz.push_back(op->mz[k]);
                fc.push_back(cplx(c[k]));
            }
            pl.nfat++;
        } else {
            d.d = (uint32_t)sp.basis.size();
            d.off = (uint32_t)tab.size();
            for (size_t i = 0; i < sp.basis.size(); ++i) d.beta[i] = sp.basis[i];
            for (uint32_t u = 0; u < 1u << d.d; ++u) {
                cd acc{0.0, 0.0};
                for (size_t kk = 0; kk < part.size(); ++kk) {
                    const cd v = c[part[kk]];
                    if (__builtin_popcountll(u & coord[first.back() + kk]) & 1) {
                        acc.re -= v.re;
                        acc.im -= v.im;
                    } else {
                        acc.re += v.re;
                        acc.im += v.im;
                    }
                }
                tab.push_back(cplx(acc));
            }
        }
        descs.push_back(d);
    };
    const Span one;  // a single string: rank 0
    for (size_t g : ord) {
        if (skip_zero && gxs[g] == 0) continue;
        if (members[g].size() == 1) {
            push(gxs[g], members[g], one, false);
            continue;
        }
        const std::vector<uint64_t> zs = masks(members[g]);
        const Span sp = gf2_span(zs, kDMax);
        if (!sp.overflow || !f32) {
            push(gxs[g], members[g], sp, sp.overflow);
            continue;
        }
        const Span full = gf2_span(zs, 64);
        std::map<uint64_t, std::vector<size_t>> parts;
        for (size_t kk = 0; kk < members[g].size(); ++kk)
            parts[full.coord[kk] >> kDMax].push_back(members[g][kk]);
        for (const auto &pt : parts) push(gxs[g], pt.second, gf2_span(masks(pt.second), kDMax), false);
    }
    first.push_back((uint32_t)mem.size());
    pl.nrgroups = (uint32_t)descs.size();
    if (descs.empty()) descs.push_back(GroupDesc{});  // keep a valid pointer
    pl.rtables = descs.size() * sizeof(GroupDesc);
    std::vector<unsigned char> img(pl.rtables + tab.size() * sizeof(Cplx<Real>));
    memcpy(img.data(), descs.data(), pl.rtables);
    if (!tab.empty()) memcpy(img.data() + pl.rtables, tab.data(), img.size() - pl.rtables);
    QR_CUDA(pl.groups.upload(img), "upload groups and tables");
    if constexpr (!f32) {
        QR_CUDA(pl.fat_z.upload(fz), "upload fat z");
        QR_CUDA(pl.fat_c.upload(fc), "upload fat c");
    }
    for (size_t i = 0; i + 1 < first.size(); ++i) {
        const GroupDesc &d = descs[i];
        const uint32_t m0 = first[i], cnt = first[i + 1] - m0;
        if (d.d != kFat) {
            if (cnt > 0xffff) return fail(QR_EINVAL, "plan: group too large");
            add_slot((uint64_t)pl.groups.p + pl.rtables + (uint64_t)d.off * sizeof(Cplx<Real>),
                     &mem[m0], &coord[m0], cnt, d.d, f32 ? 0 : 1);
        } else {
            for (uint32_t kk = 0; kk < cnt; ++kk)
                add_slot((uint64_t)pl.fat_c.p + (uint64_t)(d.off + kk) * sizeof(Cplx<Real>),
                         &mem[m0 + kk], nullptr, 1, 0, 2);
        }
    }
    return QR_OK;
}

// Entry lists of a string plan (qr_apply_strings.cu): the merged strings
// outside the diagonal by partner tile, in blocks, and the parts of about
// equal work that the CTAs of a cluster of 1 ... kStrMaxSplit take.
template <typename AddSlot>
int build_strings(qr_op *op, Plan &pl, const std::vector<cd> &c,
                  const std::vector<size_t> &diag_terms, AddSlot &&add_slot) {
    const size_t M = op->mx.size();
    std::vector<char> diag(M, 0);
    for (size_t k : diag_terms) diag[k] = 1;
    std::vector<uint32_t> ord;
    for (size_t k = 0; k < M; ++k)
        if (!diag[k]) ord.push_back((uint32_t)k);
    std::stable_sort(ord.begin(), ord.end(), [&](uint32_t a, uint32_t b) {
        return (op->mx[a] >> 12) < (op->mx[b] >> 12);
    });
    StrSplit &sp = pl.str;
    sp.nstr = (uint32_t)ord.size();
    // states of 2^19 amplitudes and more fill the SMs with whole tiles: two
    // partner tiles per block halve the ring's bookkeeping.  Below, tiles are
    // split over clusters and a block holds at most a 32nd of the strings, so
    // that parts balance
    sp.tpb = op->n >= kStrPairN ? 2 : 1;
    const uint32_t cap =
        sp.tpb > 1 ? kStrEntCap
                   : std::min(kStrEntCap, std::max(16u, (sp.nstr + 31u) / 32u));
    std::vector<uint4> ent, blk;
    std::vector<uint32_t> mem;  // entry -> merged string (0xffffffff: header)
    auto open = [&](uint64_t hi, bool dg) {
        blk.push_back(make_uint4((uint32_t)hi, 0xffffffffu, (uint32_t)ent.size(), 0));
        ent.push_back(make_uint4(0, dg ? 1u : 0u, 0, 0));
        mem.push_back(0xffffffffu);
    };
    bool has_diag = !diag_terms.empty();
    if (has_diag && (ord.empty() || (op->mx[ord[0]] >> 12) != 0)) {
        open(0, true);
        has_diag = false;
    }
    for (size_t i = 0; i < ord.size(); ++i) {
        const uint64_t x = op->mx[ord[i]], z = op->mz[ord[i]], h = x >> 12;
        if (i == 0 || (op->mx[ord[i - 1]] >> 12) != h || blk.back().w >= cap) {
            // a tile's strings stay together where they fit a block
            size_t j = i;
            while (j < ord.size() && (op->mx[ord[j]] >> 12) == h && j - i < cap) ++j;
            if (sp.tpb > 1 && !blk.empty() && blk.back().y == 0xffffffffu &&
                blk.back().x != (uint32_t)h && blk.back().w + (j - i) <= cap) {
                blk.back().y = (uint32_t)h;
            } else {
                open(h, has_diag && h == 0);
                if (h == 0) has_diag = false;
            }
        }
        uint4 &bl = blk.back();
        ++bl.w;
        ++ent[bl.z].x;
        const uint32_t half = bl.x != (uint32_t)h ? 1u : 0u;
        const uint32_t w = (uint32_t)(x & 1u) | ((uint32_t)(x >> 1) & 511u) << 4 |
                           ((uint32_t)(x >> 10) & 3u) << 13 | half << 15 | (uint32_t)(z & 1u) << 16 |
                           ((uint32_t)(z >> 10) & 3u) << 17 | (uint32_t)(z >> 32) << 24;
        const float fr = (float)c[ord[i]].re, fi = (float)c[ord[i]].im;
        uint32_t br, bi;
        memcpy(&br, &fr, 4);
        memcpy(&bi, &fi, 4);
        ent.push_back(make_uint4(w, (uint32_t)z & ~0xc01u, br, bi));
        mem.push_back(ord[i]);
    }
    // a block costs about two strings beside its own
    std::vector<uint64_t> upto(blk.size() + 1, 0);
    for (size_t j = 0; j < blk.size(); ++j) upto[j + 1] = upto[j] + 2 + blk[j].w;
    for (uint32_t k = 1; k <= kStrMaxSplit; ++k) {
        uint32_t *part = sp.part[k - 1];
        uint32_t j = 0;
        part[0] = 0;
        for (uint32_t r = 1; r <= k; ++r) {
            const uint64_t end = upto.back() * r / k;
            // the boundary nearest to the r-th share
            while (j < blk.size() && upto[j + 1] + upto[j] <= 2 * end) ++j;
            if (r == k) j = (uint32_t)blk.size();
            part[r] = j;
        }
    }
    sp.nblk = (uint32_t)blk.size();
    QR_CUDA(pl.ent.upload(ent), "upload string entries");
    QR_CUDA(pl.sblk.upload(blk), "upload string blocks");
    for (size_t i = 0; i < mem.size(); ++i)
        if (mem[i] != 0xffffffffu)
            add_slot((uint64_t)pl.ent.p + i * sizeof(uint4) + 8, &mem[i], nullptr, 1, 0, 0);
    return QR_OK;
}

// Sub-groups of a coset plan (qr_apply_cosets.cu), blocks and tables; *fits is
// false, and nothing is made, when they do not fit the kernel's shared memory.
//
// A thread's rows are t' + 512 m, t' = t ^ 256 for odd popc(m): the coset of
// the even-weight subsets of row bits 8 ... 11.  Within a tile, x = (xt, xm),
// xm its bits 9-11, moves the coset by c = xt ^ (256 for odd popc(xm)) and m by
// xm; a string's sign is (-1)^(popc(t & z) + popc(m & zm)), zm = its bits 9-11,
// complemented when bit 8 is set.  A sub-group holds the strings of one x with
// one zm, their z differences (bits 9-11 aside) of rank <= 2.
template <typename AddSlot>
int build_cosets(qr_op *op, Plan &pl, const std::vector<cd> &c, const std::vector<uint64_t> &gxs,
                 const std::vector<std::vector<size_t>> &members, bool has_diag, bool *fits,
                 AddSlot &&add_slot) {
    struct Sub {
        uint64_t hi, x;
        uint32_t off, xm, zm;
        uint64_t z0;
        Span sp;
        std::vector<size_t> part;
    };
    auto zm_of = [&](size_t k) {
        const uint32_t z = (uint32_t)(op->mz[k] >> 8) & 15u;
        return (z >> 1) ^ ((z & 1u) ? 7u : 0u);
    };
    auto masked = [&](const std::vector<size_t> &part) {
        std::vector<uint64_t> zs;
        for (size_t k : part) zs.push_back(op->mz[k] & ~0xe00ull);
        return zs;
    };
    std::vector<Sub> subs;
    std::vector<size_t> byzm[8];
    for (size_t g = 0; g < gxs.size(); ++g) {
        if (has_diag && gxs[g] == 0) continue;
        const uint32_t lo = (uint32_t)(gxs[g] & 4095u), xm = lo >> 9;
        const uint32_t off = ((lo & 511u) ^ ((__builtin_popcount(xm) & 1) ? 256u : 0u)) << 3;
        auto push = [&](uint32_t zm, std::vector<size_t> part, Span sp) {
            Sub sg;
            sg.hi = gxs[g] >> 12;
            sg.x = gxs[g];
            sg.off = off;
            sg.xm = xm;
            sg.zm = zm;
            sg.z0 = op->mz[part[0]] & ~0xe00ull;
            sg.sp = std::move(sp);
            sg.part = std::move(part);
            subs.push_back(std::move(sg));
        };
        for (auto &v : byzm) v.clear();
        for (size_t k : members[g]) byzm[zm_of(k)].push_back(k);
        for (uint32_t zm = 0; zm < 8; ++zm) {
            if (byzm[zm].empty()) continue;
            Span full = gf2_span(masked(byzm[zm]), 64);
            if (full.basis.size() <= 2) {
                push(zm, byzm[zm], std::move(full));
                continue;
            }
            std::map<uint64_t, std::vector<size_t>> parts;
            for (size_t kk = 0; kk < byzm[zm].size(); ++kk)
                parts[full.coord[kk] >> 2].push_back(byzm[zm][kk]);
            for (auto &pt : parts) {
                Span sp = gf2_span(masked(pt.second), 2);
                push(zm, std::move(pt.second), std::move(sp));
            }
        }
    }
    *fits = !subs.empty() && subs.size() <= (size_t)kTabCap;
    if (!*fits) return QR_OK;
    std::stable_sort(subs.begin(), subs.end(), [](const Sub &a, const Sub &b) {
        return a.hi != b.hi ? a.hi < b.hi : a.off < b.off;
    });
    // partner tiles and their sub-groups
    struct Tile {
        uint64_t hi;
        uint32_t g0, g1;
    };
    std::vector<Tile> tiles;
    if (has_diag && subs[0].hi != 0) tiles.push_back({0, 0, 0});
    for (uint32_t i = 0; i < subs.size(); ++i) {
        if (tiles.empty() || tiles.back().hi != subs[i].hi) tiles.push_back({subs[i].hi, i, i});
        tiles.back().g1 = i + 1;
    }
    // Tiles in pairs, heavy with heavy and light (one sub-group) with light, the
    // heavy pairs spread evenly among the light ones, each closing a run of
    // them: a ring of three pairs does not hide its refill behind a run of light
    // pairs, and the tile's last pair is heavy, so the ring refills across the
    // table rebuild.  The diagonal's tile is tile 0 of its pair.
    std::vector<uint32_t> heavy, light;
    for (uint32_t j = 0; j < tiles.size(); ++j)
        ((tiles[j].g1 - tiles[j].g0 > 1 || tiles[j].hi == 0) ? heavy : light).push_back(j);
    std::vector<std::pair<uint32_t, uint32_t>> hp, lp, seq;
    constexpr uint32_t none = 0xffffffffu;
    size_t l0 = 0;
    for (size_t i = 0; i < heavy.size(); i += 2) {
        if (i + 1 < heavy.size()) hp.push_back({heavy[i], heavy[i + 1]});
        else if (!light.empty()) hp.push_back({heavy[i], light[l0++]});
        else hp.push_back({heavy[i], none});
    }
    for (size_t i = l0; i < light.size(); i += 2)
        lp.push_back({light[i], i + 1 < light.size() ? light[i + 1] : none});
    size_t ih = 0, il = 0;
    const size_t tot = hp.size() + lp.size();
    for (size_t k = 0; k < tot; ++k) {
        if (ih < hp.size() && (il >= lp.size() || k >= (ih + 1) * tot / hp.size() - 1))
            seq.push_back(hp[ih++]);
        else seq.push_back(lp[il++]);
    }
    std::vector<uint4> blk, td;
    std::vector<TileDataC64> data;
    std::vector<const Sub *> placed;
    auto thread_var = [](const Sub &g) {
        uint64_t m = g.z0;
        for (uint64_t b : g.sp.basis) m |= b;
        return (m & 511u) != 0;
    };
    // role and masks of a merged pair: one table index and sign for both
    struct Merge {
        uint64_t role = 0;
        uint32_t b0t = 0, b1t = 0;
    };
    auto merge_of = [](const Sub &a, const Sub &b) {
        Merge m;
        auto bt = [](const Sub &s, size_t i) {
            return i < s.sp.basis.size() ? (uint32_t)s.sp.basis[i] & 511u : 0u;
        };
        const uint32_t mu = (uint32_t)(a.z0 ^ b.z0) & 511u;
        if (mu == 0 && bt(a, 0) == bt(b, 0) && bt(a, 1) == bt(b, 1) &&
            a.sp.basis.size() == b.sp.basis.size()) {
            m = {kMergedBasis, bt(a, 0), bt(a, 1)};
        } else if (a.sp.basis.size() <= 1 && b.sp.basis.size() <= 1 &&
                   (a.sp.basis.empty() || b.sp.basis.empty() || bt(a, 0) == bt(b, 0))) {
            m = {kMergedSign, bt(a.sp.basis.empty() ? b : a, 0), mu};
        }
        return m;
    };
    std::vector<uint32_t> rank;  // of placed, as its table is filled
    auto push = [&](const Sub &g, uint32_t half, bool load, uint32_t key, uint64_t role = 0,
                    Merge m = Merge()) {
        const uint64_t b0 = g.sp.basis.size() > 0 ? g.sp.basis[0] : 0,
                       b1 = g.sp.basis.size() > 1 ? g.sp.basis[1] : 0;
        const uint32_t b0t = m.role ? m.b0t : (uint32_t)b0 & 511u,
                       b1t = m.role ? m.b1t : (uint32_t)b1 & 511u;
        td.push_back(make_uint4(g.off | half << 15 | (load ? 1u << 16 : 0u) | key << 17 |
                                    (m.role && role != kMergedSecond ? 1u << 24 : 0u),
                                (uint32_t)g.z0 & 511u, b0t, b1t));
        TileDataC64 d;
        memset(&d, 0, sizeof(d));
        d.z0h = g.z0 >> 12;
        d.b0h = b0 >> 12;
        d.b1h = b1 >> 12;
        d.role = role;
        // a rank-0 table beside a rank-1 one repeats its entry
        const uint32_t rk = m.role == kMergedSign ? 1u : (uint32_t)g.sp.basis.size();
        for (uint32_t u = 0; u < 1u << rk; ++u) {
            cd acc{0.0, 0.0};
            for (size_t kk = 0; kk < g.part.size(); ++kk) {
                const cd v = c[g.part[kk]];
                if (__builtin_popcountll(u & g.sp.coord[kk]) & 1) {
                    acc.re -= v.re;
                    acc.im -= v.im;
                } else {
                    acc.re += v.re;
                    acc.im += v.im;
                }
            }
            d.T[u] = make_float2((float)acc.re, (float)acc.im);
        }
        data.push_back(d);
        placed.push_back(&g);
        rank.push_back(rk);
    };
    for (const auto &pr : seq) {
        struct Item {
            uint32_t first, half;  // coset: sub-groups [first, last)
            uint32_t last;
        };
        std::vector<Item> uniform, bythread, others;
        const uint32_t two[2] = {pr.first, pr.second};
        for (uint32_t h = 0; h < 2; ++h) {
            if (two[h] == none) continue;
            const Tile &tl = tiles[two[h]];
            for (uint32_t i = tl.g0; i < tl.g1;) {
                uint32_t j = i + 1;
                while (j < tl.g1 && subs[j].off == subs[i].off) ++j;
                const bool lone = j == i + 1 && subs[i].xm == 0 && subs[i].zm == 0;
                (lone ? (thread_var(subs[i]) ? bythread : uniform) : others).push_back({i, h, j});
                i = j;
            }
        }
        const uint32_t g0 = (uint32_t)td.size();
        for (const Item &it : uniform) push(subs[it.first], it.half, true, 0);
        for (const Item &it : bythread) push(subs[it.first], it.half, true, 0);
        // cosets of several: pairs of one x whose patterns differ by DL(xm); four
        // merged pairs with a Jordan-Wigner hop's patterns make a quad
        struct Placed {
            uint32_t a, b;  // sub-groups, b == none: alone
            uint32_t key;
            Merge m;
        };
        static const uint32_t quad_zm[4] = {0, 7, 6, 4};
        uint32_t nquad = 0;
        std::vector<std::pair<uint32_t, std::vector<Placed>>> rest;  // half, sub-groups
        for (const Item &it : others) {
            std::vector<char> used(it.last - it.first, 0);
            std::vector<Placed> out;
            for (uint32_t i = it.first; i < it.last; ++i) {
                if (used[i - it.first]) continue;
                const Sub &a = subs[i];
                const uint32_t f =
                    a.xm == 0 ? 0u : a.xm == 1 ? 1u : a.xm == 2 ? 2u : a.xm == 4 ? 3u : 4u;
                const uint32_t dl = f == 0 ? 7u : a.xm;
                uint32_t mate = none;
                for (uint32_t j = i + 1; j < it.last && f < 4 && mate == none; ++j)
                    if (!used[j - it.first] && subs[j].x == a.x && (subs[j].zm ^ a.zm) == dl)
                        mate = j;
                if (mate == none) {
                    out.push_back({i, none, a.xm | a.zm << 3, Merge()});
                    continue;
                }
                used[mate - it.first] = 1;
                uint32_t p0 = i, p1 = mate;
                if (subs[p1].zm == quad_zm[f]) std::swap(p0, p1);
                const Merge m = merge_of(subs[p0], subs[p1]);
                if (m.role == 0) {  // no common table: two sub-groups on one set of loads
                    out.push_back({i, none, a.xm | a.zm << 3, Merge()});
                    out.push_back({mate, none, a.xm | subs[mate].zm << 3, Merge()});
                } else {
                    out.push_back({p0, p1, 64u + (f | subs[p0].zm << 2), m});
                }
            }
            std::vector<Placed> q(4, Placed{none, none, 0, Merge()});
            bool quad = out.size() == 4 && nquad < 63;
            for (const Placed &o : out) {
                const uint32_t f = o.key & 3u;
                quad = quad && o.key >= 64u && q[f].a == none && subs[o.a].zm == quad_zm[f];
                if (quad) q[f] = o;
            }
            if (!quad) {
                rest.push_back({it.half, out});
                continue;
            }
            ++nquad;
            for (uint32_t f = 0; f < 4; ++f) {
                push(subs[q[f].a], it.half, f == 0, q[f].key, q[f].m.role, q[f].m);
                push(subs[q[f].b], it.half, false, 0, kMergedSecond, q[f].m);
            }
        }
        for (const auto &r : rest) {
            bool load = true;
            for (const Placed &o : r.second) {
                push(subs[o.a], r.first, load, o.key, o.m.role, o.m);
                if (o.b != none) push(subs[o.b], r.first, false, 0, kMergedSecond, o.m);
                load = false;
            }
        }
        const bool dg = has_diag && tiles[pr.first].hi == 0;
        const bool cheap = uniform.size() == 2 && bythread.empty() && others.empty() &&
                           uniform[0].half != uniform[1].half &&
                           subs[uniform[0].first].off == 0 && subs[uniform[1].first].off == 0;
        blk.push_back(make_uint4((uint32_t)tiles[pr.first].hi,
                                 pr.second == none ? none : (uint32_t)tiles[pr.second].hi,
                                 g0 | (uint32_t)uniform.size() << 10 | (cheap ? 1u << 30 : 0u) |
                                     (dg ? 1u << 31 : 0u),
                                 (uint32_t)bythread.size() | nquad << 10 |
                                     ((uint32_t)td.size() - g0 - (uint32_t)uniform.size() -
                                      (uint32_t)bythread.size() - 8 * nquad)
                                         << 16));
    }
    *fits = coset_smem_bytes((uint32_t)td.size(), (uint32_t)blk.size(), 2, 1) <=
            kCosetSmem;
    if (!*fits) return QR_OK;
    pl.ncblk = (uint32_t)blk.size();
    pl.ncsub = (uint32_t)td.size();
    QR_CUDA(pl.cblk.upload(blk), "upload coset blocks");
    QR_CUDA(pl.ctdesc.upload(td), "upload coset descriptors");
    QR_CUDA(pl.ctdata.upload(data), "upload coset tile data");
    for (size_t i = 0; i < placed.size(); ++i) {
        const Sub &g = *placed[i];
        if (g.part.size() > 0xffff) return fail(QR_EINVAL, "plan: sub-group too large");
        std::vector<uint32_t> mem(g.part.begin(), g.part.end());
        std::vector<uint8_t> coord(g.sp.coord.begin(), g.sp.coord.end());
        add_slot((uint64_t)pl.ctdata.p + i * sizeof(TileDataC64) + offsetof(TileDataC64, T),
                 mem.data(), coord.data(), mem.size(), rank[i], 0);
    }
    return QR_OK;
}

// Rows up to which a complex64 call runs over rows, by what it would run on
// otherwise: a tile kernel takes one SM per 4,096 rows.  Measured (us, tiles
// against rows).  String kernel, which splits a tile over a cluster, 2^14 rows:
// n = 12, 1,000 strings 33 / 29, 4,000 88 / 90, n = 13, 2,000 53 / 53, n = 14,
// 1,000 31 / 32, 5,000 128 / 121; 2^15: n = 12, 1,000 33 / 41, 2,000 51 / 76,
// n = 14, 5,000 128 / 194; 2^17: n = 12, 4,000 167 / 426; it takes 12 us at
// least, so few x groups run over more rows: 28 groups 2^17 12 / 8, 328 2^14
// 21 / 16, 2^15 22 / 23.  Cosets and per-tile tables, 2^17 rows: Jordan-Wigner of
// 92 x groups 25 / 25, 121 31 / 31, molecular sums of 286 173 / 127, 981 507 /
// 377, 1,941 900 / 597, chain 13 / 9; 2^18: 121 31 / 55, 286 174 / 235, 981 507 /
// 707, 1,941 901 / 1,108.  Below 12 qubits a tile is smaller and costs 0.05-0.1
// us per x group: n = 11, 500 groups, 52 against 12 (one state), even at
// 2^15-2^16 rows.
uint64_t c64_rows_limit(int n, bool strings, uint64_t groups) {
    // a tile of fewer than 32 rows is less than a warp, which the per-tile-table
    // kernel does not run on
    if (n < 5) return ~0ull;
    if (strings) return std::min(1ull << 17, std::max(1ull << 14, (1ull << 23) / groups));
    return n >= 12 ? 1ull << 17 : 1ull << 15;
}

// Whether a call of this many states runs over rows.
bool over_rows(const qr_op *op, const Plan &pl, int32_t call_states) {
    return pl.dtype == QR_C128 ||
           (pl.rows && op->N * (uint64_t)call_states <= c64_rows_limit(op->n, pl.strings, op->Ga));
}

// The plan's diagonal from its strings' coefficients on the device.
cudaError_t run_diag(const qr_op *op, const Plan &pl, cudaStream_t st) {
    const unsigned char *p = pl.dg.as<unsigned char>();
    return launch_diag(pl.dtype, op->n, pl.dg_db, op->N >> pl.dg_db,
                       reinterpret_cast<const uint64_t *>(p + pl.dg_bz),
                       reinterpret_cast<const uint32_t *>(p + pl.dg_boff), pl.dg_nbins,
                       reinterpret_cast<const uint64_t *>(p + pl.dg_tz),
                       reinterpret_cast<const double *>(p), pl.diag.p, st);
}

int build_plan(qr_op *op, int dtype, int adjoint, int tile_bits = -1) {
    Plan &pl = tile_bits >= 0 ? op->bplans[tile_bits] : op->plans[dtype][adjoint];
    if (pl.built) return QR_OK;
    {
        const int rc = sync_host_coeffs(op);
        if (rc) return rc;
    }
    pl.dtype = dtype;
    pl.adjoint = adjoint;
    // coefficient program (see CoefSlot): members packed per slot
    std::vector<CoefSlot> slots;
    std::vector<uint32_t> cmem;
    std::vector<uint8_t> ccoord;
    auto add_slot = [&](uint64_t dst, const uint32_t *mem, const uint8_t *coord, size_t cnt,
                        uint32_t d, uint8_t kind) {
        CoefSlot sl;
        sl.dst = dst;
        sl.m0 = (uint32_t)cmem.size();
        sl.cnt = (uint16_t)cnt;
        sl.d = (uint8_t)d;
        sl.kind = kind;
        for (size_t k = 0; k < cnt; ++k) {
            cmem.push_back(mem[k]);
            ccoord.push_back(coord ? coord[k] : 0);
        }
        slots.push_back(sl);
    };
    const int n = op->n;
    const bool f32 = dtype == QR_C64C;
    pl.b = tile_bits < 0 ? std::min(n, 12) : std::min(n, tile_bits);
    const int tmax = !f32 ? 512 : (1 << kC64ThreadBits);
    pl.threads = std::min(1 << pl.b, tmax);
    pl.amps = (1 << pl.b) / pl.threads;
    pl.tb = 0;
    while ((1 << pl.tb) < pl.threads) ++pl.tb;
    const uint64_t tmask = (1ull << pl.b) - 1;

    // coefficients of this plan (adjoint: conj(c) * (-1)^popc(x & z))
    const size_t M = op->mx.size();
    std::vector<cd> c(M);
    for (size_t k = 0; k < M; ++k) {
        c[k] = op->mc[k];
        if (adjoint) {
            c[k].im = -c[k].im;
            if (__builtin_popcountll(op->mx[k] & op->mz[k]) & 1) {
                c[k].re = -c[k].re;
                c[k].im = -c[k].im;
            }
        }
    }
    // x-groups of the merged strings in first-occurrence order (grouped on
    // the device at creation)
    std::vector<uint64_t> gxs(op->Ga);
    std::vector<std::vector<size_t>> members(op->Ga);
    for (size_t g = 0; g < op->Ga; ++g) {
        members[g].assign(op->ag_mem.begin() + op->ag_off[g], op->ag_mem.begin() + op->ag_off[g + 1]);
        gxs[g] = op->mx[members[g][0]];
    }
    // The compensated-c64 kernel keeps a sub-group's factor thread-constant
    // up to a Walsh sign over the register bits [tb, tb + log2 amps): split
    // each x-group by its terms' z bits there.  The c128 kernel does not split.
    int abits = 0;
    while ((1 << abits) < pl.amps) ++abits;
    const uint64_t mmask = f32 ? (((1ull << abits) - 1) << pl.tb) : 0;
    std::vector<size_t> diag_terms;
    // sub-groups: x group, strings (none listed: all of the group's)
    std::vector<std::pair<size_t, std::vector<size_t>>> pieces;
    for (size_t g = 0; g < gxs.size(); ++g) {
        if (gxs[g] == 0) {
            std::vector<uint64_t> zs;
            for (size_t k : members[g]) zs.push_back(op->mz[k]);
            if (gf2_span(zs, kDMax).overflow) {
                diag_terms = members[g];
                continue;
            }
        }
        if (!f32) continue;  // whole groups (build_rows)
        if (members[g].size() == 1) {
            pieces.emplace_back(g, std::vector<size_t>());
            continue;
        }
        std::vector<uint64_t> pkeys;
        std::vector<std::vector<size_t>> parts;
        for (size_t k : members[g]) {
            const uint64_t key = op->mz[k] & mmask;
            size_t pi = 0;
            while (pi < pkeys.size() && pkeys[pi] != key) ++pi;
            if (pi == pkeys.size()) {
                pkeys.push_back(key);
                parts.emplace_back();
            }
            parts[pi].push_back(k);
        }
        // split further until every sub-group has rank <= 2 (strings whose z
        // differences agree beyond the first two basis vectors)
        for (auto &part : parts) {
            std::vector<uint64_t> zs;
            for (size_t k : part) zs.push_back(op->mz[k]);
            Span full = gf2_span(zs, 64);
            if (full.basis.size() <= 2) {
                pieces.push_back({g, std::move(part)});
                continue;
            }
            std::vector<uint64_t> hk;
            std::vector<std::vector<size_t>> hp;
            for (size_t kk = 0; kk < part.size(); ++kk) {
                const uint64_t key = full.coord[kk] >> 2;
                size_t pi = 0;
                while (pi < hk.size() && hk[pi] != key) ++pi;
                if (pi == hk.size()) {
                    hk.push_back(key);
                    hp.emplace_back();
                }
                hp[pi].push_back(part[kk]);
            }
            for (auto &h : hp) pieces.push_back({g, std::move(h)});
        }
    }
    pl.has_diag = !diag_terms.empty();
    // One entry per string where an x group holds about one: a string costs
    // 0.6 of a sub-group of the per-tile table kernel (n = 20, 2,000 random
    // strings: 735 against 1,231 us) and, at up to 512 sub-groups, the coset
    // kernel is the better one from a third more strings than sub-groups on
    // (chain n = 22, 64 strings in 47: 111 against 93).
    const size_t nstr = M - diag_terms.size();
    const double most = (pieces.size() <= (size_t)kTabCap ? 1.3 : 1.6) * (double)pieces.size();
    pl.strings = f32 && tile_bits < 0 && n >= 12 && nstr > 0 && (double)nstr <= most;
    pl.rows = !f32 || (tile_bits < 0 && op->N <= c64_rows_limit(n, pl.strings, op->Ga));
    pl.nsub = (uint32_t)pieces.size();
    // partner tiles, one with more than kTabCap sub-groups (the per-tile table's
    // size) visited as several consecutive blocks
    std::vector<uint64_t> his;
    for (const auto &pc : pieces) his.push_back(gxs[pc.first] >> pl.b);
    std::sort(his.begin(), his.end());
    std::vector<uint64_t> bhi;
    std::vector<uint32_t> bg0;
    if (pl.has_diag && (his.empty() || his[0] != 0)) {
        bhi.push_back(0);
        bg0.push_back(0);
    }
    for (size_t i = 0; i < his.size(); ++i)
        if (i == 0 || his[i] != his[i - 1] || i - bg0.back() == (size_t)kTabCap) {
            bhi.push_back(his[i]);
            bg0.push_back((uint32_t)i);
        }
    bg0.push_back((uint32_t)his.size());
    pl.nblocks = (uint32_t)bhi.size();

    pl.nfat = 0;
    if (pl.rows) {
        const int rc = f32 ? build_rows<float>(op, pl, c, gxs, members, pl.has_diag, add_slot)
                           : build_rows<double>(op, pl, c, gxs, members, pl.has_diag, add_slot);
        if (rc) return rc;
    }
    if (pl.strings) {
        const int rc = build_strings(op, pl, c, diag_terms, add_slot);
        if (rc) return rc;
    }
    pl.cosets = false;
    if (f32 && !pl.strings && tile_bits < 0 && n >= 12) {
        const int rc = build_cosets(op, pl, c, gxs, members, pl.has_diag, &pl.cosets, add_slot);
        if (rc) return rc;
    }
    if (f32 && !pl.strings && !pl.cosets) {
        // per-tile-table kernel arrays
        pl.diag_block = -1;
        for (size_t j = 0; j < bhi.size() && pl.diag_block < 0; ++j)
            if (bhi[j] == 0) pl.diag_block = (int)j;
        std::vector<SubGroup> subs;
        for (const auto &pc : pieces) {
            const std::vector<size_t> &part = pc.second.empty() ? members[pc.first] : pc.second;
            std::vector<uint64_t> zs;
            for (size_t k : part) zs.push_back(op->mz[k]);
            const Span sp = gf2_span(zs, 2);
            if (sp.overflow || part.size() > 0xffff)
                return fail(QR_EINVAL, "plan: sub-group of rank > 2 in a complex64 plan");
            SubGroup sg;
            sg.hi = gxs[pc.first] >> pl.b;
            sg.lo = (uint32_t)(gxs[pc.first] & tmask);
            sg.z0 = zs[0];
            sg.d = (uint32_t)sp.basis.size();
            sg.zm = (uint32_t)((sg.z0 & mmask) >> pl.tb);
            if (sg.d > 0) sg.b0 = sp.basis[0];
            if (sg.d > 1) sg.b1 = sp.basis[1];
            for (size_t kk = 0; kk < part.size(); ++kk) {
                sg.mem.push_back((uint32_t)part[kk]);
                sg.coord.push_back((uint8_t)sp.coord[kk]);
            }
            for (uint32_t u = 0; u < 1u << sg.d; ++u) {
                cd acc{0.0, 0.0};
                for (size_t kk = 0; kk < part.size(); ++kk) {
                    const cd v = c[part[kk]];
                    if (__builtin_popcountll(u & sp.coord[kk]) & 1) {
                        acc.re -= v.re;
                        acc.im -= v.im;
                    } else {
                        acc.re += v.re;
                        acc.im += v.im;
                    }
                }
                sg.table[u] = acc;
            }
            subs.push_back(std::move(sg));
        }
        const uint64_t tmask_t = (uint64_t)pl.threads - 1;
        // run key: register-bit sign pattern zm, register bits in the partner
        // XOR (xm), and whether the factor depends on the thread index (tv)
        auto runkey = [&](const SubGroup &g) -> uint32_t {
            const uint32_t tv = ((g.z0 | g.b0 | g.b1) & tmask_t) != 0 ? 1u : 0u;
            return (g.zm & 15u) | (((g.lo >> pl.tb) != 0 ? 1u : 0u) << 4) | (tv << 5);
        };
        // order: partner tile ascending, then run key
        std::vector<size_t> ord(subs.size());
        for (size_t i = 0; i < ord.size(); ++i) ord[i] = i;
        std::stable_sort(ord.begin(), ord.end(), [&](size_t a, size_t b) {
            if (subs[a].hi != subs[b].hi) return subs[a].hi < subs[b].hi;
            return runkey(subs[a]) < runkey(subs[b]);
        });
        std::vector<uint4> td;
        std::vector<TileDataC64> tdd;
        std::vector<uint32_t> r0v, rg0, rkey;
        for (size_t i = 0; i < ord.size(); ++i) {
            const SubGroup &sg = subs[ord[i]];
            const uint32_t zt = (uint32_t)(sg.z0 & tmask_t), bt0 = (uint32_t)(sg.b0 & tmask_t),
                           bt1 = (uint32_t)(sg.b1 & tmask_t);
            const uint32_t tvar = (zt | bt0 | bt1) != 0 ? 1u : 0u;
            // byte-offset XOR of the partner within the tile: thread bits of lo
            // (x 8 bytes) and register bits of lo (x 8 x threads); needs
            // threads == 1 << kC64ThreadBits whenever lo has register bits
            const uint32_t lt = (uint32_t)(sg.lo & tmask_t), lm = sg.lo >> pl.tb;
            const uint32_t dx = (lt << 3) | (lm << (pl.tb + 3));
            td.push_back(make_uint4(dx | (tvar << 31), zt, bt0, bt1));
            TileDataC64 d;
            memset(&d, 0, sizeof(d));
            d.z0h = sg.z0 >> pl.b;
            d.b0h = sg.b0 >> pl.b;
            d.b1h = sg.b1 >> pl.b;
            for (uint32_t u = 0; u < 1u << sg.d; ++u)
                d.T[u] = make_float2((float)sg.table[u].re, (float)sg.table[u].im);
            tdd.push_back(d);
        }
        // runs per block
        for (uint32_t j = 0; j < pl.nblocks; ++j) {
            r0v.push_back((uint32_t)rkey.size());
            for (uint32_t g = bg0[j]; g < bg0[j + 1]; ++g) {
                const uint32_t k = runkey(subs[ord[g]]);
                if (g == bg0[j] || k != rkey.back()) {
                    rkey.push_back(k);
                    rg0.push_back(g);
                }
            }
        }
        r0v.push_back((uint32_t)rkey.size());
        rg0.push_back((uint32_t)ord.size());
        // chunks: consecutive blocks holding at most kTabCap sub-groups; the
        // kernel rebuilds its table (and staged run lists) at each chunk start
        std::vector<uint4> ch;
        for (uint32_t j = 0; j < pl.nblocks; ++j) {
            if (ch.empty() || bg0[j + 1] - ch.back().x > kTabCap)
                ch.push_back(make_uint4(bg0[j], r0v[j], j, 0));
        }
        if (ch.empty()) ch.push_back(make_uint4(0, 0, 0, 0));
        pl.nchunks = (uint32_t)ch.size();
        ch.push_back(make_uint4((uint32_t)ord.size(), (uint32_t)rkey.size(), pl.nblocks, 0));
        QR_CUDA(pl.chunks.upload(ch), "upload chunks");
        if (td.empty()) {
            td.push_back(make_uint4(0, 0, 0, 0));
            TileDataC64 z;
            memset(&z, 0, sizeof(z));
            tdd.push_back(z);
        }
        QR_CUDA(pl.tdesc.upload(td), "upload thread descriptors");
        QR_CUDA(pl.tdata.upload(tdd), "upload tile data");
        for (size_t i = 0; i < ord.size(); ++i) {
            const SubGroup &sg = subs[ord[i]];
            add_slot((uint64_t)pl.tdata.p + i * sizeof(TileDataC64) + offsetof(TileDataC64, T),
                     sg.mem.data(), sg.coord.data(), sg.mem.size(), sg.d, 0);
        }
        QR_CUDA(pl.blk_r0.upload(r0v), "upload block runs");
        QR_CUDA(pl.run_g0.upload(rg0), "upload runs");
        QR_CUDA(pl.run_key.upload(rkey), "upload run keys");
        pl.nruns = (uint32_t)rkey.size();
        QR_CUDA(pl.blk_hi.upload(bhi), "upload blocks");
    }

    if (pl.has_diag) {
        // Tile of the diagonal's transform: 2^8 rows up to n = 16, so that many
        // CTAs share it, 2^12 from n = 20 on, where more tiles form their bins
        // from all the terms more often; larger ones where a bin would hold
        // many terms, which one thread adds up.  Measured, a coefficient update
        // with tiles of 2^5 / 2^8 / 2^10 / 2^12 rows (us): n = 14, 300 terms 23 /
        // 20 / 27 / 49, 16,000 164 / 51 / 62 / 94; n = 16, 60,000 1,251 / 173 /
        // 151 / 192; n = 18, 300 58 / 31 / 32 / 49, 3,000 195 / 55 / 43 / 64,
        // 200,000 14,500 / 1,558 / 555 / 500; n = 20, 30,000 8,560 / 861 / 314 /
        // 183.
        const size_t nd = diag_terms.size();
        int db = std::min(n, std::min(12, std::max(8, n - (nd >= 1024 ? 8 : 9))));
        while (db < std::min(n, 12) && nd >> db > (n < 17 ? 64u : 32u)) ++db;
        const uint64_t dmask = (1ull << db) - 1;
        std::vector<size_t> dt = diag_terms;
        std::stable_sort(dt.begin(), dt.end(), [&](size_t a, size_t b) {
            return (op->mz[a] & dmask) < (op->mz[b] & dmask);
        });
        std::vector<uint64_t> tz, bz;
        std::vector<double> tcv;
        std::vector<uint32_t> boff;
        for (size_t i = 0; i < dt.size(); ++i) {
            const uint64_t zl = op->mz[dt[i]] & dmask;
            if (i == 0 || zl != bz.back()) {
                bz.push_back(zl);
                boff.push_back((uint32_t)i);
            }
            tz.push_back(op->mz[dt[i]]);
            tcv.push_back(c[dt[i]].re);
            tcv.push_back(c[dt[i]].im);
        }
        boff.push_back((uint32_t)dt.size());
        pl.dg_tz = tcv.size() * sizeof(double);
        pl.dg_bz = pl.dg_tz + tz.size() * sizeof(uint64_t);
        pl.dg_boff = pl.dg_bz + bz.size() * sizeof(uint64_t);
        std::vector<unsigned char> img(pl.dg_boff + boff.size() * sizeof(uint32_t));
        memcpy(img.data(), tcv.data(), pl.dg_tz);
        memcpy(img.data() + pl.dg_tz, tz.data(), pl.dg_bz - pl.dg_tz);
        memcpy(img.data() + pl.dg_bz, bz.data(), pl.dg_boff - pl.dg_bz);
        memcpy(img.data() + pl.dg_boff, boff.data(), img.size() - pl.dg_boff);
        QR_CUDA(pl.dg.upload(img), "upload diagonal strings");
        pl.dg_nbins = (uint32_t)bz.size();
        pl.dg_db = db;
        for (size_t i = 0; i < dt.size(); ++i) {
            const uint32_t mi = (uint32_t)dt[i];
            add_slot((uint64_t)pl.dg.p + i * 2 * sizeof(double), &mi, nullptr, 1, 0, 2);
        }
        const size_t esz = f32 ? sizeof(Cplx<float>) : sizeof(Cplx<double>);
        QR_CUDA(pl.diag.alloc(op->N * esz), "alloc diagonal");
        QR_CUDA(run_diag(op, pl, nullptr), "diagonal kernel");
        QR_CUDA(cudaDeviceSynchronize(), "diagonal kernel sync");
    }
    if (slots.empty()) slots.push_back(CoefSlot{});  // keep valid pointers
    pl.prog_mem = slots.size() * sizeof(CoefSlot);
    pl.prog_coord = pl.prog_mem + cmem.size() * sizeof(uint32_t);
    std::vector<unsigned char> prog(pl.prog_coord + ccoord.size());
    memcpy(prog.data(), slots.data(), pl.prog_mem);
    if (!cmem.empty()) {
        memcpy(prog.data() + pl.prog_mem, cmem.data(), cmem.size() * sizeof(uint32_t));
        memcpy(prog.data() + pl.prog_coord, ccoord.data(), ccoord.size());
    }
    QR_CUDA(pl.prog.upload(prog), "upload coefficient program");
    pl.ebits = 0;
    for (const CoefSlot &sl : slots) pl.ebits = std::max(pl.ebits, (int)sl.d);
    pl.nslots = cmem.empty() ? 0u : (uint32_t)slots.size();
    pl.built = true;
    return QR_OK;
}

// bound of every mbarrier wait of the apply kernels
constexpr uint64_t kDefaultWaitNs = 2000000000ull;

// Creation: upload the terms once, then group them on the device
// (qr_group.cu) -- CSR order and groups, merged strings, the apply plan's
// x-groups -- and fold the merged coefficients (merge_coeffs_kernel).  The
// host keeps copies of what the apply plan builder reads.
int create_tables(qr_op *op, const uint64_t *x, const uint64_t *z, const uint8_t *phase,
                  const double *coeff) {
    const uint64_t T = op->T;
    QR_CUDA(op->d_err.alloc(sizeof(int)), "qr_op_create: device allocation");
    QR_CUDA(cudaMemset(op->d_err.p, 0, sizeof(int)), "qr_op_create: clear error word");
    QR_CUDA(op->d_x.alloc(T * 8), "alloc x masks");
    QR_CUDA(op->d_z.alloc(T * 8), "alloc z masks");
    QR_CUDA(op->d_ph.alloc(T), "alloc phases");
    QR_CUDA(op->d_coef.alloc(T * sizeof(cd)), "alloc coefficients");
    QR_CUDA(cudaMemcpy(op->d_x.p, x, T * 8, cudaMemcpyHostToDevice), "upload x masks");
    QR_CUDA(cudaMemcpy(op->d_z.p, z, T * 8, cudaMemcpyHostToDevice), "upload z masks");
    QR_CUDA(cudaMemcpy(op->d_ph.p, phase, T, cudaMemcpyHostToDevice), "upload phases");
    QR_CUDA(cudaMemcpy(op->d_coef.p, coeff, T * sizeof(cd), cudaMemcpyHostToDevice),
            "upload coefficients");
    DevBuf *u32s[] = {&op->d_order, &op->d_mmap, &op->d_mm_terms, &op->d_ag_mem};
    for (DevBuf *b : u32s) QR_CUDA(b->alloc(T * 4), "alloc grouping tables");
    DevBuf *offs[] = {&op->d_goff, &op->d_mm_off, &op->d_ag_off};
    for (DevBuf *b : offs) QR_CUDA(b->alloc((T + 1) * 4), "alloc grouping offsets");
    DevBuf *u64s[] = {&op->d_tz, &op->d_gx, &op->d_mx, &op->d_mz};
    for (DevBuf *b : u64s) QR_CUDA(b->alloc(T * 8), "alloc grouping masks");
    QR_CUDA(op->d_madj.alloc(T), "alloc adjoint signs");
    TermGroupsOut o{op->d_order.as<uint32_t>(), op->d_tz.as<uint64_t>(), op->d_gx.as<uint64_t>(),
                    op->d_goff.as<uint32_t>(), op->d_mmap.as<uint32_t>(),
                    op->d_mm_off.as<uint32_t>(), op->d_mm_terms.as<uint32_t>(),
                    op->d_mx.as<uint64_t>(), op->d_mz.as<uint64_t>(), op->d_madj.as<uint8_t>(),
                    op->d_ag_off.as<uint32_t>(), op->d_ag_mem.as<uint32_t>()};
    TermGroupCounts cnt;
    QR_CUDA(group_terms(op->n, T, op->d_x.as<uint64_t>(), op->d_z.as<uint64_t>(), o, &cnt,
                        nullptr),
            "qr_op_create: grouping terms");
    op->G = cnt.G;
    op->M = cnt.M;
    op->Ga = cnt.Ga;
    QR_CUDA(op->d_mc.alloc(op->M * sizeof(cd)), "alloc merged coefficients");
    QR_CUDA(launch_merge_coeffs((uint32_t)op->M, op->d_mm_off.as<uint32_t>(),
                                op->d_mm_terms.as<uint32_t>(), op->d_coef.as<double2>(),
                                op->d_ph.as<uint8_t>(), op->d_mc.as<double2>(), nullptr),
            "merge coefficients");
    op->gx.resize(op->G);
    op->goff.resize(op->G + 1);
    op->mx.resize(op->M);
    op->mz.resize(op->M);
    op->mc.resize(op->M);
    op->ag_off.resize(op->Ga + 1);
    op->ag_mem.resize(op->M);
    QR_CUDA(cudaMemcpy(op->gx.data(), op->d_gx.p, op->G * 8, cudaMemcpyDeviceToHost), "fetch gx");
    QR_CUDA(cudaMemcpy(op->goff.data(), op->d_goff.p, (op->G + 1) * 4, cudaMemcpyDeviceToHost),
            "fetch group offsets");
    QR_CUDA(cudaMemcpy(op->mx.data(), op->d_mx.p, op->M * 8, cudaMemcpyDeviceToHost), "fetch mx");
    QR_CUDA(cudaMemcpy(op->mz.data(), op->d_mz.p, op->M * 8, cudaMemcpyDeviceToHost), "fetch mz");
    QR_CUDA(cudaMemcpy(op->mc.data(), op->d_mc.p, op->M * sizeof(cd), cudaMemcpyDeviceToHost),
            "fetch merged coefficients");
    QR_CUDA(cudaMemcpy(op->ag_off.data(), op->d_ag_off.p, (op->Ga + 1) * 4,
                       cudaMemcpyDeviceToHost),
            "fetch x-group offsets");
    QR_CUDA(cudaMemcpy(op->ag_mem.data(), op->d_ag_mem.p, op->M * 4, cudaMemcpyDeviceToHost),
            "fetch x-group members");
    return QR_OK;
}

int check_device(const qr_op *op) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
    if (dev != op->device)
        return fail(QR_ESTATE, "operator lives on device %d but device %d is current", op->device,
                    dev);
    return QR_OK;
}

int check_kernel_error(qr_op *op) {
    int h = 0;
    QR_CUDA(cudaMemcpy(&h, op->d_err.p, sizeof(int), cudaMemcpyDeviceToHost), "read error word");
    if (h != kErrNone) {
        int z = 0;
        cudaMemcpy(op->d_err.p, &z, sizeof(int), cudaMemcpyHostToDevice);
        return fail(QR_EKERNEL, "kernel reported error %d (%s)", h,
                    h == kErrMbarTimeout ? "bounded mbarrier wait expired"
                                         : "CSR position out of range");
    }
    return QR_OK;
}

}  // namespace

extern "C" {

int qr_op_create(int32_t n, uint64_t nterms, const uint64_t *x, const uint64_t *z,
                 const uint8_t *phase, const double *coeff, qr_op **out) {
    if (!out) return fail(QR_EINVAL, "qr_op_create: out is null");
    *out = nullptr;
    if (n < 1 || n > 63) return fail(QR_EINVAL, "qr_op_create: n=%d outside [1, 63]", n);
    if (nterms == 0)
        return fail(QR_EINVAL, "SparsePauliOp::new: at least one pauli must be supplied");
    if (nterms > 0xffffffffull) return fail(QR_EINVAL, "qr_op_create: too many terms");
    if (!x || !z || !phase || !coeff) return fail(QR_EINVAL, "qr_op_create: null term array");
    const uint64_t lim = (n == 64) ? ~0ull : ((1ull << n) - 1);
    for (uint64_t k = 0; k < nterms; ++k) {
        if ((x[k] & ~lim) || (z[k] & ~lim))
            return fail(QR_EINVAL, "qr_op_create: term %llu has mask bits beyond n=%d",
                        (unsigned long long)k, n);
        if (phase[k] > 3)
            return fail(QR_EINVAL, "qr_op_create: term %llu phase %u > 3", (unsigned long long)k,
                        (unsigned)phase[k]);
    }
    qr_op *op = new (std::nothrow) qr_op();
    if (!op) return fail(QR_ENOMEM, "qr_op_create: out of host memory");
    op->n = n;
    op->N = 1ull << n;
    op->T = nterms;
    cudaError_t e = cudaGetDevice(&op->device);
    if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(&op->nsm, cudaDevAttrMultiProcessorCount, op->device);
    if (e != cudaSuccess) {
        delete op;
        return cuda_fail(e, "qr_op_create: no usable CUDA device");
    }
    const int rc = create_tables(op, x, z, phase, coeff);
    if (rc) {
        delete op;
        return rc;
    }
    *out = op;
    return QR_OK;
}

int qr_op_destroy(qr_op *op) {
    if (!op) return QR_OK;
    int dev = -1;
    cudaGetDevice(&dev);
    const int home = op->device;
    if (dev != home) cudaSetDevice(home);
    if (op->hstream) cudaStreamDestroy(op->hstream);
    if (op->cstream) cudaStreamDestroy(op->cstream);
    if (op->cev) cudaEventDestroy(op->cev);
    delete op;
    if (dev >= 0 && dev != home) cudaSetDevice(dev);
    return QR_OK;
}

int qr_check(qr_op *op, void *stream) {
    if (!op) return fail(QR_EINVAL, "qr_check: null operator");
    int rc = check_device(op);
    if (rc) return rc;
    QR_CUDA(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)), "qr_check sync");
    return check_kernel_error(op);
}

int qr_op_get_info(const qr_op *op_c, qr_op_info *info) {
    if (!op_c || !info) return fail(QR_EINVAL, "qr_op_get_info: null argument");
    qr_op *op = const_cast<qr_op *>(op_c);
    int rc = check_device(op);
    if (rc) return rc;
    rc = build_plan(op, QR_C64C, 0);
    if (rc) return rc;
    rc = build_plan(op, QR_C128, 0);
    if (rc) return rc;
    const Plan &pl = op->plans[QR_C64C][0];
    info->n = op->n;
    info->tile_bits = pl.b;
    info->nterms = op->T;
    info->ngroups = op->G;
    info->nmerged = op->M;
    info->nblocks = pl.nblocks;
    info->nfat = op->plans[QR_C128][0].nfat;
    info->nsub = pl.nsub;
    info->has_diag = pl.has_diag ? 1 : 0;
    info->device = op->device;
    return QR_OK;
}

int qr_op_get_groups(const qr_op *op, uint64_t *ngroups, uint64_t *gx, uint32_t *goff,
                     uint32_t *order, uint32_t *mmap) {
    if (!op || !ngroups) return fail(QR_EINVAL, "qr_op_get_groups: null argument");
    int rc = check_device(op);
    if (rc) return rc;
    *ngroups = op->G;
    QR_CUDA(cudaDeviceSynchronize(), "qr_op_get_groups sync");
    if (gx) std::memcpy(gx, op->gx.data(), op->G * sizeof(uint64_t));
    if (goff) std::memcpy(goff, op->goff.data(), (op->G + 1) * sizeof(uint32_t));
    if (order)
        QR_CUDA(cudaMemcpy(order, op->d_order.p, op->T * 4, cudaMemcpyDeviceToHost),
                "fetch term order");
    if (mmap)
        QR_CUDA(cudaMemcpy(mmap, op->d_mmap.p, op->T * 4, cudaMemcpyDeviceToHost),
                "fetch merged-string map");
    return QR_OK;
}

int qr_csr_size(const qr_op *op, uint64_t *nrows, uint64_t *nnz) {
    if (!op || !nrows || !nnz) return fail(QR_EINVAL, "qr_csr_size: null argument");
    *nrows = op->N;
    if (op->G != 0 && op->N > ~0ull / op->G) return fail(QR_EINVAL, "qr_csr_size: nnz overflows");
    *nnz = op->N * op->G;
    return QR_OK;
}

int qr_csr_build(qr_op *op, uint64_t *indptr, uint64_t *indices, double *data, int32_t mem,
                 void *stream) {
    if (!op || !indptr || !indices || !data) return fail(QR_EINVAL, "qr_csr_build: null argument");
    if (mem != QR_MEM_DEVICE && mem != QR_MEM_HOST)
        return fail(QR_EINVAL, "qr_csr_build: mem must be QR_MEM_DEVICE or QR_MEM_HOST");
    int rc = check_device(op);
    if (rc) return rc;
    rc = upload_csr_tables(op);
    if (rc) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    CsrArgs a = csr_args(op);
    // fold-mode values buffer (nfold x rows) for the staged fill; without
    // it the fold entries are stored in place after the fill
    auto fold_buffer = [&](uint64_t rows) {
        a.fvals = nullptr;
        if (op->nfold == 0 || op->G > 256 || a.inline_fold) return;
        // One such group: in place after the fill, which costs a sector per entry,
        // where the fill has many rows, or groups of several classes, whose stages
        // the placing lengthens (us, placed by the fill / in place): Jordan-Wigner,
        // 60 Z strings, n = 18 268 / 230, n = 19 534 / 454, n = 20 1,034 / 847; 60
        // strings with x masks of their own and such a group n = 18 101 / 114, n = 20
        // 342 / 331.  More groups: n = 18, 4 of 150 193 / 236, 16 322 / 475.
        if (op->nfold == 1 && (op->n >= 20 || (op->n >= 18 && op->nctab >= 4 * op->G))) return;
        if (op->d_fv.alloc((size_t)op->nfold * rows * sizeof(double2)) == cudaSuccess)
            a.fvals = op->d_fv.as<double2>();
        else
            (void)cudaGetLastError();  // allocation failure is not sticky: clear it
    };
    if (mem == QR_MEM_DEVICE) {
        fold_buffer(op->N);
        a.indptr = indptr;
        a.indices = indices;
        a.data = data;
        a.row0 = 0;
        a.nrows = op->N;
        QR_CUDA(launch_csr_fill(a, op->nsm, st), "csr fill launch");
        return QR_OK;
    }
    // host destination: build in row chunks of <= ~1 GiB on the device
    const uint64_t per_row = op->G * 24;
    uint64_t rows = (1ull << 30) / (per_row ? per_row : 1);
    // whole chunks (of 512 rows for one group, 256 at most otherwise), so that every
    // launch starts on a chunk boundary
    rows = rows < 512 ? 256 : rows & ~511ull;
    if (rows > op->N) rows = op->N;
    DevBuf d_ptr, d_idx, d_dat;
    QR_CUDA(d_ptr.alloc((op->N + 1) * sizeof(uint64_t)), "alloc indptr staging");
    QR_CUDA(d_idx.alloc(rows * op->G * sizeof(uint64_t)), "alloc indices staging");
    QR_CUDA(d_dat.alloc(rows * op->G * 2 * sizeof(double)), "alloc data staging");
    fold_buffer(rows);
    for (uint64_t r0 = 0; r0 < op->N; r0 += rows) {
        const uint64_t nr = std::min(rows, op->N - r0);
        a.indptr = (r0 == 0) ? d_ptr.as<uint64_t>() : nullptr;
        a.indices = d_idx.as<uint64_t>();
        a.data = d_dat.as<double>();
        a.row0 = r0;
        a.nrows = nr;
        QR_CUDA(launch_csr_fill(a, op->nsm, st), "csr fill launch");
        QR_CUDA(cudaMemcpyAsync(indices + r0 * op->G, d_idx.p, nr * op->G * sizeof(uint64_t),
                                cudaMemcpyDeviceToHost, st),
                "copy indices");
        QR_CUDA(cudaMemcpyAsync(data + 2 * r0 * op->G, d_dat.p, nr * op->G * 2 * sizeof(double),
                                cudaMemcpyDeviceToHost, st),
                "copy data");
    }
    QR_CUDA(cudaMemcpyAsync(indptr, d_ptr.p, (op->N + 1) * sizeof(uint64_t),
                            cudaMemcpyDeviceToHost, st),
            "copy indptr");
    QR_CUDA(cudaStreamSynchronize(st), "csr build sync");
    return check_kernel_error(op);
}

// psi and y (bytes each) share memory
static bool states_overlap(const void *psi, const void *y, uint64_t bytes) {
    const char *p = static_cast<const char *>(psi), *q = static_cast<const char *>(y);
    return p < q + bytes && q < p + bytes;
}

// call_states: states of the caller's whole call, of which these nstates are
// a part (the same work split, and so the same bits, for each of them)
static int apply_impl(const char *name, qr_op *op, int32_t dtype, const void *psi, void *y,
                      int32_t nstates, int32_t call_states, int32_t adjoint, void *stream,
                      const void *v, const double *alpha, const double *beta) {
    if (!op || !psi || !y) return fail(QR_EINVAL, "%s: null argument", name);
    if (dtype != QR_C128 && dtype != QR_C64C)
        return fail(QR_EINVAL, "%s: dtype must be QR_C128 or QR_C64C", name);
    if (nstates < 1) return fail(QR_EINVAL, "%s: nstates=%d < 1", name, nstates);
    if (adjoint != 0 && adjoint != 1) return fail(QR_EINVAL, "%s: adjoint must be 0 or 1", name);
    if (op->n > 40) return fail(QR_EINVAL, "%s: n=%d too large for a state vector", name, op->n);
    const size_t esz = dtype == QR_C128 ? 16 : 8;
    const uint64_t bytes = (uint64_t)nstates * op->N * esz;
    const char *yb = static_cast<const char *>(y);
    if (states_overlap(psi, y, bytes)) return fail(QR_EINVAL, "%s: psi and y overlap", name);
    if ((reinterpret_cast<uintptr_t>(psi) | reinterpret_cast<uintptr_t>(y)) & 15)
        return fail(QR_EINVAL, "%s: psi and y must be 16-byte aligned", name);
    if (v) {
        // v is only read: it may be psi, or y itself (each element of y is
        // read by the thread that then writes it), but not a shifted view of y
        const char *vb = static_cast<const char *>(v);
        if (vb != yb && vb < yb + bytes && yb < vb + bytes)
            return fail(QR_EINVAL, "%s: v overlaps y without being y", name);
        if (reinterpret_cast<uintptr_t>(v) & 15)
            return fail(QR_EINVAL, "%s: v must be 16-byte aligned", name);
    }
    int rc = check_device(op);
    if (rc) return rc;
    rc = build_plan(op, dtype, adjoint);
    if (rc) return rc;
    const Plan &pl = op->plans[dtype][adjoint];
    ApplyArgs a{};
    a.psi = psi;
    a.y = y;
    a.N = op->N;
    a.n = op->n;
    a.b = pl.b;
    a.tb = pl.tb;
    a.nstates = nstates;
    a.ntiles = op->N >> pl.b;
    a.nitems = (uint64_t)nstates * a.ntiles;
    a.groups = pl.groups.as<GroupDesc>();
    a.ngroups = pl.nrgroups;
    a.tables = pl.groups.as<unsigned char>() + pl.rtables;
    a.fat_z = pl.fat_z.as<uint64_t>();
    a.fat_c = pl.fat_c.p;
    a.blk_hi = pl.blk_hi.as<uint64_t>();
    a.nblocks = pl.nblocks;
    a.diag = pl.has_diag ? pl.diag.p : nullptr;
    a.diag_block = pl.diag_block;
    a.err = op->d_err.as<int>();
    a.nsub = pl.nsub;
    a.tdesc = pl.tdesc.as<uint4>();
    a.tdata = pl.tdata.as<TileDataC64>();
    a.blk_r0 = pl.blk_r0.as<uint32_t>();
    a.run_g0 = pl.run_g0.as<uint32_t>();
    a.run_key = pl.run_key.as<uint32_t>();
    a.nruns = pl.nruns;
    a.chunks = pl.chunks.as<uint4>();
    a.nchunks = pl.nchunks;
    a.cblk = pl.cblk.as<uint4>();
    a.ctdesc = pl.ctdesc.as<uint4>();
    a.ctdata = pl.ctdata.as<TileDataC64>();
    a.ncblk = pl.ncblk;
    a.ncsub = pl.ncsub;
    a.ent = pl.ent.as<uint4>();
    a.sblk = pl.sblk.as<uint4>();
    a.wait_ns = op->test_wait_ns ? op->test_wait_ns : kDefaultWaitNs;
    a.withhold = op->test_withhold;
    a.wide = op->test_wide;
    a.v = v;
    if (v) {
        a.ar = alpha[0];
        a.ai = alpha[1];
        a.br = beta[0];
        a.bi = beta[1];
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (over_rows(op, pl, call_states))
        QR_CUDA(launch_rows(dtype, a, (uint64_t)call_states * op->N, st), "apply launch");
    else if (pl.strings)
        QR_CUDA(launch_c64c_strings(a, pl.str, (uint64_t)call_states * a.ntiles, op->nsm, st),
                "apply launch");
    else if (pl.cosets)
        QR_CUDA(launch_c64c_cosets(a, op->nsm, st), "apply launch");
    else
        QR_CUDA(launch_apply(a, pl.amps, pl.threads, op->nsm, st), "apply launch");
    return QR_OK;
}

int qr_apply(qr_op *op, int32_t dtype, const void *psi, void *y, int32_t nstates, int32_t adjoint,
             void *stream) {
    return apply_impl("qr_apply", op, dtype, psi, y, nstates, nstates, adjoint, stream, nullptr,
                      nullptr, nullptr);
}

int qr_apply_axpby(qr_op *op, int32_t dtype, const double *alpha, const void *psi,
                   const double *beta, const void *v, void *y, int32_t nstates, void *stream) {
    if (!alpha || !beta || !v) return fail(QR_EINVAL, "qr_apply_axpby: null argument");
    return apply_impl("qr_apply_axpby", op, dtype, psi, y, nstates, nstates, 0, stream, v, alpha,
                      beta);
}

int qr_apply_host(qr_op *op, int32_t dtype, const void *psi_host, void *y_host, int32_t nstates,
                  int32_t adjoint) {
    if (!op || !psi_host || !y_host) return fail(QR_EINVAL, "qr_apply_host: null argument");
    if (dtype != QR_C128 && dtype != QR_C64C)
        return fail(QR_EINVAL, "qr_apply_host: dtype must be QR_C128 or QR_C64C");
    if (nstates < 1) return fail(QR_EINVAL, "qr_apply_host: nstates=%d < 1", nstates);
    int rc = check_device(op);
    if (rc) return rc;
    const size_t esz = dtype == QR_C128 ? 16 : 8;
    const uint64_t bytes = (uint64_t)nstates * op->N * esz;
    if (!op->hstream) QR_CUDA(cudaStreamCreateWithFlags(&op->hstream, cudaStreamNonBlocking),
                              "create stream");
    if (op->stage_in.bytes < bytes) QR_CUDA(op->stage_in.alloc(bytes), "alloc psi staging");
    // Pinned (page-locked, mapped) y: the kernel stores each finished output
    // tile straight into host memory, so the write-back overlaps the
    // computation instead of following it.  Pageable y: device staging + copy.
    void *y_dev = nullptr;
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, y_host) == cudaSuccess && at.type == cudaMemoryTypeHost &&
        at.devicePointer != nullptr)
        y_dev = at.devicePointer;
    cudaGetLastError();  // a pageable pointer may leave a benign error behind
    if (!y_dev && op->stage_out.bytes < bytes)
        QR_CUDA(op->stage_out.alloc(bytes), "alloc y staging");
    const char *pb = static_cast<const char *>(psi_host);
    char *yb = static_cast<char *>(y_host);
    if (nstates > 1 && (pb + bytes <= yb || yb + bytes <= pb)) {
        // Several states, psi and y apart: state s + 1 is copied in on a
        // second stream while the kernel works on state s (an event orders
        // each state's kernel after its copy), so only the first copy is
        // not hidden.
        if (!op->cstream)
            QR_CUDA(cudaStreamCreateWithFlags(&op->cstream, cudaStreamNonBlocking), "create stream");
        if (!op->cev) QR_CUDA(cudaEventCreateWithFlags(&op->cev, cudaEventDisableTiming), "event");
        const uint64_t b1 = op->N * esz;
        char *in = static_cast<char *>(op->stage_in.p);
        char *out = static_cast<char *>(y_dev ? y_dev : op->stage_out.p);
        for (int32_t st = 0; st < nstates; ++st) {
            QR_CUDA(cudaMemcpyAsync(in + st * b1, pb + st * b1, b1, cudaMemcpyHostToDevice,
                                    op->cstream),
                    "copy psi to device");
            QR_CUDA(cudaEventRecord(op->cev, op->cstream), "record copy");
            QR_CUDA(cudaStreamWaitEvent(op->hstream, op->cev, 0), "order apply after copy");
            rc = apply_impl("qr_apply_host", op, dtype, in + st * b1, out + st * b1, 1, nstates,
                            adjoint, op->hstream, nullptr, nullptr, nullptr);
            if (rc) return rc;
            if (!y_dev)
                QR_CUDA(cudaMemcpyAsync(yb + st * b1, out + st * b1, b1, cudaMemcpyDeviceToHost,
                                        op->hstream),
                        "copy y to host");
        }
        QR_CUDA(cudaStreamSynchronize(op->hstream), "apply_host sync");
        return check_kernel_error(op);
    }
    QR_CUDA(cudaMemcpyAsync(op->stage_in.p, psi_host, bytes, cudaMemcpyHostToDevice, op->hstream),
            "copy psi to device");
    rc = qr_apply(op, dtype, op->stage_in.p, y_dev ? y_dev : op->stage_out.p, nstates, adjoint,
                  op->hstream);
    if (rc) return rc;
    if (!y_dev)
        QR_CUDA(cudaMemcpyAsync(y_host, op->stage_out.p, bytes, cudaMemcpyDeviceToHost,
                                op->hstream),
                "copy y to host");
    QR_CUDA(cudaStreamSynchronize(op->hstream), "apply_host sync");
    return check_kernel_error(op);
}

int qr_csr_spmv(uint64_t nrows, uint64_t ncols, const uint64_t *indptr, const uint64_t *indices,
                const double *data, const double *v, double *y, void *stream) {
    if (!indptr || !indices || !data || !v || !y) return fail(QR_EINVAL, "qr_csr_spmv: null argument");
    int dev = 0, nsm = 0;
    QR_CUDA(cudaGetDevice(&dev), "cudaGetDevice");
    QR_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev), "device attribute");
    QR_CUDA(launch_csr_spmv(nrows, ncols, indptr, indices, data, v, y, nsm,
                            static_cast<cudaStream_t>(stream)),
            "csr spmv launch");
    return QR_OK;
}

// ---------------------------------------------------------------- vector helpers
static int current_nsm(int *nsm) {
    int dev = 0;
    QR_CUDA(cudaGetDevice(&dev), "cudaGetDevice");
    QR_CUDA(cudaDeviceGetAttribute(nsm, cudaDevAttrMultiProcessorCount, dev), "device attribute");
    return QR_OK;
}

static int vec_call(const char *name, int op, int32_t dtype, uint64_t len, const void *x,
                    const void *y, void *z, const double *a, const double *b, double tol,
                    void *stream) {
    if (dtype != QR_C128 && dtype != QR_C64C)
        return fail(QR_EINVAL, "%s: dtype must be QR_C128 or QR_C64C", name);
    if (len == 0) return QR_OK;
    if (!x || !z || (op != 2 && !y) || !a) return fail(QR_EINVAL, "%s: null argument", name);
    int nsm = 0;
    int rc = current_nsm(&nsm);
    if (rc) return rc;
    QR_CUDA(launch_vec_op(op, dtype == QR_C64C, len, x, y, z, a, b, tol, nsm,
                          static_cast<cudaStream_t>(stream)),
            name);
    return QR_OK;
}

int qr_axpby(int32_t dtype, uint64_t len, const double *a, const void *x, const double *b,
             const void *y, void *z, void *stream) {
    if (len && !b) return fail(QR_EINVAL, "qr_axpby: null argument");
    return vec_call("qr_axpby", 0, dtype, len, x, y, z, a, b, 0.0, stream);
}

int qr_axpy(int32_t dtype, uint64_t len, const double *a, const void *x, const void *y, void *z,
            void *stream) {
    return vec_call("qr_axpy", 1, dtype, len, x, y, z, a, nullptr, 0.0, stream);
}

int qr_ax(int32_t dtype, uint64_t len, const double *a, const void *x, void *z, void *stream) {
    return vec_call("qr_ax", 2, dtype, len, x, nullptr, z, a, nullptr, 0.0, stream);
}

int qr_precond2(int32_t dtype, uint64_t len, const void *diag, const void *dx, const double *e,
                double tol, void *out, void *stream) {
    return vec_call("qr_precond2", 3, dtype, len, diag, dx, out, e, nullptr, tol, stream);
}

int qr_csr_diagonal(uint64_t nrows, uint64_t ncols, const uint64_t *indptr,
                    const uint64_t *indices, const double *data, double *out, void *stream) {
    const uint64_t nd = nrows < ncols ? nrows : ncols;
    if (nd == 0) return QR_OK;
    if (!indptr || !indices || !data || !out)
        return fail(QR_EINVAL, "qr_csr_diagonal: null argument");
    int nsm = 0;
    int rc = current_nsm(&nsm);
    if (rc) return rc;
    QR_CUDA(launch_csr_diag(nd, indptr, indices, data, out, nsm,
                            static_cast<cudaStream_t>(stream)),
            "csr diagonal launch");
    return QR_OK;
}

int qr_op_diagonal(qr_op *op, int32_t dtype, void *out, void *stream) {
    if (!op || !out) return fail(QR_EINVAL, "qr_op_diagonal: null argument");
    if (dtype != QR_C128 && dtype != QR_C64C)
        return fail(QR_EINVAL, "qr_op_diagonal: dtype must be QR_C128 or QR_C64C");
    int rc = check_device(op);
    if (rc) return rc;
    rc = upload_csr_tables(op);
    if (rc) return rc;
    // groups are sorted by x ascending, so an x = 0 group is group 0
    const uint32_t nt = (op->G > 0 && op->gx[0] == 0) ? op->goff[1] - op->goff[0] : 0;
    QR_CUDA(launch_op_diag(op->N, nt, op->d_tz.as<uint64_t>(), op->d_tc.as<double>(), out,
                           dtype == QR_C64C, op->nsm, static_cast<cudaStream_t>(stream)),
            "operator diagonal launch");
    return QR_OK;
}

// Merged coefficients and the built CSR tables from d_coef, on stream st.
static int recompute_coeffs(qr_op *op, cudaStream_t st) {
    QR_CUDA(launch_merge_coeffs((uint32_t)op->M, op->d_mm_off.as<uint32_t>(),
                                op->d_mm_terms.as<uint32_t>(), op->d_coef.as<double2>(),
                                op->d_ph.as<uint8_t>(), op->d_mc.as<double2>(), st),
            "merge coefficients");
    if (op->csr_ready) return refresh_csr_values(op, st);
    return QR_OK;
}

int qr_op_set_coeffs(qr_op *op, const double *coeff) {
    if (!op || !coeff) return fail(QR_EINVAL, "qr_op_set_coeffs: null argument");
    int rc = check_device(op);
    if (rc) return rc;
    QR_CUDA(cudaDeviceSynchronize(), "qr_op_set_coeffs sync");
    QR_CUDA(cudaMemcpy(op->d_coef.p, coeff, op->T * sizeof(cd), cudaMemcpyHostToDevice),
            "upload coefficients");
    rc = recompute_coeffs(op, nullptr);
    if (rc) return rc;
    op->host_coef_stale = true;  // plans built below fetch the new merged sums
    for (int d = 0; d < 2; ++d)
        for (int j = 0; j < 2; ++j) op->plans[d][j].built = false;
    // plans are rebuilt on next use into the buffers they already hold
    for (Plan &bp : op->bplans) bp.built = false;
    ++op->coef_gen;
    return QR_OK;
}

int qr_op_set_coeffs_device(qr_op *op, const double *coeff, void *stream) {
    if (!op || !coeff) return fail(QR_EINVAL, "qr_op_set_coeffs_device: null argument");
    int rc = check_device(op);
    if (rc) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    QR_CUDA(cudaMemcpyAsync(op->d_coef.p, coeff, op->T * sizeof(cd), cudaMemcpyDeviceToDevice,
                            st),
            "copy device coefficients");
    rc = recompute_coeffs(op, st);
    if (rc) return rc;
    auto refresh = [&](Plan &pl) -> int {
        if (!pl.built) return QR_OK;
        const unsigned char *prog = pl.prog.as<unsigned char>();
        QR_CUDA(launch_coef_program(pl.prog.as<CoefSlot>(), pl.nslots, pl.ebits,
                                    reinterpret_cast<const uint32_t *>(prog + pl.prog_mem),
                                    prog + pl.prog_coord, op->d_mc.as<double2>(),
                                    op->d_madj.as<uint8_t>(), pl.adjoint, st),
                "coefficient program");
        if (pl.has_diag)
            QR_CUDA(run_diag(op, pl, st), "diagonal kernel");
        return QR_OK;
    };
    for (int d = 0; d < 2; ++d)
        for (int j = 0; j < 2; ++j) {
            rc = refresh(op->plans[d][j]);
            if (rc) return rc;
        }
    for (Plan &bp : op->bplans) {
        rc = refresh(bp);
        if (rc) return rc;
    }
    op->host_coef_stale = true;
    return QR_OK;
}

int qr_op_set_test_hooks(qr_op *op, uint32_t flags, uint64_t wait_ns, int64_t withhold_step) {
    if (!op) return fail(QR_EINVAL, "qr_op_set_test_hooks: null operator");
    if (flags & ~(uint32_t)QR_TEST_FORCE_WIDE)
        return fail(QR_EINVAL, "qr_op_set_test_hooks: unknown flag bits 0x%x", flags);
    if (wait_ns != 0 && wait_ns < 1000000ull)
        return fail(QR_EINVAL, "qr_op_set_test_hooks: wait_ns below 1 ms");
    if (withhold_step < -1) return fail(QR_EINVAL, "qr_op_set_test_hooks: withhold_step < -1");
    op->test_wide = (flags & QR_TEST_FORCE_WIDE) ? 1 : 0;
    op->test_wait_ns = wait_ns;
    op->test_withhold = withhold_step;
    return QR_OK;
}

int qr_op_apply_form(qr_op *op, int32_t dtype, int32_t adjoint, int32_t nstates) {
    if (!op) return fail(QR_EINVAL, "qr_op_apply_form: null operator");
    if (dtype != QR_C128 && dtype != QR_C64C) return fail(QR_EINVAL, "qr_op_apply_form: bad dtype");
    if (adjoint != 0 && adjoint != 1) return fail(QR_EINVAL, "qr_op_apply_form: bad adjoint");
    if (nstates < 1) return fail(QR_EINVAL, "qr_op_apply_form: nstates=%d < 1", nstates);
    int rc = check_device(op);
    if (rc) return rc;
    rc = build_plan(op, dtype, adjoint);
    if (rc) return rc;
    const Plan &pl = op->plans[dtype][adjoint];
    return over_rows(op, pl, nstates) ? QR_FORM_ROWS
           : pl.strings               ? QR_FORM_STRINGS
           : pl.cosets                ? QR_FORM_COSETS
                                      : QR_FORM_TABLES;
}

int qr_vdot(int32_t n, int32_t dtype, const void *a, const void *b, int32_t nstates, double *out,
            void *stream) {
    if (!a || !b || !out) return fail(QR_EINVAL, "qr_vdot: null argument");
    if (n < 1 || n > 40) return fail(QR_EINVAL, "qr_vdot: n=%d outside [1, 40]", n);
    if (dtype != QR_C128 && dtype != QR_C64C) return fail(QR_EINVAL, "qr_vdot: bad dtype");
    if (nstates < 1) return fail(QR_EINVAL, "qr_vdot: nstates=%d < 1", nstates);
    // one grid row per state (gridDim.y)
    if (nstates > 65535) return fail(QR_EINVAL, "qr_vdot: nstates=%d > 65535", nstates);
    int dev = 0, nsm = 0;
    QR_CUDA(cudaGetDevice(&dev), "cudaGetDevice");
    QR_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev), "device attribute");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const uint64_t N = 1ull << n;
    const uint32_t nblk = vdot_blocks(N, nsm);
    void *partial = nullptr;
    QR_CUDA(cudaMallocAsync(&partial, (size_t)nstates * nblk * sizeof(double2), st),
            "vdot scratch");
    cudaError_t e = launch_vdot(dtype, N, a, b, nstates, static_cast<double2 *>(partial), nblk,
                                reinterpret_cast<double2 *>(out), st);
    cudaFreeAsync(partial, st);
    if (e != cudaSuccess) return cuda_fail(e, "vdot launch");
    return QR_OK;
}

int qr_expect(qr_op *op, int32_t dtype, const void *psi, int32_t nstates, double *out,
              void *stream) {
    if (!op || !psi || !out) return fail(QR_EINVAL, "qr_expect: null argument");
    if (dtype != QR_C128 && dtype != QR_C64C) return fail(QR_EINVAL, "qr_expect: bad dtype");
    if (nstates < 1) return fail(QR_EINVAL, "qr_expect: nstates=%d < 1", nstates);
    if (nstates > 65535) return fail(QR_EINVAL, "qr_expect: nstates=%d > 65535", nstates);
    int rc = check_device(op);
    if (rc) return rc;
    const size_t esz = dtype == QR_C128 ? 16 : 8;
    const uint64_t bytes = (uint64_t)nstates * op->N * esz;
    if (op->expect_y.bytes < bytes) QR_CUDA(op->expect_y.alloc(bytes), "alloc expect buffer");
    rc = qr_apply(op, dtype, psi, op->expect_y.p, nstates, 0, stream);
    if (rc) return rc;
    return qr_vdot(op->n, dtype, psi, op->expect_y.p, nstates, out, stream);
}

// Chunks of rows of the string-by-string gradients: about 8 work items of four
// strings per SM, chunks of at least 4,096 rows.
static uint64_t grad_chunks(uint64_t strings, uint64_t N, int nsm) {
    const uint64_t items = (strings + 3) / 4;
    if (items == 0) return 1;
    return std::max<uint64_t>(1, std::min(((uint64_t)nsm * 8 + items - 1) / items, N / 4096));
}

int qr_term_grad(qr_op *op, int32_t dtype, const void *psi, const void *g, int32_t nstates,
                 double *out, void *stream) {
    if (!op || !psi || !g || !out) return fail(QR_EINVAL, "qr_term_grad: null argument");
    if (dtype != QR_C128 && dtype != QR_C64C) return fail(QR_EINVAL, "qr_term_grad: bad dtype");
    if (nstates < 1) return fail(QR_EINVAL, "qr_term_grad: nstates=%d < 1", nstates);
    if (op->n > 40) return fail(QR_EINVAL, "qr_term_grad: n=%d too large", op->n);
    int rc = check_device(op);
    if (rc) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    qr_op::GradPlan &tg = op->tg[dtype];
    const bool tiles = dtype == QR_C64C && op->n >= 12;
    // The first call inside a stream capture, where no plan can be uploaded:
    // string by string from the merged masks on the device (the tiled kernel
    // needs its batches)
    bool unplanned = false;
    if (!tg.ready && !tiles) {
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        QR_CUDA(cudaStreamIsCapturing(st, &cap), "term-grad capture status");
        unplanned = cap == cudaStreamCaptureStatusActive;
    }
    if (!tg.ready && !unplanned) {
        // complex128: x groups of many strings to the transform; the others in order of
        // partner tile, input order kept within one; batches of <= 8 never
        // span two partner tiles, largest first
        std::vector<uint32_t> ord, word;
        std::vector<GradBatch> wb;
        uint64_t many = 0;  // strings that the transform could take
        for (size_t g = 0; g < op->Ga; ++g) {
            const uint32_t k = op->ag_off[g + 1] - op->ag_off[g];
            if (k >= kGradWhtMin) many += k;
        }
        // rows that an SM passes four strings over, one by one
        auto direct_rows = [&](uint64_t k) {
            const uint64_t chunks = grad_chunks(k, op->N, op->nsm);
            const uint64_t rounds = ((k + 3) / 4 * chunks + op->nsm - 1) / op->nsm;
            return rounds * (op->N / chunks);
        };
        const bool wht = dtype == QR_C128 && many > 0 &&
                         direct_rows(op->M) >= direct_rows(op->M - many) + kGradWhtRows;
        for (size_t g = 0; g < op->Ga; ++g) {
            const uint32_t a0 = op->ag_off[g], a1 = op->ag_off[g + 1];
            if (!wht || a1 - a0 < kGradWhtMin) {
                ord.insert(ord.end(), op->ag_mem.begin() + a0, op->ag_mem.begin() + a1);
                continue;
            }
            for (uint32_t k = a0; k < a1; k += kGradWhtBatch) {
                const uint32_t cnt = std::min(kGradWhtBatch, a1 - k);
                wb.push_back(GradBatch{op->mx[op->ag_mem[k]], (uint32_t)word.size(), cnt});
                word.insert(word.end(), op->ag_mem.begin() + k, op->ag_mem.begin() + k + cnt);
            }
        }
        std::sort(ord.begin(), ord.end());
        std::stable_sort(ord.begin(), ord.end(), [&](uint32_t a, uint32_t b) {
            return (op->mx[a] >> 12) < (op->mx[b] >> 12);
        });
        const uint32_t nd = (uint32_t)ord.size();
        std::vector<uint64_t> sx(nd), sz(nd), wz;
        for (uint32_t i = 0; i < nd; ++i) {
            sx[i] = op->mx[ord[i]];
            sz[i] = op->mz[ord[i]];
        }
        for (uint32_t k : word) wz.push_back(op->mz[k]);
        std::vector<uint2> bat;
        for (uint32_t i = 0; i < nd;) {
            uint32_t j = i + 1;
            while (j < nd && j - i < 8 && (sx[j] >> 12) == (sx[i] >> 12)) ++j;
            bat.push_back(make_uint2(i, j - i));
            i = j;
        }
        std::stable_sort(bat.begin(), bat.end(),
                         [](const uint2 &a, const uint2 &b) { return a.y > b.y; });
        QR_CUDA(tg.x.upload(sx), "upload gradient strings");
        QR_CUDA(tg.z.upload(sz), "upload gradient strings");
        QR_CUDA(tg.perm.upload(ord), "upload gradient order");
        QR_CUDA(tg.bat.upload(bat), "upload gradient batches");
        QR_CUDA(tg.wz.upload(wz), "upload gradient strings");
        QR_CUDA(tg.wperm.upload(word), "upload gradient order");
        QR_CUDA(tg.wbat.upload(wb), "upload gradient batches");
        tg.ndirect = nd;
        tg.nbatch = (uint32_t)bat.size();
        tg.nwht = (uint32_t)word.size();
        tg.nwbatch = (uint32_t)wb.size();
        tg.ready = true;
    }
    GradPlanArgs p{};
    p.sx = unplanned ? op->d_mx.as<uint64_t>() : tg.x.as<uint64_t>();
    p.sz = unplanned ? op->d_mz.as<uint64_t>() : tg.z.as<uint64_t>();
    p.batches = tg.bat.as<uint2>();
    p.nbatch = tg.nbatch;
    p.wz = tg.wz.as<uint64_t>();
    p.wbatches = tg.wbat.as<GradBatch>();
    p.nwbatch = tg.nwbatch;
    const uint32_t nd = unplanned ? (uint32_t)op->M : tg.ndirect;
    uint64_t nchunk = 1, nwchunk = 1;
    if (!tiles) {
        nchunk = grad_chunks(nd, op->N, op->nsm);
    } else if (nd > 0) {
        // about 8 batches per SM, chunks of at least 16 tiles
        nchunk = std::min(((uint64_t)op->nsm * 8 + tg.nbatch - 1) / tg.nbatch,
                          (op->N >> 12) * (uint64_t)nstates / 16);
        if (nchunk < 1) nchunk = 1;
    }
    if (tg.nwbatch > 0) {
        // about 4 CTAs per SM, each of at least 8 blocks of 256 rows
        const uint64_t blocks = std::max<uint64_t>(op->N / 256, 1) * (uint64_t)nstates;
        nwchunk = std::min(((uint64_t)op->nsm * 4 + tg.nwbatch - 1) / tg.nwbatch,
                           (blocks + 7) / 8);
    }
    p.direct = GradStrings{unplanned ? nullptr : tg.perm.as<uint32_t>(), nd, (uint32_t)nchunk};
    p.wht = GradStrings{tg.wperm.as<uint32_t>(), tg.nwht, (uint32_t)nwchunk};
    void *scratch = nullptr;
    const size_t np = (size_t)nd * nchunk + (size_t)tg.nwht * nwchunk;
    QR_CUDA(cudaMallocAsync(&scratch, np * sizeof(double2) + 16, st), "term-grad scratch");
    double2 *partial = static_cast<double2 *>(scratch);
    auto *counter = reinterpret_cast<unsigned long long *>(partial + np);
    const uint32_t *mo = op->d_mm_off.as<uint32_t>(), *mt = op->d_mm_terms.as<uint32_t>();
    double2 *o = reinterpret_cast<double2 *>(out);
    const cudaError_t e =
        tiles ? launch_term_grad_tiles(op->N, nstates, p, psi, g, partial, mo, mt,
                                       op->d_ph.as<uint8_t>(), o, counter, op->nsm, st)
              : launch_term_grad(dtype, op->N, nstates, p, psi, g, partial, mo, mt,
                                 op->d_ph.as<uint8_t>(), o, st);
    cudaFreeAsync(scratch, st);
    if (e != cudaSuccess) return cuda_fail(e, "term-grad launch");
    return QR_OK;
}

}  // extern "C"

// tile width of the persistent batched kernel: 512 threads x 8 amplitudes
constexpr int kBatchTileBits = 12;

struct qr_batch {
    static constexpr int kForks = 4;  // parallel branches of the per-operator graph
    int device = 0, nsm = 0;
    std::vector<qr_op *> ops;
    std::vector<int32_t> nstates;
    int tile_bits = 0;
    // 0: one persistent work-list kernel, 1: graph of per-operator kernels,
    // 2: one graph of the persistent kernel for the small operators (fewer
    // work items than half the SMs), the string kernel's batch for those that
    // their own launch would give to it, and one kernel per other operator
    int mode = 0;
    int force_mode = -1;  // -1: the autotuner chooses
    std::vector<char> sel;    // operators in the persistent kernel's work list
    std::vector<char> small;  // operators with fewer items than half the SMs
    std::vector<char> str;    // operators in the string batch's work list
    DevBuf d_ops, d_items, d_ptrs, d_err;
    DevBuf d_sops, d_sitems, d_sctr;  // string batch
    uint32_t nitems = 0, nsitems = 0;
    std::vector<const void *> cur_psi;
    std::vector<void *> cur_y;
    bool ptrs_changed = false;
    std::vector<uint64_t> gens;  // each operator's coef_gen when the graph was made
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaStream_t cap = nullptr;
    cudaStream_t fork[kForks] = {};
    cudaEvent_t fork_ev[kForks + 1] = {};
};

namespace {

// Operator tables and the work list for tile width tb; items are ordered by
// decreasing per-tile work so the persistent CTAs' round-robin balances.
int batch_build(qr_batch *bt, int tb) {
    std::vector<BatchOp> bo(bt->ops.size());
    std::vector<std::pair<double, size_t>> cost;
    for (size_t i = 0; i < bt->ops.size(); ++i) {
        if (!bt->sel[i]) continue;  // applied by its own kernel (modes 1, 2)
        qr_op *op = bt->ops[i];
        int rc = build_plan(op, QR_C64C, 0, tb);
        if (rc) return rc;
        const Plan &pl = op->bplans[tb];
        BatchOp &o = bo[i];
        memset(&o, 0, sizeof(o));
        o.N = op->N;
        o.ntiles = op->N >> pl.b;
        o.b = pl.b;
        o.mcount = pl.amps;
        o.tact = pl.threads;
        o.diag_block = pl.diag_block;
        o.nblocks = pl.nblocks;
        o.nsub = pl.nsub;
        o.nruns = pl.nruns;
        o.nchunks = pl.nchunks;
        o.tdesc = pl.tdesc.as<uint4>();
        o.tdata = pl.tdata.as<TileDataC64>();
        o.blk_hi = pl.blk_hi.as<uint64_t>();
        o.blk_r0 = pl.blk_r0.as<uint32_t>();
        o.run_g0 = pl.run_g0.as<uint32_t>();
        o.run_key = pl.run_key.as<uint32_t>();
        o.chunks = pl.chunks.as<uint4>();
        o.diag = pl.has_diag ? pl.diag.as<float2>() : nullptr;
        // work per output tile: the sub-groups' inner steps plus per-block
        // bookkeeping, over the tile's amplitudes
        cost.push_back({(double)(pl.nsub + 2 * pl.nblocks + 4 * pl.nchunks) * (double)(1u << pl.b),
                        i});
    }
    std::stable_sort(cost.begin(), cost.end(),
                     [](const std::pair<double, size_t> &a, const std::pair<double, size_t> &b) {
                         return a.first > b.first;
                     });
    std::vector<BatchItem> items;
    for (auto &c : cost) {
        const size_t i = c.second;
        for (int32_t st = 0; st < bt->nstates[i]; ++st)
            for (uint64_t q = 0; q < bo[i].ntiles; ++q)
                items.push_back(BatchItem{(uint32_t)i, (uint32_t)st, (uint32_t)q, 0u});
    }
    if (items.size() > 0xffffffffull) return fail(QR_EINVAL, "qr_batch: work list too long");
    bt->nitems = (uint32_t)items.size();
    QR_CUDA(bt->d_ops.upload(bo), "upload batch operators");
    QR_CUDA(bt->d_items.upload(items), "upload batch work list");
    bt->tile_bits = tb;
    return QR_OK;
}

// The string batch's operator table and work list (largest items first).
int str_batch_build(qr_batch *bt) {
    std::vector<StrOp> so(bt->ops.size(), StrOp{});
    std::vector<std::pair<double, size_t>> cost;
    for (size_t i = 0; i < bt->ops.size(); ++i) {
        if (!bt->str[i]) continue;
        // as a launch of its own would
        if (states_overlap(bt->cur_psi[i], bt->cur_y[i],
                           (uint64_t)bt->nstates[i] * bt->ops[i]->N * sizeof(float2)))
            return fail(QR_EINVAL, "qr_batch_apply: psi and y overlap");
        const int rc = build_plan(bt->ops[i], QR_C64C, 0);
        if (rc) return rc;
        const Plan *pl = &bt->ops[i]->plans[QR_C64C][0];
        so[i].sblk = pl->sblk.as<uint4>();
        so[i].ent = pl->ent.as<uint4>();
        so[i].diag = pl->has_diag ? pl->diag.as<float2>() : nullptr;
        so[i].N = bt->ops[i]->N;
        so[i].err = bt->ops[i]->d_err.as<int>();
        so[i].nblk = pl->str.nblk;
        cost.push_back({(double)pl->str.nstr + 2.0 * pl->str.nblk, i});
    }
    std::stable_sort(cost.begin(), cost.end(),
                     [](const std::pair<double, size_t> &a, const std::pair<double, size_t> &b) {
                         return a.first > b.first;
                     });
    std::vector<BatchItem> items;
    for (auto &c : cost) {
        const size_t i = c.second;
        for (int32_t st = 0; st < bt->nstates[i]; ++st)
            for (uint64_t q = 0; q < bt->ops[i]->N >> 12; ++q)
                items.push_back(BatchItem{(uint32_t)i, (uint32_t)st, (uint32_t)q, 0u});
    }
    // the counter runs up to two past the list per CTA
    if (items.size() > 0xfffff000ull) return fail(QR_EINVAL, "qr_batch: work list too long");
    bt->nsitems = (uint32_t)items.size();
    QR_CUDA(bt->d_sops.upload(so), "upload string batch operators");
    QR_CUDA(bt->d_sitems.upload(items), "upload string batch work list");
    QR_CUDA(bt->d_sctr.alloc(sizeof(uint32_t)), "alloc string batch counter");
    return QR_OK;
}

StrBatchArgs str_batch_args(qr_batch *bt) {
    StrBatchArgs a;
    a.ops = bt->d_sops.as<StrOp>();
    a.nops = (uint32_t)bt->ops.size();
    a.items = bt->d_sitems.as<BatchItem>();
    a.nitems = bt->nsitems;
    float2 **pp = bt->d_ptrs.as<float2 *>();
    a.psi = pp;
    a.y = pp + bt->ops.size();
    a.counter = bt->d_sctr.as<uint32_t>();
    a.err = bt->d_err.as<int>();
    a.wait_ns = kDefaultWaitNs;
    a.withhold = -1;
    // test hooks of the operators, read when the graph is made (as a launch of
    // an operator's own reads them)
    for (size_t i = 0; i < bt->ops.size(); ++i) {
        if (!bt->str[i]) continue;
        if (bt->ops[i]->test_wait_ns != 0) a.wait_ns = std::min(a.wait_ns, bt->ops[i]->test_wait_ns);
        a.withhold = std::max(a.withhold, bt->ops[i]->test_withhold);
    }
    return a;
}

BatchArgs batch_args(qr_batch *bt) {
    BatchArgs a;
    a.ops = bt->d_ops.as<BatchOp>();
    a.items = bt->d_items.as<BatchItem>();
    a.nitems = bt->nitems;
    float2 **pp = bt->d_ptrs.as<float2 *>();
    a.psi = pp;
    a.y = pp + bt->ops.size();
    a.err = bt->d_err.as<int>();
    a.wait_ns = kDefaultWaitNs;
    return a;
}

int batch_upload_ptrs(qr_batch *bt, const void *const *psi, void *const *y, cudaStream_t st) {
    const size_t n = bt->ops.size();
    bool same = bt->cur_psi.size() == n;
    for (size_t i = 0; same && i < n; ++i) same = bt->cur_psi[i] == psi[i] && bt->cur_y[i] == y[i];
    if (same) return QR_OK;
    for (size_t i = 0; i < n; ++i) {
        if (!psi[i] || !y[i]) return fail(QR_EINVAL, "qr_batch_apply: null state pointer");
        if ((reinterpret_cast<uintptr_t>(psi[i]) | reinterpret_cast<uintptr_t>(y[i])) & 15)
            return fail(QR_EINVAL, "qr_batch_apply: states must be 16-byte aligned");
    }
    QR_CUDA(cudaStreamSynchronize(st), "qr_batch_apply sync before pointer update");
    std::vector<const void *> h(2 * n);
    for (size_t i = 0; i < n; ++i) {
        h[i] = psi[i];
        h[n + i] = y[i];
    }
    QR_CUDA(cudaMemcpy(bt->d_ptrs.p, h.data(), h.size() * sizeof(void *), cudaMemcpyHostToDevice),
            "upload batch pointers");
    bt->cur_psi.assign(psi, psi + n);
    bt->cur_y.assign(y, y + n);
    bt->ptrs_changed = true;
    return QR_OK;
}

// The batch's graph on the current pointers, on kForks parallel branches:
// the persistent work-list kernel over the selected operators (branch 0),
// one compensated-c64 apply per other operator (round-robin over the
// remaining branches, or all of them when nothing is selected) and, on
// the last branch and behind the persistent kernel, the string batch, whose CTAs
// take work until there is none.  The selected operators' tables
// and work lists (batch_build, str_batch_build) and the other operators'
// plans must already exist.
int capture_graph(qr_batch *bt, cudaGraph_t *graph) {
    cudaStream_t cap = bt->cap;
    bool any_sel = false;
    for (char c : bt->sel) any_sel |= c != 0;
    QR_CUDA(cudaStreamBeginCapture(cap, cudaStreamCaptureModeRelaxed), "begin capture");
    bool any_str = false;
    for (char c : bt->str) any_str |= c != 0;
    cudaError_t e = cudaSuccess;
    if (any_str) e = cudaMemsetAsync(bt->d_sctr.p, 0, sizeof(uint32_t), cap);
    if (e == cudaSuccess) e = cudaEventRecord(bt->fork_ev[qr_batch::kForks], cap);
    for (int k = 0; k < qr_batch::kForks && e == cudaSuccess; ++k)
        e = cudaStreamWaitEvent(bt->fork[k], bt->fork_ev[qr_batch::kForks], 0);
    int rc = QR_OK;
    if (any_sel && e == cudaSuccess) e = launch_batch_c64c(batch_args(bt), bt->nsm, bt->fork[0]);
    const int first = any_sel ? 1 : 0, nbr = qr_batch::kForks - first - (any_str ? 1 : 0);
    int k = 0;
    for (size_t i = 0; i < bt->ops.size() && e == cudaSuccess && !rc; ++i) {
        if (bt->sel[i] || bt->str[i]) continue;
        rc = apply_impl("qr_batch_apply", bt->ops[i], QR_C64C, bt->cur_psi[i], bt->cur_y[i],
                        bt->nstates[i], bt->nstates[i], 0, bt->fork[first + (k++ % nbr)], nullptr, nullptr,
                        nullptr);
    }
    if (any_str && e == cudaSuccess && !rc) {
        // leave the persistent kernel its SMs, and take them over after it
        const uint32_t k = any_sel ? std::min(bt->nitems, (uint32_t)bt->nsm / 2) : 0u;
        e = launch_strings_batch(str_batch_args(bt), (uint32_t)bt->nsm - k,
                                 bt->fork[qr_batch::kForks - 1]);
        if (k > 0 && e == cudaSuccess) e = launch_strings_batch(str_batch_args(bt), k, bt->fork[0]);
    }
    for (int f = 0; f < qr_batch::kForks && e == cudaSuccess; ++f) {
        e = cudaEventRecord(bt->fork_ev[f], bt->fork[f]);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(cap, bt->fork_ev[f], 0);
    }
    cudaError_t e2 = cudaStreamEndCapture(cap, graph);
    if (rc) return rc;
    if (e != cudaSuccess) return cuda_fail(e, "batch graph capture");
    if (e2 != cudaSuccess) return cuda_fail(e2, "end capture");
    return QR_OK;
}

void drop_graph(qr_batch *bt) {
    if (bt->exec) cudaGraphExecDestroy(bt->exec);
    if (bt->graph) cudaGraphDestroy(bt->graph);
    bt->exec = nullptr;
    bt->graph = nullptr;
}

// Select the operators of a mode, build what the graph needs (work list
// and tables of the selected ones, plans of the others, uncaptured) and
// capture and instantiate it.
int instantiate_mode(qr_batch *bt, int mode) {
    drop_graph(bt);
    int rc = QR_OK;
    for (size_t i = 0; i < bt->ops.size() && !rc; ++i) {
        bt->str[i] = 0;
        if (mode != 0) rc = build_plan(bt->ops[i], QR_C64C, 0);
        const Plan &pl = bt->ops[i]->plans[QR_C64C][0];
        // string plans of more than 2^13 rows, whatever a launch of their own would
        // take: the operators share the SMs, so few tiles leave none idle (24
        // operators of 10-18 qubits, four of several strings per group: 1,335 us,
        // 1,347 with those in the persistent kernel)
        if (mode == 2 && !rc)
            bt->str[i] = pl.strings && pl.str.tpb == 1 &&
                         bt->ops[i]->N * (uint64_t)bt->nstates[i] > (1ull << 13);
        bt->sel[i] = mode == 0 ? 1 : (mode == 1 ? 0 : bt->small[i] && !bt->str[i]);
    }
    if (!rc) rc = batch_build(bt, kBatchTileBits);
    if (!rc) rc = str_batch_build(bt);
    if (!rc) rc = capture_graph(bt, &bt->graph);
    if (rc) return rc;
    QR_CUDA(cudaGraphInstantiate(&bt->exec, bt->graph, 0), "graph instantiate");
    bt->mode = mode;
    return QR_OK;
}

uint64_t graph_kernels(const qr_batch *bt) {
    uint64_t k = 0;
    bool any_sel = false, any_str = false;
    for (size_t i = 0; i < bt->ops.size(); ++i) {
        if (bt->sel[i]) any_sel = true;
        else if (bt->str[i]) any_str = true;
        else ++k;
    }
    return k + (any_sel ? 1 : 0) + (any_str ? (any_sel ? 2 : 1) : 0);
}

void record_gens(qr_batch *bt) {
    bt->gens.resize(bt->ops.size());
    for (size_t i = 0; i < bt->ops.size(); ++i) bt->gens[i] = bt->ops[i]->coef_gen;
}

// An operator's coefficients changed since the graph was made: its plan
// tables are rebuilt (outside any capture) and the graph made again.
int refresh_after_coeffs(qr_batch *bt, cudaStream_t st) {
    bool stale = bt->gens.size() != bt->ops.size();
    for (size_t i = 0; !stale && i < bt->ops.size(); ++i)
        stale = bt->gens[i] != bt->ops[i]->coef_gen;
    if (!stale) return QR_OK;
    QR_CUDA(cudaStreamSynchronize(st), "qr_batch_apply sync before plan rebuild");
    int rc = instantiate_mode(bt, bt->mode);
    if (!rc) record_gens(bt);
    return rc;
}

}  // namespace

extern "C" {

int qr_batch_create(int32_t nops, qr_op *const *ops, const int32_t *nstates, qr_batch **out) {
    if (!out || !ops || !nstates || nops < 1) return fail(QR_EINVAL, "qr_batch_create: bad arguments");
    *out = nullptr;
    int dev = -1;
    QR_CUDA(cudaGetDevice(&dev), "cudaGetDevice");
    for (int32_t i = 0; i < nops; ++i) {
        if (!ops[i]) return fail(QR_EINVAL, "qr_batch_create: null operator %d", i);
        if (ops[i]->device != dev)
            return fail(QR_ESTATE, "qr_batch_create: operator %d is on another device", i);
        if (ops[i]->n > 32) return fail(QR_EINVAL, "qr_batch_create: operator %d has n > 32", i);
        if (nstates[i] < 1) return fail(QR_EINVAL, "qr_batch_create: nstates[%d] < 1", i);
    }
    qr_batch *bt = new (std::nothrow) qr_batch();
    if (!bt) return fail(QR_ENOMEM, "qr_batch_create: out of host memory");
    bt->device = dev;
    bt->ops.assign(ops, ops + nops);
    bt->nstates.assign(nstates, nstates + nops);
    cudaError_t e = cudaDeviceGetAttribute(&bt->nsm, cudaDevAttrMultiProcessorCount, dev);
    bt->sel.assign(nops, 1);
    bt->small.assign(nops, 0);
    bt->str.assign(nops, 0);
    for (int32_t i = 0; i < nops; ++i) {
        const int b = std::min(ops[i]->n, kBatchTileBits);
        const uint64_t items = (ops[i]->N >> b) * (uint64_t)nstates[i];
        bt->small[i] = 2 * items <= (uint64_t)bt->nsm ? 1 : 0;
    }
    if (e == cudaSuccess) e = bt->d_ptrs.alloc(2 * (size_t)nops * sizeof(void *));
    if (e == cudaSuccess) e = bt->d_err.alloc(sizeof(int));
    if (e == cudaSuccess) e = cudaMemset(bt->d_err.p, 0, sizeof(int));
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&bt->cap, cudaStreamNonBlocking);
    for (int k = 0; k < qr_batch::kForks && e == cudaSuccess; ++k)
        e = cudaStreamCreateWithFlags(&bt->fork[k], cudaStreamNonBlocking);
    for (int k = 0; k <= qr_batch::kForks && e == cudaSuccess; ++k)
        e = cudaEventCreateWithFlags(&bt->fork_ev[k], cudaEventDisableTiming);
    if (e != cudaSuccess) {
        delete bt;
        return cuda_fail(e, "qr_batch_create");
    }
    *out = bt;
    return QR_OK;
}

int qr_batch_destroy(qr_batch *bt) {
    if (!bt) return QR_OK;
    if (bt->cap) cudaStreamSynchronize(bt->cap);
    drop_graph(bt);
    for (auto &f : bt->fork)
        if (f) cudaStreamDestroy(f);
    for (auto &ev : bt->fork_ev)
        if (ev) cudaEventDestroy(ev);
    if (bt->cap) cudaStreamDestroy(bt->cap);
    delete bt;
    return QR_OK;
}

int qr_batch_tile_bits(const qr_batch *bt) { return bt ? bt->tile_bits : 0; }

int qr_batch_mode(const qr_batch *bt) { return bt && bt->exec ? bt->mode : -1; }

int qr_batch_set_mode(qr_batch *bt, int32_t mode) {
    if (!bt || mode < -1 || mode > 2) return fail(QR_EINVAL, "qr_batch_set_mode: bad arguments");
    if (bt->exec) return fail(QR_ESTATE, "qr_batch_set_mode: the first apply has already chosen");
    bt->force_mode = mode;
    return QR_OK;
}

int qr_batch_apply(qr_batch *bt, const void *const *psi, void *const *y, void *stream) {
    if (!bt || !psi || !y) return fail(QR_EINVAL, "qr_batch_apply: null argument");
    int dev = -1;
    QR_CUDA(cudaGetDevice(&dev), "cudaGetDevice");
    if (dev != bt->device) return fail(QR_ESTATE, "qr_batch_apply: wrong current device");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int rc = batch_upload_ptrs(bt, psi, y, st);
    if (rc) return rc;
    if (bt->exec) {
        rc = refresh_after_coeffs(bt, st);
        if (rc) return rc;
    }
    if (bt->exec && bt->mode != 0 && bt->ptrs_changed) {
        // per-operator graph nodes carry the state pointers: capture again
        rc = instantiate_mode(bt, bt->mode);
        if (rc) return rc;
    }
    bt->ptrs_changed = false;
    if (!bt->exec) {
        // autotuner: time each form on these buffers (one warm-up, three
        // timed launches of its graph) -- the persistent work-list kernel,
        // a graph of one kernel per operator, and, when the batch has both
        // small and large operators, the persistent kernel for the small
        // ones beside per-operator kernels for the large ones
        bool any_small = false, any_large = false;
        for (char c : bt->small) (c ? any_small : any_large) = true;
        std::vector<int> cands;
        if (bt->force_mode >= 0) cands.push_back(bt->force_mode);
        else {
            cands = {0, 1};
            if (any_small && any_large) cands.push_back(2);
        }
        int best = -1;
        float best_ms = 0.f;
        cudaEvent_t e0, e1;
        QR_CUDA(cudaEventCreate(&e0), "event");
        QR_CUDA(cudaEventCreate(&e1), "event");
        for (int m : cands) {
            rc = instantiate_mode(bt, m);
            if (rc) break;
            if (cands.size() == 1) {
                best = m;
                break;
            }
            cudaError_t e = cudaGraphLaunch(bt->exec, bt->cap);
            if (e == cudaSuccess) e = cudaEventRecord(e0, bt->cap);
            for (int k = 0; k < 3 && e == cudaSuccess; ++k) e = cudaGraphLaunch(bt->exec, bt->cap);
            if (e == cudaSuccess) e = cudaEventRecord(e1, bt->cap);
            if (e == cudaSuccess) e = cudaEventSynchronize(e1);
            float ms = 0.f;
            if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
            if (e != cudaSuccess) {
                rc = cuda_fail(e, "qr_batch autotune");
                break;
            }
            if (best < 0 || ms < best_ms) {
                best = m;
                best_ms = ms;
            }
        }
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        if (rc) return rc;
        if (bt->mode != best) {
            rc = instantiate_mode(bt, best);
            if (rc) return rc;
        }
        bt->tile_bits = kBatchTileBits;
        record_gens(bt);
        QR_CUDA(cudaStreamSynchronize(bt->cap), "autotune sync");
        int h = 0;
        QR_CUDA(cudaMemcpy(&h, bt->d_err.p, sizeof(int), cudaMemcpyDeviceToHost), "error word");
        if (h) return fail(QR_EKERNEL, "batched kernel reported error %d", h);
        for (qr_op *op : bt->ops) {
            rc = check_kernel_error(op);
            if (rc) return rc;
        }
    }
    QR_CUDA(cudaGraphLaunch(bt->exec, st), "graph launch");
    count_launch(graph_kernels(bt));  // kernels the graph runs
    return QR_OK;
}

int qr_last_error(char *buf, size_t len) {
    const int L = (int)g_err.size();
    if (buf && len > 0) {
        size_t c = std::min(len - 1, g_err.size());
        memcpy(buf, g_err.data(), c);
        buf[c] = '\0';
    }
    return L;
}

uint64_t qr_launch_count(void) { return g_launches.load(std::memory_order_relaxed); }

}  // extern "C"
