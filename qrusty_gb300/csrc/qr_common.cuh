// qr_common.cuh -- internal types shared by the host layer and the kernels
// of libqrusty_gpu (not part of the public C ABI in include/qrusty_gpu.h).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace qr {

// Largest rank of a group's z-difference span that qr_apply evaluates with
// a 2^d-entry table; groups above it are evaluated term by term ("fat").
constexpr int kDMax = 4;
constexpr uint32_t kFat = 0xffffffffu;

// One x-group (or a piece of one) of a rows plan (qr_apply_rows.cu).  All terms of the group share the x mask;
// their z masks are z0 ^ delta_k with delta_k in span(beta[0..d)).  The
// group's diagonal factor at row r is
//   D(r) = (-1)^popc(r & z0) * table[off + pi(r)],  pi(r)_i = popc(r & beta_i) & 1.
// Fat groups (d == kFat) list their cnt terms at fat_z/fat_c[off ...].
struct alignas(16) GroupDesc {
    uint64_t z0;
    uint64_t beta[kDMax];
    uint64_t x;
    uint32_t d;     // rank, or kFat
    uint32_t off;   // table offset (entries) or fat-term offset
    uint32_t cnt;   // fat-term count
    uint32_t pad;
};
static_assert(sizeof(GroupDesc) == 64, "GroupDesc layout");

template <typename Real> struct Cplx;
template <> struct alignas(8) Cplx<float> { float re, im; };
template <> struct alignas(16) Cplx<double> { double re, im; };

// Per-sub-group data of the per-tile table of the compensated-c64 kernel:
// the masks' tile-index parts (>> b) and the FP32 table T[u] of the factor.
struct alignas(16) TileDataC64 {
    uint64_t z0h, b0h, b1h;
    uint64_t role;  // coset plans: 0, or a merged pair's (kMerged...)
    float2 T[4];
};
enum : uint64_t { kMergedBasis = 1, kMergedSign = 2, kMergedSecond = 3 };
static_assert(sizeof(TileDataC64) == 64, "TileDataC64 is read as four 16-byte words");

// String plans: consumer threads, strings per block, CTAs per cluster at most.
constexpr uint32_t kStrThreads = 512, kStrEntCap = 255, kStrMaxSplit = 8;

// qubits from which a block holds two partner tiles and tiles are not split
constexpr int kStrPairN = 19;
struct StrSplit {
    uint32_t nblk = 0, nstr = 0, tpb = 1;  // blocks, strings, partner tiles per block
    uint32_t part[kStrMaxSplit][kStrMaxSplit + 1] = {};
};

struct ApplyArgs {
    const void *psi;
    void *y;
    uint64_t N;             // 2^n amplitudes per state
    int n;
    int b;                  // tile bits
    int tb;                 // log2(threads)
    int nstates;
    uint64_t ntiles;        // N >> b
    uint64_t nitems;        // nstates * ntiles
    const GroupDesc *groups;
    uint32_t ngroups;
    const void *tables;     // Cplx<Real>
    const uint64_t *fat_z;
    const void *fat_c;      // Cplx<Real>
    const uint64_t *blk_hi; // partner-tile XOR per block
    uint32_t nblocks;
    const void *diag;       // Cplx<Real>[N] or null (only read in block hi == 0)
    int diag_block;         // index of the hi == 0 block, or -1
    int *err;               // device error word
    // compensated-c64 plan: sub-groups (see qr_apply.cu)
    uint32_t nsub;
    // per-tile-table kernel: per sub-group a 16-byte thread descriptor
    // {partner byte-offset XOR | tvar << 31, z0_t, beta0_t, beta1_t} (the
    // thread-bit parts of z0 and of the basis) and its TileDataC64;
    // sub-groups of a block in runs of equal key
    const uint4 *tdesc;
    const TileDataC64 *tdata;
    const uint32_t *blk_r0;   // runs of block j: [blk_r0[j], blk_r0[j+1])
    const uint32_t *run_g0;   // sub-groups of run r: [run_g0[r], run_g0[r+1])
    const uint32_t *run_key;  // key = zm | xm << 4 | tv << 5 (factor depends on the thread)
    uint32_t nruns;
    // chunks of consecutive blocks with at most kTabCap sub-groups:
    // {first sub-group, first run, first block, 0}, nchunks + 1 entries
    const uint4 *chunks;
    uint32_t nchunks;
    // string plans (qr_apply_strings.cu): nsblk blocks of one or two partner
    // tiles, {XOR of tile 0, of tile 1 (or ~0), first 16-byte entry, strings};
    // a block's entries are a header {strings, diagonal flag} and one per
    // string; rank r of a cluster takes blocks [part[r], part[r + 1])
    const uint4 *ent, *sblk;
    uint32_t nsblk;
    uint32_t part[kStrMaxSplit + 1];
    // coset plans (qr_apply_cosets.cu): blocks {XOR of tile 0, of tile 1 (or
    // ~0), first sub-group | lone uniform ones << 10 | cheap << 30 | diagonal
    // << 31, lone ones by thread | quads << 10 | others << 16}; per sub-group
    // {partner offset within the slot | new loads << 16 | key << 17 | merged
    // pair << 24, thread parts of z0, beta0, beta1} and its tile data
    const uint4 *cblk, *ctdesc;
    const TileDataC64 *ctdata;
    uint32_t ncblk, ncsub;
    // fused epilogue y = alpha * (H psi) + beta * v when v != nullptr
    const void *v;
    double ar, ai, br, bi;
    // bound of every mbarrier wait (ns); 2 s unless a test shortens it
    uint64_t wait_ns;
    // test hook (qr_op_set_test_hooks): the ring step whose partner-tile copy
    // CTA 0 never issues, so that its wait runs out; -1 = none
    int64_t withhold;
    // 64-bit row words (the n > 32 instantiations) forced at any n (test hook)
    int wide;
};



// One operator of a batched compensated-c64 launch (device copy): the
// per-tile-table plan of the operator and its tile geometry.
struct BatchOp {
    uint64_t N, ntiles;
    int32_t b, mcount, tact, diag_block;  // tile bits, amplitudes / threads used, x = 0 block
    uint32_t nblocks, nsub, nruns, nchunks;
    const uint4 *tdesc;
    const TileDataC64 *tdata;
    const uint64_t *blk_hi;
    const uint32_t *blk_r0, *run_g0, *run_key;
    const uint4 *chunks;
    const float2 *diag;
};
struct BatchItem {
    uint32_t op, state, tile, pad;
};
struct BatchArgs {
    const BatchOp *ops;
    const BatchItem *items;  // sorted by decreasing work per tile
    uint32_t nitems;
    const float2 *const *psi;  // per operator: its first state; state s at + s * N
    float2 *const *y;
    int *err;
    uint64_t wait_ns;          // bound of every mbarrier wait
};
cudaError_t launch_batch_c64c(const BatchArgs &a, int nsm, cudaStream_t st);

// One entry of a plan's coefficient program (qr_op_set_coeffs_device): the
// value(s) at dst computed from merged strings [m0, m0 + cnt) of the plan's
// coefficients c_m (the merged coefficients, or for an adjoint plan
// conj(c_m) (-1)^popc(x_m & z_m)).  kind 0: 2^d FP32 table entries (float2),
// entry u = the fold from 0 of +-c_m in member order, sign (-1)^popc(u &
// coord_m); kind 1: the same in FP64 (double2); kind 2: c_m itself (double2,
// cnt = 1).  The additions are those of the host plan builder, in its order.
struct CoefSlot {
    uint64_t dst;
    uint32_t m0;
    uint16_t cnt;
    uint8_t d, kind;
};
static_assert(sizeof(CoefSlot) == 16, "CoefSlot layout");

// qr_coef.cu
cudaError_t launch_merge_coeffs(uint32_t M, const uint32_t *mm_off, const uint32_t *mm_terms,
                                const double2 *coeff, const uint8_t *phase, double2 *mc,
                                cudaStream_t st);
cudaError_t launch_coef_program(const CoefSlot *slots, uint32_t nslots, int ebits,
                                const uint32_t *mem, const uint8_t *coord, const double2 *mc,
                                const uint8_t *madj, int adjoint, cudaStream_t st);

// c'_k = m(phase_k) * c_k (make_params, qrusty/src/accel.rs:141-157):
// m = (1, -i, -1, +i)[phase], num-complex's product (ar br - ai bi,
// ar bi + ai br) with every operation rounded on its own (no FMA).
__device__ __forceinline__ double2 make_param(double2 b, uint32_t phase) {
    const uint32_t ph = phase & 3u;
    const double ar = ph == 0 ? 1.0 : (ph == 2 ? -1.0 : 0.0);
    const double ai = ph == 1 ? -1.0 : (ph == 3 ? 1.0 : 0.0);
    return make_double2(__dsub_rn(__dmul_rn(ar, b.x), __dmul_rn(ai, b.y)),
                        __dadd_rn(__dmul_rn(ar, b.y), __dmul_rn(ai, b.x)));
}

// Device error codes written to the error word.
enum : int { kErrNone = 0, kErrMbarTimeout = 1, kErrCsrPos = 2 };

// num-complex 0.4 arithmetic with every operation an explicit round-to-nearest
// intrinsic (no FMA contraction): a * b = (ar br - ai bi, ar bi + ai br).
// a*x + b*y is the axpby of qrusty/src/accel.rs:374-379.
__device__ __forceinline__ double2 cx_axpby(double ar, double ai, double2 x, double br, double bi,
                                            double2 y) {
    const double ur = __dsub_rn(__dmul_rn(ar, x.x), __dmul_rn(ai, x.y));
    const double ui = __dadd_rn(__dmul_rn(ar, x.y), __dmul_rn(ai, x.x));
    const double vr = __dsub_rn(__dmul_rn(br, y.x), __dmul_rn(bi, y.y));
    const double vi = __dadd_rn(__dmul_rn(br, y.y), __dmul_rn(bi, y.x));
    return make_double2(__dadd_rn(ur, vr), __dadd_rn(ui, vi));
}
__device__ __forceinline__ float2 cx_axpby(float ar, float ai, float2 x, float br, float bi,
                                           float2 y) {
    const float ur = __fsub_rn(__fmul_rn(ar, x.x), __fmul_rn(ai, x.y));
    const float ui = __fadd_rn(__fmul_rn(ar, x.y), __fmul_rn(ai, x.x));
    const float vr = __fsub_rn(__fmul_rn(br, y.x), __fmul_rn(bi, y.y));
    const float vi = __fadd_rn(__fmul_rn(br, y.y), __fmul_rn(bi, y.x));
    return make_float2(__fadd_rn(ur, vr), __fadd_rn(ui, vi));
}

// sub-groups of one per-tile factor table of the compensated-complex64 kernel
constexpr uint32_t kTabCap = 512;

// log2 of the thread count of the compensated-complex64 kernels (the
// single-operator kernels and the batched kernel, see qr_apply.cu).
constexpr int kC64ThreadBits = 9;

// Records msg as the calling thread's last error (qr_last_error) and returns code.
int set_error(int code, const char *msg);

// Per-process launch counter (all launches issued through this library).
void count_launch(uint64_t k = 1);

// cudaFuncSetAttribute(MaxDynamicSharedMemorySize) for kernel fn on the
// current device, only when `bytes` exceeds what was set before: steady-state
// launches (and launches inside a stream capture) make no attribute calls.
cudaError_t ensure_dyn_smem(const void *fn, size_t bytes);

// Kernel launchers (qr_apply.cu / qr_csr.cu).
cudaError_t launch_apply(const ApplyArgs &a, int amps, int threads, int nsm,
                         cudaStream_t st);
// Batched string operators (apply_c64c_strings_batch): n >= 12, one partner
// tile per block.
struct StrOp {
    const uint4 *sblk, *ent;
    const float2 *diag;  // or null
    uint64_t N;
    int *err;            // the operator's error word (null: not in the work list)
    uint32_t nblk;
};
struct StrBatchArgs {
    const StrOp *ops;         // by operator of the batch
    uint32_t nops;
    const BatchItem *items;   // largest first
    uint32_t nitems;
    const float2 *const *psi;
    float2 *const *y;
    uint32_t *counter;
    int *err;
    uint64_t wait_ns;
    int64_t withhold;         // test hook: ring step of CTA 0 never issued, -1 = off
};
// The counter is zeroed before; launches that share it share the items.
cudaError_t launch_strings_batch(const StrBatchArgs &a, uint32_t ctas, cudaStream_t st);

// qr_apply_strings.cu
// call_items: output tiles of the caller's whole call
cudaError_t launch_c64c_strings(const ApplyArgs &a, const StrSplit &sp, uint64_t call_items,
                                int nsm, cudaStream_t st);
// qr_apply_cosets.cu
constexpr size_t kCosetSmem = 227u * 1024u - 256u;  // dynamic shared memory, at most
size_t coset_smem_bytes(uint32_t nsub, uint32_t nblk, uint32_t slots, uint32_t ntab);
cudaError_t launch_c64c_cosets(const ApplyArgs &a, int nsm, cudaStream_t st);
// qr_apply_rows.cu
// call_rows: rows of the caller's whole call, which the split over warps follows
cudaError_t launch_rows(int dtype, const ApplyArgs &a, uint64_t call_rows, cudaStream_t st);
cudaError_t launch_diag(int dtype, int n, int db, uint64_t ntiles, const uint64_t *bin_zlo,
                        const uint32_t *bin_off, uint32_t nbins, const uint64_t *tz,
                        const double *tc, void *out, cudaStream_t st);

// CSR fill.  Per group g (x masks ascending): the sigma values of its
// position formula, and either a class table -- the term-order fold of
// the group's +-c'_k for each of the 2^(d+1) sign classes of a row, class
// bit 0 = parity(r & z0), bit j+1 = parity(r & beta_j) -- or, when the z
// span has rank > kCsrMaxRank, the term range to fold per row.
constexpr int kCsrMaxRank = 4;
constexpr uint32_t kCsrFold = 0xffffffffu;
// Fold-mode groups: the longest leading run of terms whose z differences span
// a bounded rank is folded per class once (table of 2^(rank+1) entries); rows
// add only the terms after it.  The tables are computed anew by every
// coefficient update, so the larger rank serves operators of few such groups
// and rows enough to pay it back.  Measured, rank 10 / 12 (us, build and
// coefficient update): chain n = 21 (one group) 377 / 358 and 19 / 27, n = 14
// 11.8 / 11.8 and 20 / 31; Jordan-Wigner n = 12 (66 groups) 75 / 13 and 29 /
// 246; 200 groups n = 16 1,174 / 1,064 and 54 / 190; 2,000 groups n = 12 656 /
// 279 and 386 / 3,745 (first build 1,269 / 4,576, tables 64 / 256 MB).  With
// rank 14 the chain's and a Jordan-Wigner operator's rows miss L1.
constexpr int kCsrPrefixRank = 12, kCsrPrefixRankMany = 10;
constexpr int kCsrDeepFolds = 8, kCsrDeepN = 16;  // at most, at least, for the larger rank
struct CsrGroup {
    uint64_t z0;
    uint64_t beta[kCsrMaxRank];
    uint32_t d;       // rank of the z differences, or kCsrFold
    uint32_t tab;     // first class-table entry (2^(d+1) entries)
    uint32_t zparts;  // fold mode: bit 0 every c'_k.re is +-0, bit 1 every c'_k.im is +-0
    uint32_t pre;     // fold mode: prefix terms (bits 0-23) folded per class, prefix rank << 24
    uint32_t k0, k1;  // terms [k0, k1) in group-stable order (fold mode)
};
static_assert(sizeof(CsrGroup) == 64, "CsrGroup layout");

struct CsrArgs {
    uint64_t N, G;
    int n;                    // qubits: row bits
    const uint64_t *gx;       // G, ascending
    const CsrGroup *grp;      // G
    const uint64_t *pmask;    // G: bits b with a nonzero sigma_{g,b}
    const int32_t *sig;       // G x n: sigma_{g,b} (0 where b is not in pmask)
    const uint16_t *tables;   // position and class terms by row bits (G <= 256)
    const uint32_t *fold;     // groups in fold mode
    uint32_t nfold;
    const double2 *ctab;      // class tables
    uint32_t nctab;           // class-table entries
    const uint64_t *tz;       // terms in group-stable order (fold mode)
    const double *tc;         // 2 doubles per term
    const uint64_t *pbeta;    // nfold x kCsrPrefixRank: prefix span bases (fold mode; zeros after)
    const double2 *ptab;      // prefix class tables (fold mode)
    double2 *fvals;           // nfold x nrows fold-mode values, or null (written in place)
    int inline_fold;          // fold-mode entries folded by the staged fill (fvals null)
    uint64_t *indptr, *indices;
    double *data;
    uint64_t row0, nrows;     // rows to fill
    int *err;                 // device error word (bad position => kErrCsrPos)
    int wide;                 // 64-bit row words (the n > 32 kernels) forced (test hook)
};
cudaError_t launch_csr_fill(const CsrArgs &a, int nsm, cudaStream_t st);
// Whether the staged fill folds nfold fold-mode groups of at most fold_rem
// terms past their prefix itself (no value buffer).
bool csr_inline_fold(uint64_t G, int n, uint32_t nfold, uint32_t fold_rem);
// The staged fill's mask tables (a.tables, csr_tables_bytes), once per operator.
size_t csr_tables_bytes(uint64_t G, int n);
cudaError_t launch_csr_tables(const CsrArgs &a, cudaStream_t st);

// qr_group.cu: term grouping on the device.  Buffers sized for T terms (the
// group counts are bounded by T).
struct TermGroupsOut {
    uint32_t *order;     // T: input index of each term, stably sorted by x (CSR order)
    uint64_t *tz;        // T: z of the terms in CSR order
    uint64_t *gx;        // G: distinct x, ascending
    uint32_t *goff;      // G + 1: CSR group g = terms [goff[g], goff[g + 1]) in CSR order
    uint32_t *mmap;      // T: merged string of each input term
    uint32_t *mm_off;    // M + 1: merged string m folds terms mm_terms[mm_off[m] ..]
    uint32_t *mm_terms;  // T: input indices, per merged string in input order
    uint64_t *mx, *mz;   // M: merged strings, first-occurrence order
    uint8_t *madj;       // M: popc(x & z) & 1 (adjoint sign)
    uint32_t *ag_off;    // Ga + 1: x-groups of the merged strings (first-occurrence order)
    uint32_t *ag_mem;    // M: merged indices per x-group, ascending
};
struct TermGroupCounts {
    uint64_t G = 0, M = 0, Ga = 0;
};
// Synchronises st; returns the counts.
cudaError_t group_terms(int n, uint64_t T, const uint64_t *x, const uint64_t *z,
                        const TermGroupsOut &o, TermGroupCounts *cnt, cudaStream_t st);

struct CsrStructOut {
    uint64_t *pmask;  // G
    int32_t *sig;     // G x n
    CsrGroup *grp;    // G
    uint16_t *coord;  // T: span coordinates of each term (CSR order)
    uint32_t *fold;   // <= G: fold-mode groups
    uint64_t *pbeta;  // <= G x kCsrPrefixRank
};
struct CsrStructCounts {
    uint64_t nctab = 0, nptab = 0;
    uint32_t nfold = 0;
    uint32_t fold_rem = 0;  // fold-mode groups: most terms past the prefix
};
// Mask-only CSR tables; synchronises st and returns the table sizes.
cudaError_t csr_structure(int n, uint64_t G, const uint64_t *gx, const uint32_t *goff,
                          const uint64_t *tz, const CsrStructOut &o, CsrStructCounts *cnt,
                          cudaStream_t st);
// Coefficient-dependent CSR tables (tc, zero-part flags, class and prefix
// tables) from the raw coefficients: stream-ordered, no synchronisation.
cudaError_t csr_values(uint64_t G, uint64_t T, const uint32_t *order, const double2 *coef,
                       const uint8_t *phase, double2 *tc, CsrGroup *grp, const uint16_t *coord,
                       double2 *ctab, double2 *ptab, bool has_fold, cudaStream_t st);
cudaError_t launch_csr_spmv(uint64_t nrows, uint64_t ncols, const uint64_t *indptr,
                            const uint64_t *indices, const double *data, const double *v,
                            double *y, int nsm, cudaStream_t st);

// qr_vec.cu (op: 0 axpby, 1 axpy, 2 ax, 3 precond2)
cudaError_t launch_vec_op(int op, int f32, uint64_t len, const void *x, const void *y, void *z,
                          const double *a, const double *b, double tol, int nsm, cudaStream_t st);
cudaError_t launch_csr_diag(uint64_t nd, const uint64_t *indptr, const uint64_t *indices,
                            const double *data, double *out, int nsm, cudaStream_t st);
cudaError_t launch_op_diag(uint64_t N, uint32_t nt, const uint64_t *tz, const double *tc, void *out,
                           int f32, int nsm, cudaStream_t st);

// qr_reduce.cu
uint32_t vdot_blocks(uint64_t N, int nsm);
cudaError_t launch_vdot(int dtype, uint64_t N, const void *a, const void *b, int nstates,
                        double2 *partial, uint32_t nblk, double2 *out, cudaStream_t st);
// Term gradients.  complex128 strings of x groups of kGradWhtMin or more go through a
// Walsh-Hadamard transform per 256 rows (wht: batches of up to kGradWhtBatch
// strings of one x), the others one by one (direct: by partner tile x >> 12 for
// the tiled complex64 kernel, n >= 12).  perm: merged index of each (null: in
// merged order); partial
// sums: direct.count x direct.nchunk, then wht.count x wht.nchunk.
constexpr uint32_t kGradWhtMin = 8, kGradWhtBatch = 256;
// Rows, passed over by each SM with four strings, that the transform has to save
// to pay for its launch (us, all strings one by one / with the transform, one
// state and eight): Jordan-Wigner n = 8 17 / 27 and 28 / 44, 300 Z strings n =
// 12 (saves none: one round of blocks in both) 33 / 51 and 151 / 169, n = 13 (two
// rounds or one) 52 / 51 and 283 / 169, H6 74 / 70 and 421 / 339.
constexpr uint64_t kGradWhtRows = 4096;
struct GradBatch {
    uint64_t x;
    uint32_t first, count;
};
struct GradStrings {
    const uint32_t *perm;
    uint32_t count, nchunk;
};
struct GradPlanArgs {
    GradStrings direct, wht;
    const uint64_t *sx, *sz;  // direct strings
    const uint2 *batches;     // tiled kernel: <= 8 strings of one partner tile (first, count)
    uint32_t nbatch;
    const uint64_t *wz;       // wht strings
    const GradBatch *wbatches;
    uint32_t nwbatch;
};
cudaError_t launch_term_grad(int dtype, uint64_t N, int nstates, const GradPlanArgs &p,
                             const void *psi, const void *g, double2 *partial,
                             const uint32_t *mm_off, const uint32_t *mm_terms,
                             const uint8_t *phase, double2 *out, cudaStream_t st);
// complex64, n >= 12.  counter: 8 bytes of device scratch (the work counter)
cudaError_t launch_term_grad_tiles(uint64_t N, int nstates, const GradPlanArgs &p,
                                   const void *psi, const void *g, double2 *partial,
                                   const uint32_t *mm_off, const uint32_t *mm_terms,
                                   const uint8_t *phase, double2 *out,
                                   unsigned long long *counter, int nsm, cudaStream_t st);

}  // namespace qr
