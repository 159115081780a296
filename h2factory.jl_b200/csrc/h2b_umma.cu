// B1 dense I2O of the FP32 form on the fifth-generation tensor cores (tcgen05, kind::tf32).
//
// Per receiving node r: l_r = sum over its pairs of op(B_pair) m_src (translateintonode!,
// src/farinteractions/traversalhelpers.jl:167-219, with the dense applycouplingkernel! of
// src/farinteractions/i2otranslations/i2otranslationcollection.jl:367-409 and the orientation rule
// of i2oprotocol.jl:87-92). For one receiver this is one GEMM whose K dimension runs over the
// concatenated pairs: D[nc x nq] = [op(B_1) op(B_2) ...] [m_1; m_2; ...].
//
// One CTA per (receiver, 128-row tile of its coefficients, tile of right-hand sides), one CTA per
// SM, warp-specialised; the K dimension streams in chunks of 32 FP32 values through UM_NS stages,
// and every hand-off is an mbarrier (no block barrier inside the loop):
//   * coupling warps (0-3), one thread per tile row: each warp bulk-copies (cp.async.bulk) a
//     quarter of the stored columns that chunk c + 3 reads (column kmap[k] of the pair's block:
//     the column permutation of a symmetry-reduced pair is which column is fetched) into a
//     shared-memory ring; every thread then reads its row of the chunk (rowmap applied by the row
//     it reads), splits the 32 values into TF32 high parts and rounded remainders and writes them
//     into a tensor-memory stage with tcgen05.st. The MMAs take this operand (A) straight from
//     tensor memory. Couplings without whole 16-byte columns are read row by row from global
//     memory into a register ring instead;
//   * moment warps (4-6), every third chunk each: cp.async the chunk's source moments into a raw
//     shared-memory stage a turn ahead, then write them as the B operand, TF32 high parts plus
//     remainders, in the canonical no-swizzle K-major layout (a complex piece is split once for its
//     two rows). All three on every chunk, joined by a named barrier, they were what the kernel
//     waited for: 10,931 points, p = 6 real, 12 right-hand sides, I2O 5.68 -> 4.82 ms (4.45 with the
//     longest interaction lists first);
//   * one MMA warp (warp 11): per 8-wide k step the products hi*hi + hi*lo + lo*hi (the lo*lo
//     term is below FP32 rounding), N = 64 columns each, into an FP32 accumulator in tensor memory;
//     one commit per chunk releases both operand stages;
//   * drain warps (7-10, one per tensor-memory lane quarter): the tensor cores round each
//     accumulation toward zero, so one FP32 accumulator over a whole interaction list loses ~1e-4;
//     accumulators live for 64 values of K (2 chunks) only, two alternate, and each finished one is
//     added into an FP64 sum in tensor memory, which the epilogue rounds once into the FP32 moments.
//
// Complex maps run as real GEMMs: with B = Br + i Bi and m = mr + i mi,
//   [Re l | Im l] = [Br Bi] (interleaved along k) x [[mr, mi]; [-mi, mr]] (interleaved rows),
// so the coupling's interleaved (re, im) storage is the A operand as it lies in memory and each
// moment value feeds two B rows (Re rows (mr, -mi), Im rows (mi, mr)). Adjoint maps conjugate B;
// symmetry-reduced couplings apply their row / column permutations in which rows and columns are
// read. FP32 dense couplings are also stored transposed, so every orientation copies columns.
//
// Every wait on an mbarrier is bounded: a wait that gives up counts itself in a device counter
// (h2b_tensor_wait_timeouts) and sets the CTA's abort flag; every role then leaves its loop, the
// MMA warp waits (with the full bound) for the products it issued, the moment warps for their
// copies, and the CTA frees its tensor memory and returns with its output tile unwritten.

#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>

#include "h2b_internal.cuh"

namespace h2b {

namespace {

constexpr int UM_M = 128;         // output rows per tile = tensor-memory lanes
constexpr int UM_KC = 32;         // FP32 K values per chunk: 8 groups of 16 bytes per B row
constexpr int UM_KG = UM_KC / 4;
constexpr int UM_NS = 4;          // operand stages: coupling in tensor memory, moments in shared memory
constexpr uint32_t UM_RAWROW = UM_KC * 4 + 16;  // raw moment row: one chunk's values + 16 bytes of padding
// chunks per accumulation segment: 64 values of K are summed in FP32 (the tensor cores' own
// rounding) before the segment is added to the FP64 sum (measured on the 65,536-point sphere:
// relative error 3.4e-7 at 64 values, 6.5e-7 at 128, 1.2e-6 at 256; time +1 % per halving)
constexpr int UM_SEG = 64 / UM_KC;
// Every hand-off between the roles costs a fixed few hundred cycles whatever the chunk holds
// (measured: with the products removed the kernel ran almost as fast as with them; 32-wide chunks
// ran 27 % faster than 16-wide ones), so chunks are as wide as the tensor-memory and shared-memory
// stages allow.
constexpr int UM_AR = 4;          // coupling column stages in shared memory (bulk-copy path)
constexpr int UM_AI = 4;          // warps that issue a chunk's column copies (KQ / UM_AI columns each)
constexpr int UM_ALA = 3;         // coupling columns copied this many chunks ahead
// 4 coupling, 3 moment, 4 drain, 1 MMA: twelve warps place three on each SM sub-partition, whose
// 16K registers then allow up to 170 per thread (a thirteenth warp would cap them at 128)
constexpr int UM_WARPS = 12;
constexpr int UM_BW = 3;           // moment warps
constexpr int UM_RS = 2 * UM_BW;   // raw moment stages, two per moment warp
constexpr int UM_THREADS = UM_WARPS * 32;
constexpr int UM_NT_MAX_REAL = 64;    // right-hand sides per tile, real maps (MMA N = 64)
constexpr int UM_NT_MAX_CPLX = 32;    // complex maps: Re and Im rows make MMA N = 64
constexpr uint32_t UM_LBO = 128;            // bytes between the two 16-byte K halves of a k step
constexpr uint32_t UM_SBO = UM_KG * 128;    // bytes between 8-row groups (4 groups of 128 bytes)
constexpr int UM_STATIC = 1024;  // bound on the kernel's static shared arrays (384 bytes), bytes
constexpr unsigned UM_SUSPEND_NS = 1000;   // suspend-time hint of one try_wait attempt
constexpr unsigned UM_SPIN = 1u << 20;      // default attempts before a wait gives up (about a second)
constexpr unsigned UM_SPIN_FINAL = 1u << 23;  // the final wait for products already issued

__device__ unsigned int g_umma_timeouts = 0;
__device__ unsigned int g_umma_wait_limit = UM_SPIN;

__device__ __forceinline__ int um_ncoef(const DSide &s, int lvl) {
    return s.shape[3 * lvl] * s.shape[3 * lvl + 1] * s.shape[3 * lvl + 2];
}

__device__ __forceinline__ uint32_t su32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Shared-memory matrix descriptor (tcgen05): start address, leading (K) and stride (M/N) byte
// offsets in 16-byte units, version 1 at bits 46-47, no swizzle.
__device__ __forceinline__ uint64_t kmajor_desc(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(UM_LBO >> 4) << 16) |
           ((uint64_t)(UM_SBO >> 4) << 32) | (1ull << 46);
}

// Instruction descriptor, kind::tf32: FP32 accumulator (bits 4-5 = 1), A and B TF32 (bits 7-9 and
// 10-12 = 2), both K-major, N >> 3 at bits 17-22, M >> 4 at bits 24-28.
__device__ __forceinline__ uint32_t tf32_idesc(int mrows, int ncols) {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(ncols >> 3) << 17) |
           ((uint32_t)(mrows >> 4) << 24);
}

// byte offset of the 16-byte group (row, kg) in a no-swizzle K-major tile of 16-wide rows
__device__ __forceinline__ uint32_t goff(int row, int kg) {
    return (uint32_t)(row >> 3) * UM_SBO + (uint32_t)kg * UM_LBO + (uint32_t)(row & 7) * 16u;
}

// nearest TF32 value (10 explicit mantissa bits, ties away from zero) as FP32 bits with the 13 low
// mantissa bits cleared: add half of their range to the magnitude, then clear them. Moments and
// couplings are finite and far below the overflow edge. (cvt.rna.tf32 is one instruction but shares a
// 16-lane pipe with the drain warps' FP32 -> FP64 conversions: 5 % slower here.)
__device__ __forceinline__ uint32_t tf32_bits(float a) {
    return (__float_as_uint(a) + 0x1000u) & 0xFFFFE000u;
}

// x = hi + lo with hi, lo TF32: the high part and the rounded remainder
__device__ __forceinline__ void split2(float x, uint32_t &hi, uint32_t &lo) {
    hi = tf32_bits(x);
    lo = tf32_bits(x - __uint_as_float(hi));
}

// four rows {r0 .. r3} of a tensor map, from x on, into this CTA's shared memory
__device__ __forceinline__ void tma_gather4(uint32_t dst, const CUtensorMap *map, int x, int4 r, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes [%0], "
        "[%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dst),
        "l"(map), "r"(x), "r"(r.x), "r"(r.y), "r"(r.z), "r"(r.w), "r"(su32(bar))
        : "memory");
}

// One lane of a converged warp, as a predicate for the two calls below. The whole warp runs the issuing
// loop and only the instruction is predicated: its operands then stay in uniform registers, and a
// product costs 10 cycles to issue (32 at N = 64, the tensor cores' own rate) against 45 from a branch
// that one lane took (measured, M = 128, tensor-memory A).
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}\n" : "=r"(e));
    return e;
}
// D (+)= A (tensor memory) * B (shared memory), kind::tf32, and the commit of the products so far.
__device__ __forceinline__ void umma_ts_if(uint32_t elected, uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc,
                                           uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %6, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}\n" ::"r"(tmem_d),
        "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u), "r"(elected));
}
__device__ __forceinline__ void umma_commit_if(uint32_t elected, uint64_t *bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}\n" ::"r"(su32(bar)),
        "r"(elected)
        : "memory");
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(su32(bar)), "r"(bytes) : "memory");
}

// bulk copy global -> this CTA's shared memory, completing `bytes` of the barrier's transaction count
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(su32(bar))
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(su32(bar)) : "memory");
}

// bounded wait for the completion of the mbarrier phase with the given parity; false when it gave
// up (counted in g_umma_timeouts). Each attempt suspends the thread until the phase completes or
// UM_SUSPEND_NS pass, so waiting warps leave the issue slots to the warps that work beside them on
// the same SM sub-partition (a spinning wait measured 2-3x slower producers).
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, unsigned limit) {
    const uint32_t a = su32(bar);
    for (unsigned it = 0; it < limit; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(a), "r"(parity), "n"(UM_SUSPEND_NS)
            : "memory");
        if (done) return true;
    }
    atomicAdd(&g_umma_timeouts, 1u);
    return false;
}

// the same wait taken by a whole warp, with one outcome for all its lanes (the warps that go on to
// warp-collective tcgen05.ld / tcgen05.st must not diverge)
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity, unsigned limit) {
    const bool ok = mbar_wait(bar, parity, limit);
    return __all_sync(0xffffffffu, ok);
}

__device__ __forceinline__ bool warp_aborted(volatile int *flag) { return __any_sync(0xffffffffu, *flag != 0); }

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
        "%13, %14, %15, %16};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
        "%14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                   "=r"(r[7])
                 : "r"(taddr));
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// element copy global -> shared; ok = false writes zeros (src is then not read)
template <int EB>
__device__ __forceinline__ void cp_elem(uint32_t dst, const void *src, bool ok) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(EB), "r"(ok ? EB : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_commit_group() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait_group() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// One chunk of a tile row (UM_KC FP32 values; complex: (re, im) of op(B)[row, k] along k' = 2k,
// 2k + 1, conjugated for adjoint maps) split into TF32 high parts and remainders and written to the
// row's tensor-memory lane: hi at columns [ta, ta + UM_KC), lo after them. Values past the block
// (element index >= kv) are zero.
template <int W>
__device__ __forceinline__ void store_split(uint32_t ta, const float (&v)[UM_KC], int kv, bool adj) {
#pragma unroll
    for (int h = 0; h < UM_KC / 16; ++h) {
        uint32_t hi[16], lo[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            const int j = 16 * h + e;
            float x = (j / W) < kv ? v[j] : 0.0f;
            if (W == 2 && adj && (j & 1)) x = -x;
            split2(x, hi[e], lo[e]);
        }
        tmem_st16(ta + 16u * h, hi);
        tmem_st16(ta + UM_KC + 16u * h, lo);
    }
    tmem_wait_st();
}

template <class T> struct UmScalar;
template <> struct UmScalar<float> {
    static constexpr int W = 1;  // FP32 values per element
};
template <> struct UmScalar<cfloat> {
    static constexpr int W = 2;
};

// The operands of one pair with the permutations of a symmetry-reduced coupling (sets
// [rowperm | rowperm^-1 | colperm | colperm^-1]) resolved.
template <class T>
struct UmPair {
    const T *B;         // coupling block
    const T *X;         // source moments of the tile's first right-hand side, column-major snc x nq
    int snc;            // source coefficients
    int nk;             // K chunks
    const int *rowmap;  // output row -> row of the (forward or transposed) stored block, or null
    const int *kmap;    // k -> column of the (forward or transposed) stored block, or null
    bool vec;           // the moment columns start on 16-byte boundaries: whole 16-byte copies
};

template <class T>
__device__ __forceinline__ UmPair<T> um_pair(const DMap &m, const DSide &r, const DSide &t, int p, int nc,
                                             bool fwd, int nrhs, int q0, const T *am) {
    constexpr int W = UmScalar<T>::W;
    UmPair<T> u;
    u.snc = um_ncoef(t, t.level[r.i2o_src[p]]);
    u.nk = (W * u.snc + UM_KC - 1) / UM_KC;
    // transposed and adjoint products read the transposed copy: column kmap[k] of the stored block
    u.B = static_cast<const T *>(fwd ? m.cpl : m.cpl_t) + r.pair_cpl[p];
    u.X = am + r.pair_src[p] * nrhs + (int64_t)q0 * u.snc;
    const int64_t ps = r.pair_perm ? r.pair_perm[p] : -1;
    u.rowmap = nullptr;
    u.kmap = nullptr;
    // both permutations act on the stored block, so the moments are read in their own order:
    if (ps >= 0) {
        if (fwd) {  // t[rp[i], cp[j]] = M[i, j]: out[i] += sum_j M[rp^-1[i], cp^-1[j]] x[j]
            u.rowmap = m.perm + ps + nc;
            u.kmap = m.perm + ps + 3 * u.snc;
        } else {    // out[j] += sum_i op(M)[cp^-1[j], rp^-1[i]] x[i]
            u.rowmap = m.perm + ps + 3 * u.snc;
            u.kmap = m.perm + ps + u.snc;
        }
    }
    constexpr int V = 16 / (int)sizeof(T);  // elements per 16 bytes
    u.vec = (r.pair_src[p] * nrhs + (int64_t)q0 * u.snc) % V == 0 && u.snc % V == 0;
    return u;
}

__device__ __forceinline__ float2 ldg2(const cfloat *p) { return __ldg(reinterpret_cast<const float2 *>(p)); }

}  // namespace

// TMA: the coupling columns come four to a gather (`blocks` names the columns of all stored blocks, `ld`
// elements each, copied `pitch` bytes apart) from a warp of its own, for blocks of at most 256 FP32
// values per column; else the coupling warps issue a bulk copy per column (or read rows from global
// memory). A gather or bulk copy costs its warp about 100 cycles: with 32 columns per chunk of a real
// block, eight in each coupling warp, those were a third of the kernel's time.
template <class T, bool TMA>
__global__ void __maxnreg__(TMA ? 128 : 168)
i2o_umma_kernel(DMap m, DSide r, DSide t, const int *__restrict__ nodes, int mode, int nrhs, int qt_max,
                const T *__restrict__ am, T *__restrict__ dm, const __grid_constant__ CUtensorMap blocks, int pitch,
                int ld) {
    constexpr int W = UmScalar<T>::W;
    constexpr int EB = sizeof(T);        // bytes per element (4 real, 8 complex)
    constexpr int KQ = UM_KC / W;        // elements along k per chunk
    extern __shared__ __align__(128) unsigned char um_smem[];
    __shared__ uint64_t a_full[UM_NS], b_full[UM_NS], empty[UM_NS], ar_full[UM_AI][UM_AR], ar_empty[UM_AR];
    __shared__ uint64_t acc_full[2], acc_empty[2], fin;
    __shared__ uint32_t tmem_slot;
    __shared__ int nchunks_s;
    __shared__ volatile int abort_s;

    const int node = nodes[blockIdx.x];
    const int nc = um_ncoef(r, r.level[node]);
    const int m0 = blockIdx.y * UM_M;
    const int nq = m.ncomp * nrhs;
    const int q0 = blockIdx.z * qt_max;
    if (m0 >= nc || q0 >= nq) return;  // whole CTA, before any barrier
    const int mt = min(UM_M, nc - m0);
    const int qt = min(qt_max, nq - q0);
    const int np = ((W * qt_max + 15) / 16) * 16;   // MMA N: B rows (real: q; complex: Re rows, then Im rows)
    const int p0 = r.i2o_ptr[node], p1 = r.i2o_ptr[node + 1];
    T *out = dm + r.mom_off[node] * nrhs;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (p0 == p1) {
        for (int o = tid; o < mt * qt; o += (int)blockDim.x) out[(int64_t)(q0 + o / mt) * nc + m0 + o % mt] = T{};
        return;
    }
    const bool fwd = mode == H2B_FORWARD, adj = mode == H2B_ADJOINT;
    const unsigned limit = g_umma_wait_limit;

    // tensor memory: two FP32 accumulators of np columns (segments alternate between them), the
    // FP64 sum (two columns per value), then UM_NS coupling stages of 2 UM_KC columns (hi, lo)
    const uint32_t col_master = 2 * (uint32_t)np;
    const uint32_t col_a = 4 * (uint32_t)np;
    const uint32_t need = col_a + UM_NS * 2 * UM_KC;
    const uint32_t ncols = need <= 64 ? 64u : (need <= 128 ? 128u : (need <= 256 ? 256u : 512u));
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(&tmem_slot)),
                     "r"(ncols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int s = 0; s < UM_NS; ++s) {
            mbar_init(&a_full[s], 128);
            mbar_init(&b_full[s], 32);
            mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&acc_full[a], 1);
            mbar_init(&acc_empty[a], 128);
        }
        for (int a = 0; a < UM_AR; ++a) {
            for (int w = 0; w < UM_AI; ++w) mbar_init(&ar_full[w][a], 1);
            mbar_init(&ar_empty[a], 128);
        }
        mbar_init(&fin, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        nchunks_s = 0;
        abort_s = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    {  // chunks of the whole interaction list
        int mine = 0;
        for (int p = p0 + tid; p < p1; p += (int)blockDim.x) mine += (W * um_ncoef(t, t.level[r.i2o_src[p]]) + UM_KC - 1) / UM_KC;
        if (mine) atomicAdd(&nchunks_s, mine);
        // rows past the right-hand sides' rows (real tiles whose width is not a multiple of 16)
        // are zero in every stage, written once
        const int zr = np - W * qt_max;
        for (int o = tid; o < UM_NS * 2 * zr * UM_KG; o += (int)blockDim.x) {
            const int rr = W * qt_max + (o / UM_KG) % zr, kg = o % UM_KG, sh = o / (UM_KG * zr);  // sh: stage and hi/lo half
            asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(su32(um_smem) + (uint32_t)sh * ((uint32_t)np * UM_KC * 4) +
                                                                         goff(rr, kg)),
                         "r"(0u));
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
    }
    const int C = nchunks_s;
    const int G = (C + UM_SEG - 1) / UM_SEG;
    const uint32_t smem0 = su32(um_smem);
    const uint32_t b_stage_bytes = 2u * (uint32_t)np * (UM_KC * 4);  // hi then lo, canonical layout
    const uint32_t raw0 = smem0 + UM_NS * b_stage_bytes;
    const uint32_t raw_stage_bytes = (uint32_t)qt_max * UM_RAWROW;
    const uint32_t acol_bytes = TMA ? (uint32_t)pitch : (uint32_t)nc * EB;  // one stored coupling column
    const uint32_t astage_bytes = ((uint32_t)KQ * acol_bytes + 127u) & ~127u;
    const uint32_t araw0 = raw0 + ((UM_RS * raw_stage_bytes + 127u) & ~127u);

    if (warp < 4 && (TMA || m.cpl_vec)) {
        // ---------------- coupling warps, bulk-copy path ----------------
        // Per chunk, lane j of issuing warp w copies column kmap[k0 + w KQ / UM_AI + j] of the pair's
        // stored block (nc contiguous values) into a shared-memory stage with a bulk copy, UM_ALA
        // chunks ahead (each issuing warp completes its own barrier of the stage); every
        // thread then reads its own row of those columns, so the scattered accesses of a permuted
        // block stay in shared memory and global memory is read in whole columns.
        const int row = 32 * warp + lane;   // tile row = tensor-memory lane
        const bool live = row < mt;
        const uint32_t tl = tmem + ((uint32_t)(32 * warp) << 16);
        int lp = p0, lk = 0;  // consumption cursor
        UmPair<T> lu = um_pair<T>(m, r, t, p0, nc, fwd, nrhs, q0, am);
        int brow = live ? (lu.rowmap ? lu.rowmap[m0 + row] : m0 + row) : 0;
        int ip = p0, ik = 0, ic = 0;  // copy cursor (issuing warps)
        UmPair<T> iu = lu;
        constexpr int JW = KQ / UM_AI;  // columns copied by each issuing warp
        const int jw = warp * JW;       // this warp's first column of a chunk
        const bool issuer = !TMA && warp < UM_AI;
        int kcol = 0;  // lane j: stored column of the copy chunk's k = ik KQ + jw + j
        auto fetch_col = [&]() {
            const int k = min(ik * KQ + jw + lane, iu.snc - 1);
            kcol = iu.kmap ? __ldg(iu.kmap + k) : k;
        };
        auto issue = [&]() -> bool {  // issuing warp: its columns of chunk ic
            const int st = ic % UM_AR;
            if (ic >= UM_AR && !warp_wait(&ar_empty[st], ((ic / UM_AR) - 1) & 1, limit)) return false;
            const int nv = max(0, min(JW, iu.snc - ik * KQ - jw));
            const uint32_t dst = araw0 + (uint32_t)st * astage_bytes + (uint32_t)jw * acol_bytes;
            if (lane == 0) mbar_expect_tx(&ar_full[warp][st], (uint32_t)nv * acol_bytes);
            __syncwarp();
            if (lane < nv)
                bulk_copy(dst + (uint32_t)lane * acol_bytes, iu.B + (int64_t)kcol * nc, acol_bytes, &ar_full[warp][st]);
            __syncwarp();
            ++ic;
            if (++ik == iu.nk) {
                ik = 0;
                if (++ip < p1) iu = um_pair<T>(m, r, t, ip, nc, fwd, nrhs, q0, am);
            }
            if (ip < p1) fetch_col();
            return true;
        };
        int cw = 0;  // chunks whose columns this warp has waited for
        if (issuer) {
            fetch_col();
            for (int u = 0; u < UM_ALA && ic < C; ++u)
                if (!issue()) abort_s = 1;
        }
        for (int c = 0; c < C; ++c) {
            if (warp_aborted(&abort_s)) break;
            if (issuer && ic < C && !issue()) {
                abort_s = 1;
                break;
            }
            const int st = c % UM_AR;
            bool landed = true;
#pragma unroll
            for (int w = 0; w < (TMA ? 1 : UM_AI); ++w)
                landed = landed && warp_wait(&ar_full[w][st], (c / UM_AR) & 1, limit);
            if (!landed) {
                abort_s = 1;
                break;
            }
            const int kv = live ? min(KQ, lu.snc - lk * KQ) : 0;
            const uint32_t src = araw0 + (uint32_t)st * astage_bytes + (uint32_t)brow * EB;
            float v[UM_KC];
#pragma unroll
            for (int j = 0; j < KQ; ++j) {
                if constexpr (W == 2) {
                    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];"
                                 : "=f"(v[2 * j]), "=f"(v[2 * j + 1])
                                 : "r"(src + (uint32_t)j * acol_bytes));
                } else {
                    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v[j]) : "r"(src + (uint32_t)j * acol_bytes));
                }
            }
            mbar_arrive(&ar_empty[st]);
            if (++lk == lu.nk) {
                lk = 0;
                if (++lp < p1) {
                    lu = um_pair<T>(m, r, t, lp, nc, fwd, nrhs, q0, am);
                    brow = live ? (lu.rowmap ? lu.rowmap[m0 + row] : m0 + row) : 0;
                }
            }
            const int s = c % UM_NS;
            if (c >= UM_NS && !warp_wait(&empty[s], ((c / UM_NS) - 1) & 1, limit)) {
                abort_s = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t ta = tl + col_a + (uint32_t)s * (2u * UM_KC);
            store_split<W>(ta, v, kv, adj);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive(&a_full[s]);
            cw = c + 1;
        }
        if (issuer) {
            // bulk copies issued but not consumed (after a wait gave up) still write this CTA's
            // shared memory: wait for this warp's, with the full bound, before the CTA can exit
            for (int cc = cw; cc < ic; ++cc) mbar_wait(&ar_full[warp][cc % UM_AR], (cc / UM_AR) & 1, UM_SPIN_FINAL);
        }
    } else if (warp < 4) {
        // ---------------- coupling warps: A operand into tensor memory ----------------
        const int row = 32 * warp + lane;   // tile row = tensor-memory lane
        const bool live = row < mt;
        const uint32_t tl = tmem + ((uint32_t)(32 * warp) << 16);
        // load cursor: pair lp, chunk lk, the pair's operands and this thread's row of op(B), one
        // chunk ahead; every load reads a valid address (clamped row and k) and the values past the
        // block are zeroed when the chunk is split, so no instruction waits on a load early
        int lp = p0, lk = 0;
        UmPair<T> lu = um_pair<T>(m, r, t, p0, nc, fwd, nrhs, q0, am);
        int brow = live ? (lu.rowmap ? lu.rowmap[m0 + row] : m0 + row) : 0;
        float ra[2][UM_KC];
        int kv[2];    // valid elements of each buffered chunk (0 for rows past the tile)
        int km[KQ];   // stored-block indices of the next chunk's k (its permutation, fetched a chunk ahead)
        auto fetch_map = [&]() {
#pragma unroll
            for (int j = 0; j < KQ; ++j) {
                const int k = min(lk * KQ + j, lu.snc - 1);
                km[j] = lu.kmap ? __ldg(lu.kmap + k) : k;
            }
        };
        auto load = [&](float (&v)[UM_KC], int &nvalid) {
            const int k0 = lk * KQ;
            nvalid = live ? min(KQ, lu.snc - k0) : 0;
#pragma unroll
            for (int j = 0; j < KQ; ++j) {
                const int k = km[j];
                const T *src = lu.B + brow + (int64_t)k * nc;
                if constexpr (W == 2) {
                    const float2 x = ldg2(src);
                    v[2 * j] = x.x;
                    v[2 * j + 1] = x.y;
                } else {
                    v[j] = __ldg(src);
                }
            }
            if (++lk == lu.nk) {
                lk = 0;
                if (++lp < p1) {
                    lu = um_pair<T>(m, r, t, lp, nc, fwd, nrhs, q0, am);
                    brow = live ? (lu.rowmap ? lu.rowmap[m0 + row] : m0 + row) : 0;
                }
            }
            if (lp < p1) fetch_map();
        };
        fetch_map();
        load(ra[0], kv[0]);
        for (int c0 = 0; c0 < C; c0 += 2) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int c = c0 + u;
                if (c >= C || warp_aborted(&abort_s)) break;
                if (c + 1 < C) load(ra[u ^ 1], kv[u ^ 1]);
                const int s = c % UM_NS;
                if (c >= UM_NS && !warp_wait(&empty[s], ((c / UM_NS) - 1) & 1, limit)) {
                    abort_s = 1;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t ta = tl + col_a + (uint32_t)s * (2u * UM_KC);
                store_split<W>(ta, ra[u], kv[u], adj);
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                mbar_arrive(&a_full[s]);
            }
            if (warp_aborted(&abort_s)) break;
        }
    } else if (warp < 4 + UM_BW) {
        // ---------------- moment warps: B operand into shared memory ----------------
        // warp bw takes every UM_BW-th chunk on its own, so nothing but the stages ties the warps
        const int bw = warp - 4;
        // copy cursor (pair cp_, chunk ck; the next pair's operands loaded a pair ahead); a chunk's raw
        // moments are qt_max rows of 128 bytes, copied as 16-byte pieces (consecutive lanes: consecutive
        // pieces of a row), element by element where a column is not 16-byte aligned or the chunk
        // runs past the pair's coefficients
        int cp_ = p0, ck = bw;
        UmPair<T> cu = um_pair<T>(m, r, t, p0, nc, fwd, nrhs, q0, am);
        UmPair<T> cn = um_pair<T>(m, r, t, min(p0 + 1, p1 - 1), nc, fwd, nrhs, q0, am);
        auto settle = [&]() {
            while (cp_ < p1 && ck >= cu.nk) {
                ck -= cu.nk;
                cu = cn;
                if (++cp_ + 1 < p1) cn = um_pair<T>(m, r, t, cp_ + 1, nc, fwd, nrhs, q0, am);
            }
        };
        settle();
        constexpr int EV = 16 / EB;  // elements per piece
        auto issue = [&](int turn) {
            const uint32_t rb = raw0 + (uint32_t)(2 * bw + (turn & 1)) * raw_stage_bytes;
            const int k0 = ck * KQ;
            for (int pc = lane; pc < qt_max * UM_KG; pc += 32) {
                const int q = pc / UM_KG, kg = pc % UM_KG, kp = k0 + kg * EV;
                const uint32_t dst = rb + (uint32_t)q * UM_RAWROW + (uint32_t)kg * 16;
                const T *src = cu.X + (int64_t)q * cu.snc + kp;
                if (cu.vec && q < qt && kp + EV <= cu.snc) {
                    cp_elem<16>(dst, src, true);
                } else {
#pragma unroll
                    for (int e = 0; e < EV; ++e) {
                        const bool ok = q < qt && kp + e < cu.snc;
                        cp_elem<EB>(dst + (uint32_t)(e * EB), ok ? src + e : cu.X, ok);
                    }
                }
            }
            ck += UM_BW;
            settle();
        };
        if (bw < C) issue(0);
        cp_commit_group();
        const int npieces = qt_max * UM_KG;  // 16-byte pieces of the raw tile
        const int q0p = lane % qt_max, kg0 = lane / qt_max;
        for (int c = bw, turn = 0; c < C; c += UM_BW, ++turn) {
            if (c + UM_BW < C) issue(turn + 1);  // into the stage of the turn before this one
            cp_commit_group();
            cp_wait_group<1>();  // this lane's copies of chunk c have landed
            __syncwarp();        // ... and the warp's
            if (warp_aborted(&abort_s)) break;
            const int s = c % UM_NS;
            // the expanded stage was last read by the products of chunk c - UM_NS
            if (c >= UM_NS && !warp_wait(&empty[s], ((c / UM_NS) - 1) & 1, limit)) {
                abort_s = 1;
                break;
            }
            const uint32_t rb = raw0 + (uint32_t)(2 * bw + (turn & 1)) * raw_stage_bytes;
            const uint32_t hb = smem0 + (uint32_t)s * b_stage_bytes;
            const uint32_t lb = hb + (uint32_t)np * (UM_KC * 4);
            // raw pieces lane, lane + 32, ... as (row q, k group kg), rows fastest: a quarter-warp
            // reads 8 rows of one k group and writes 8 consecutive rows of the expanded tile
            // (conflict-free); a complex piece (mr, mi) of two k is split once and written to
            // both its rows, Re (mr, -mi) and Im (mi, mr): negation is exact in TF32 parts
            int q = q0p, kg = kg0;
            for (int pc = lane; pc < npieces; pc += 32) {
                if (pc != lane) {
                    q += 32;
                    while (q >= qt_max) {
                        q -= qt_max;
                        ++kg;
                    }
                }
                float w[4];
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                             : "=f"(w[0]), "=f"(w[1]), "=f"(w[2]), "=f"(w[3])
                             : "r"(rb + (uint32_t)q * UM_RAWROW + (uint32_t)kg * 16));
                uint32_t h[4], l[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) split2(w[e], h[e], l[e]);
                const uint32_t o = goff(q, kg);
                if constexpr (W == 1) {
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(hb + o), "r"(h[0]), "r"(h[1]),
                                 "r"(h[2]), "r"(h[3]));
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(lb + o), "r"(l[0]), "r"(l[1]),
                                 "r"(l[2]), "r"(l[3]));
                } else {
                    constexpr uint32_t S = 0x80000000u;
                    const uint32_t oi = goff(qt_max + q, kg);
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(hb + o), "r"(h[0]), "r"(h[1] ^ S),
                                 "r"(h[2]), "r"(h[3] ^ S));
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(lb + o), "r"(l[0]), "r"(l[1] ^ S),
                                 "r"(l[2]), "r"(l[3] ^ S));
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(hb + oi), "r"(h[1]), "r"(h[0]),
                                 "r"(h[3]), "r"(h[2]));
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(lb + oi), "r"(l[1]), "r"(l[0]),
                                 "r"(l[3]), "r"(l[2]));
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_arrive(&b_full[s]);
            __syncwarp();  // this turn's raw stage is copied into in the next one
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (TMA && warp == UM_WARPS) {
        // ---------------- copy warp: a chunk's columns, UM_AR chunks ahead ----------------
        // lane j: the columns 4 j .. 4 j + 3 of a chunk (past the block: its last one), loaded a chunk before
        // they are used
        int ip = p0, ik = 0, c = 0;
        UmPair<T> u = um_pair<T>(m, r, t, p0, nc, fwd, nrhs, q0, am);
        int col0 = (int)(r.pair_cpl[p0] / ld);
        auto columns = [&](int k) -> int4 {
            int v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int kk = min(k * KQ + 4 * lane + e, u.snc - 1);
                v[e] = u.kmap ? __ldg(u.kmap + kk) : kk;
            }
            return make_int4(v[0], v[1], v[2], v[3]);
        };
        int4 cols = make_int4(0, 0, 0, 0);
        if (lane < KQ / 4) cols = columns(0);
        for (; c < C; ++c) {
            const int st = c % UM_AR, groups = (min(KQ, u.snc - ik * KQ) + 3) / 4, first = col0;
            int4 next = cols;
            if (++ik == u.nk) {
                ik = 0;
                if (++ip < p1) {
                    u = um_pair<T>(m, r, t, ip, nc, fwd, nrhs, q0, am);
                    col0 = (int)(r.pair_cpl[ip] / ld);
                }
            }
            if (c + 1 < C && lane < KQ / 4) next = columns(ik);
            if (warp_aborted(&abort_s) || (c >= UM_AR && !warp_wait(&ar_empty[st], ((c / UM_AR) - 1) & 1, limit))) {
                abort_s = 1;
                break;
            }
            if (lane == 0) mbar_expect_tx(&ar_full[0][st], (uint32_t)(4 * groups) * acol_bytes);
            __syncwarp();
            if (lane < groups)
                tma_gather4(araw0 + (uint32_t)st * astage_bytes + (uint32_t)lane * (4 * acol_bytes), &blocks, 0,
                            make_int4(cols.x + first, cols.y + first, cols.z + first, cols.w + first), &ar_full[0][st]);
            __syncwarp();
            cols = next;
        }
        // copies in flight write this CTA's shared memory: all have landed before the CTA can exit
        for (int cc = max(0, c - UM_AR); cc < c; ++cc) mbar_wait(&ar_full[0][cc % UM_AR], (cc / UM_AR) & 1, UM_SPIN_FINAL);
    } else if (warp < UM_WARPS - 1) {
        // ---------------- drain warps: FP64 sum of the segments, then the epilogue ----------------
        const int lq = warp & 3;
        const int row = 32 * lq + lane;
        const uint32_t tl = tmem + ((uint32_t)(32 * lq) << 16);
        bool ok = true;
        for (int g = 0; g < G; ++g) {
            const int a = g & 1;
            if (!warp_wait(&acc_full[a], (g >> 1) & 1, limit)) {
                abort_s = 1;
                ok = false;
                break;
            }
            if (warp_aborted(&abort_s)) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int j = 0; j < np; j += 16) {
                uint32_t f[16], w0[16], w1[16];
                tmem_ld16(tl + (uint32_t)(a * np + j), f);
                if (g > 0) {
                    tmem_ld16(tl + col_master + 2u * (uint32_t)j, w0);
                    tmem_ld16(tl + col_master + 2u * (uint32_t)j + 16u, w1);
                }
                tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    uint32_t &lo = e < 8 ? w0[2 * e] : w1[2 * (e - 8)];
                    uint32_t &hi = e < 8 ? w0[2 * e + 1] : w1[2 * (e - 8) + 1];
                    const double prev = g > 0 ? __hiloint2double((int)hi, (int)lo) : 0.0;
                    const double v = prev + (double)__uint_as_float(f[e]);
                    lo = (uint32_t)__double2loint(v);
                    hi = (uint32_t)__double2hiint(v);
                }
                tmem_st16(tl + col_master + 2u * (uint32_t)j, w0);
                tmem_st16(tl + col_master + 2u * (uint32_t)j + 16u, w1);
            }
            tmem_wait_st();
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive(&acc_empty[a]);
        }
        if (ok && !warp_aborted(&abort_s)) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int j8 = 0; j8 * 8 < qt; ++j8) {
                uint32_t wr[16], wi[16];
                tmem_ld16(tl + col_master + 2 * (uint32_t)(8 * j8), wr);
                if constexpr (W == 2) tmem_ld16(tl + col_master + 2 * (uint32_t)(qt_max + 8 * j8), wi);
                tmem_wait_ld();
                if (row < mt) {
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const int q = 8 * j8 + e;
                        if (q >= qt) break;
                        const double re = __hiloint2double((int)wr[2 * e + 1], (int)wr[2 * e]);
                        T *o = out + (int64_t)(q0 + q) * nc + m0 + row;
                        if constexpr (W == 2) {
                            const double im = __hiloint2double((int)wi[2 * e + 1], (int)wi[2 * e]);
                            *o = T{(float)re, (float)im};
                        } else {
                            *o = (float)re;
                        }
                    }
                }
            }
        }
    } else {
        // ---------------- MMA warp: twelve products of N = np columns per chunk ----------------
        const uint32_t idesc = tf32_idesc(UM_M, np), el = elect_one();
        const uint64_t desc0 = kmajor_desc(smem0);
        for (int c = 0; c < C; ++c) {
            const int s = c % UM_NS, g = c / UM_SEG, a = g & 1;
            if (c % UM_SEG == 0 && g >= 2 && !warp_wait(&acc_empty[a], ((g >> 1) - 1) & 1, limit)) abort_s = 1;
            if (!warp_aborted(&abort_s) && !warp_wait(&a_full[s], (c / UM_NS) & 1, limit)) abort_s = 1;
            if (!warp_aborted(&abort_s) && !warp_wait(&b_full[s], (c / UM_NS) & 1, limit)) abort_s = 1;
            if (warp_aborted(&abort_s)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t d = tmem + (uint32_t)(a * np);
            const uint32_t ta = tmem + col_a + (uint32_t)s * (2u * UM_KC);
            const uint64_t bh = desc0 + (uint64_t)(((uint32_t)s * b_stage_bytes) >> 4);
            const uint64_t bl = bh + (uint64_t)(((uint32_t)np * (UM_KC * 4)) >> 4);
#pragma unroll
            for (int j = 0; j < UM_KC / 8; ++j) {
                const uint64_t dbh = bh + (uint64_t)((j * 2 * UM_LBO) >> 4), dbl = bl + (uint64_t)((j * 2 * UM_LBO) >> 4);
                umma_ts_if(el, d, ta + 8u * j, dbh, idesc, (c % UM_SEG != 0 || j > 0) ? 1u : 0u);
                umma_ts_if(el, d, ta + 8u * j, dbl, idesc, 1u);
                umma_ts_if(el, d, ta + UM_KC + 8u * j, dbh, idesc, 1u);
            }
            umma_commit_if(el, &empty[s]);
            if (c % UM_SEG == UM_SEG - 1 || c == C - 1) umma_commit_if(el, &acc_full[a]);
        }
        umma_commit_if(el, &fin);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();  // every role has left its loop
    // products already issued (all of them, after a wait gave up) may still read the operand stages and
    // write tensor memory: they are waited for, with the full bound, before the CTA frees its memory
    if (warp == UM_WARPS - 1 && lane == 0) mbar_wait(&fin, 0, UM_SPIN_FINAL);
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols) : "memory");
}

// ---------------------------------------------------------------------------------------------
// The same products by stored block: one tile of the pairs that read one block through one column
// permutation (PairTiles::tile32) instead of one receiving node, so the split of a block's chunk
// into TF32 parts serves all the columns of a tile (pairs x right-hand sides, packed without gaps)
// instead of one pair's, and no column of the product is padding. Per (tile, 128 of the block's
// rows, 64 product columns) item a persistent CTA runs the pipeline above over the K values of the
// block; chunks, segments and the order of the products inside them are those of i2o_umma_kernel
// (an item's chunk count is even, so no segment spans two pairs there either), hence the same FP32
// segment sums. Each pair's FP64 sum goes to its column of the pair-product buffer; the row
// permutation is left to i2o_pairs_sum_kernel, so the rows of a tile are contiguous in the block.
//
// What bounds it: the roles' instructions, about 2,700 per chunk (1,360 cycles against 384 for the
// chunk's products; ncu: 0.51 issued per scheduler and cycle, tensor operands and L2 far from full).
// Taking one role's work away gains 4-10 % each (the coupling's split most). Measured (I2O per
// product, 65,536-point Helmholtz sphere, p = 6): 8 right-hand sides 14.2 -> 3.2 ms, 32 right-hand
// sides 15.1 -> 11.3 ms (2 of them the sums) against one receiving node per CTA.
// Roles (24 warps, six warpgroups):
//   * scheduler: turns the CTA's items into records in a ring (the block, and every column's moments
//     and product), so that no other role chases the plan's arrays;
//   * a copy warp: the rows of each chunk's columns into a ring of UP_AR stages, four columns per TMA
//     gather (a column permutation is which columns are named; one bulk copy per column cost its warp
//     about 100 cycles each, and 16-byte cp.async pieces held every role up behind the SM's own
//     load path);
//   * a second copy warp for the moments, four columns of the product per TMA gather, where the
//     moment columns are whole 16 bytes; else the moment warps copy them with cp.async a turn ahead;
//   * eight coupling warps, four per chunk in turn: read, split, write to tensor memory;
//   * four moment warps, one chunk each in turn: split its moments into shared memory; operand stages
//     hold a whole segment (two chunks), so the MMA warp waits once per 24 products;
//   * the MMA warp; eight drain warps, which keep the FP64 sums (32 each) in registers: the kernel starts
//     with 80 registers a thread and moves them to the drain warps (setmaxnreg; 256 threads each at 64,
//     64 and 112 make the 240 x 256 that the block was launched with).
// ---------------------------------------------------------------------------------------------
constexpr int UP_N = 64;                  // product columns per item
constexpr int UP_NS = 3;                  // operand stages, one accumulation segment each
template <int W> constexpr int up_ar() { return W == 2 ? 4 : 3; }  // coupling column stages
// Item records: a moment warp that splits a chunk of record n has its copy cursor one turn (four
// chunks) past the next turn's, at most four records of two chunks ahead, before it is done with n.
constexpr int UP_IR = 8;
constexpr int UP_B0 = 8, UP_COPY = 12, UP_MMA = 14, UP_SCHED = 15, UP_D0 = 16;  // first warps of the roles
constexpr int UP_WARPS = 24, UP_THREADS = UP_WARPS * 32;
constexpr int UP_BW = UP_COPY - UP_B0;    // moment warps
constexpr int UP_RS = 2 * UP_BW;          // raw moment stages: a ring, or two per moment warp
constexpr int UP_READERS = UP_WARPS - 1;  // warps that read the item records
static_assert(UM_SEG == 2, "an operand stage holds two chunks, one per half of the coupling warps");
constexpr int UP_REG_A = 64, UP_REG_B = 64, UP_REG_D = 112;
static_assert(UP_BW == 2 * UM_SEG && UP_NS * UM_SEG > UP_BW, "two moment warps fill a stage");

// elements of a block's column as stored for the column copies: whole 16 bytes
template <class T> __host__ __device__ constexpr int up_ld(int nc) {
    return (nc + 16 / (int)sizeof(T) - 1) / (16 / (int)sizeof(T)) * (16 / (int)sizeof(T));
}

// a raw moment stage: rows of a chunk's 128 bytes, swizzled (TMA) or padded (cp.async)
template <bool TMA> constexpr uint32_t up_raw_row() { return TMA ? UM_KC * 4 : UM_RAWROW; }

struct UpArgs {
    const int4 *rec;           // per pair: {moment offset (low, high), permutation set or -1, pair}
    const int4 *tile;          // {first record, pairs, rows, k}
    const int64_t *tile_off;   // element offset of the tile's block
    int tile0, mt;             // the unit's first tile; row tiles of a block
    int more[PAIR_TILE];       // tiles of the unit with more than c pairs
    int mode, nrhs, q0, qn, pbase, pstride;
    int ld, pitch, rowbox;     // elements of a stored block column, bytes of a copied one; moment rows per copy
};

template <int NC> struct UpItem {
    int nk, ncol, snc, rows;   // nk = 0: no more items
    int m0, col;               // first row of the block, column index of the block in its tensor map
    int64_t perm;              // k -> stored column in DMap::perm, -1: identity
    int64_t src[NC], out[NC];  // per column: its moments (TMA: its row in their map), its product
};

// the tensor map's box (its rows from r on), from x on
__device__ __forceinline__ void tma_box(uint32_t dst, const CUtensorMap *map, int x, int r, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(map), "r"(x), "r"(r), "r"(su32(bar))
        : "memory");
}

// mbar_wait (for a whole warp, with one outcome, when WARP) that also ends (false, uncounted) once the CTA has given up: the flag is
// read only after an attempt that found the phase incomplete, so a wait that finds it complete costs
// one instruction
template <bool WARP> __device__ __forceinline__ bool up_wait(uint64_t *bar, uint32_t parity, unsigned limit, volatile int *abort) {
    const uint32_t a = su32(bar);
    uint32_t done = 0;
    unsigned it = 0;
    for (; it < limit; ++it) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(a), "r"(parity), "n"(UM_SUSPEND_NS)
            : "memory");
        if (done || *abort) break;
    }
    if (it == limit && !done) atomicAdd(&g_umma_timeouts, 1u);
    if constexpr (WARP) return __all_sync(0xffffffffu, done != 0);
    return done != 0;
}

__device__ __forceinline__ void cp16_cg(uint32_t dst, const void *src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}

// product rows of one part (real, imaginary) of `ncol` columns: MMA N is a multiple of 16
template <int W> __device__ __forceinline__ int up_part(int ncol) {
    return W == 2 ? (ncol + 7) & ~7 : (ncol + 15) & ~15;
}

template <class T, bool TMA>
__global__ void __launch_bounds__(UP_THREADS, 1)
i2o_umma_pairs_kernel(DMap m, UpArgs g, const __grid_constant__ CUtensorMap blocks,
                      const __grid_constant__ CUtensorMap moments, const T *__restrict__ am,
                      typename ScalarTraits<T>::Acc *__restrict__ prod) {
    constexpr int W = UmScalar<T>::W;
    constexpr int EB = sizeof(T);
    constexpr int KQ = UM_KC / W;       // elements along k per chunk
    constexpr int NC = UP_N / W;        // columns (pairs x right-hand sides) per item
    constexpr uint32_t B_CHUNK = 2u * UP_N * UM_KC * 4, B_STAGE = UM_SEG * B_CHUNK;  // per chunk: hi then lo
    constexpr uint32_t RAW_ROW = up_raw_row<TMA>(), RAW_STAGE = (uint32_t)NC * RAW_ROW;
    constexpr uint32_t A_STAGE = KQ * UM_M * EB;
    const uint32_t A_COL = (uint32_t)g.pitch;
    constexpr uint32_t COL_A = 2 * UP_N;  // tensor memory: two accumulators, then the coupling stages
    extern __shared__ __align__(128) unsigned char um_smem[];
    constexpr int UP_AR = up_ar<W>();
    __shared__ uint64_t full[UP_NS], empty[UP_NS], ar_full[UP_AR], ar_empty[UP_AR], br_full[UP_RS], br_empty[UP_RS];
    __shared__ uint64_t acc_full[2], acc_empty[2], it_full[UP_IR], it_empty[UP_IR], fin;
    __shared__ UpItem<NC> rec[UP_IR];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_s;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool fwd = g.mode == H2B_FORWARD, adj = g.mode == H2B_ADJOINT;
    const unsigned limit = g_umma_wait_limit;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(&tmem_slot)), "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int s = 0; s < UP_NS; ++s) {
            mbar_init(&full[s], 256 + 32 * UM_SEG);
            mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&acc_full[a], 1);
            mbar_init(&acc_empty[a], 256);
        }
        for (int a = 0; a < UP_AR; ++a) {
            mbar_init(&ar_full[a], 1);
            mbar_init(&ar_empty[a], 128);
        }
        for (int a = 0; a < UP_RS; ++a) {
            mbar_init(&br_full[a], 1);
            mbar_init(&br_empty[a], 32);
        }
        for (int a = 0; a < UP_IR; ++a) {
            mbar_init(&it_full[a], 1);
            mbar_init(&it_empty[a], UP_READERS);
        }
        mbar_init(&fin, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        abort_s = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    const uint32_t smem0 = (su32(um_smem) + 1023u) & ~1023u;
    const uint32_t raw0 = smem0 + UP_NS * B_STAGE;
    const uint32_t araw0 = raw0 + ((UP_RS * RAW_STAGE + 1023u) & ~1023u);
    // record n of the ring, for a whole warp; false when the wait gave up
    auto wait = [&](uint64_t *bar, uint32_t parity) -> bool { return up_wait<true>(bar, parity, limit, &abort_s); };
    auto item = [&](int n) -> bool { return wait(&it_full[n % UP_IR], (n / UP_IR) & 1); };
    auto item_done = [&](int n) {
        __syncwarp();
        if (lane == 0) mbar_arrive(&it_empty[n % UP_IR]);
    };

    if (warp < UP_B0) {
        // ---------------- coupling warps: one tile row per thread, alternate chunks ----------------
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(UP_REG_A));
        const int grp = warp >> 2, row = tid & 127;
        const uint32_t tl = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
        int c = 0;  // chunks of the items before this one
        bool run = true;
        for (int n = 0; run; ++n) {
            if (!(run = item(n))) break;
            const UpItem<NC> &it = rec[n % UP_IR];
            const int nk = it.nk, snc = it.snc;
            if (nk == 0) break;
            // (rows past the tile split whatever their stage holds: their products are never stored)
            for (int k = grp; k < nk; k += 2) {
                const int cc = c + k, st = cc % UP_AR, sg = cc / UM_SEG, s = sg % UP_NS;
                if (!(run = wait(&ar_full[st], (cc / UP_AR) & 1))) break;
                const uint32_t src = araw0 + (uint32_t)st * A_STAGE + (uint32_t)row * EB;
                const uint32_t ta = tl + COL_A + (uint32_t)(s * UM_SEG + grp) * (2u * UM_KC);
                const int kv = snc - k * KQ;  // values past the block are zeroed (in its last, partial chunk)
#pragma unroll
                for (int h = 0; h < 2; ++h) {  // 16 values at a time
                    float v[16];
#pragma unroll
                    for (int j = 0; j < 16 / W; ++j) {
                        const uint32_t sj = src + (uint32_t)(j + h * 16 / W) * A_COL;
                        if constexpr (W == 2)
                            asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v[2 * j]), "=f"(v[2 * j + 1]) : "r"(sj));
                        else
                            asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v[j]) : "r"(sj));
                    }
                    uint32_t hi[16], lo[16];
                    if (kv < KQ) {
#pragma unroll
                        for (int e = 0; e < 16; ++e)
                            if ((16 * h + e) / W >= kv) v[e] = 0.0f;
                    }
#pragma unroll
                    for (int e = 0; e < 16; ++e) split2(v[e], hi[e], lo[e]);
                    if (h == 1) {
                        mbar_arrive(&ar_empty[st]);
                    } else {
                        if (sg >= UP_NS && !(run = wait(&empty[s], ((sg / UP_NS) - 1) & 1))) break;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    }
                    tmem_st16(ta + 16u * h, hi);
                    tmem_st16(ta + UM_KC + 16u * h, lo);
                }
                if (!run) break;
                tmem_wait_st();
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                mbar_arrive(&full[s]);
            }
            c += nk;
            item_done(n);
        }
        if (!run) abort_s = 1;
    } else if (warp < UP_D0) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(UP_REG_B));
        if (warp < UP_COPY) {
            // ---------------- moment warps: B operand into shared memory ----------------
            // warp bw takes every fourth chunk on its own, so nothing but the stages ties the warps
            const int bw = warp - UP_B0;
            constexpr int EV = 16 / EB;  // elements per 16-byte piece
            const uint32_t S = 0x80000000u, s_re = adj ? 0u : S, s_im = adj ? S : 0u;
            int in = 0, ik = bw, turn = 0;  // copy cursor (cp.async): record, chunk of it, chunks copied
            bool run = TMA || item(0), more = !TMA && run;
            // moves the cursor to the next record with a chunk for this warp (at once: a record is
            // reused after its last chunk)
            auto enter = [&]() {
                while (more && rec[in % UP_IR].nk != 0 && ik >= rec[in % UP_IR].nk) {
                    ik -= rec[in % UP_IR].nk;
                    more = run = item(++in);
                }
                more = more && rec[in % UP_IR].nk != 0;
            };
            auto copy = [&]() {
                const UpItem<NC> &it = rec[in % UP_IR];
                const uint32_t rb = raw0 + (uint32_t)(2 * bw + (turn & 1)) * RAW_STAGE;
                const int ncol = it.ncol, snc = it.snc, ncp = up_part<W>(ncol);
                const int kg = lane & 7, kp = ik * KQ + kg * EV;
#pragma unroll
                for (int u = 0; u < NC / 4; ++u) {
                    const int q = (lane >> 3) + 4 * u;
                    const uint32_t dst = rb + (uint32_t)q * UM_RAWROW + (uint32_t)kg * 16;
                    if (q < ncol) {
                        const int64_t o = it.src[q] + kp;
                        if (kp + EV <= snc && o % EV == 0) {
                            cp16_cg(dst, am + o, true);
                        } else {
#pragma unroll
                            for (int e = 0; e < EV; ++e) {
                                const bool ok = kp + e < snc;
                                cp_elem<EB>(dst + (uint32_t)(e * EB), ok ? am + o + e : am, ok);
                            }
                        }
                    } else if (q < ncp) {
                        cp16_cg(dst, am, false);
                    }
                }
                ++turn;
                ik += UP_BW;
            };
            if constexpr (!TMA) {
                enter();
                if (more) copy();
                enter();
                cp_commit_group();
            }
            int c = 0;  // chunks of the records before record n
            for (int n = 0, done = 0; run; ++n) {
                if (!(run = item(n))) break;
                const UpItem<NC> &it = rec[n % UP_IR];
                const int nk = it.nk, ncp = up_part<W>(it.ncol);
                if (nk == 0) break;
                for (int k = (bw - c) & (UP_BW - 1); k < nk; k += UP_BW, ++done) {
                    const int cc = c + k, sg = cc / UM_SEG, s = sg % UP_NS, rs = TMA ? cc % UP_RS : 2 * bw + (done & 1);
                    if constexpr (TMA) {
                        if (!(run = wait(&br_full[rs], (cc / UP_RS) & 1))) break;
                    } else {
                        if (more) copy();  // the next turn's, into the stage of the turn before this one
                        enter();
                        if (!run) break;
                        cp_commit_group();
                        cp_wait_group<1>();
                        __syncwarp();
                    }
                    if (sg >= UP_NS && !(run = wait(&empty[s], ((sg / UP_NS) - 1) & 1))) break;
                    const uint32_t rb = raw0 + (uint32_t)rs * RAW_STAGE;
                    const uint32_t hb = smem0 + (uint32_t)s * B_STAGE + (uint32_t)(cc % UM_SEG) * B_CHUNK;
                    const uint32_t lb = hb + UP_N * UM_KC * 4;
                    // lane: column (and column + 32 of a real tile)
#pragma unroll
                    for (int g2 = 0; g2 < NC / 32; ++g2) {
                        const int q = lane + 32 * g2;
                        if (q >= ncp) continue;
                        const uint32_t o0 = goff(q, 0), oi0 = W == 2 ? goff(ncp + q, 0) : 0;
                        // all of the column's loads before the first store
                        float w[UM_KG][4];
#pragma unroll
                        for (int kg = 0; kg < UM_KG; ++kg)
                            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                                         : "=f"(w[kg][0]), "=f"(w[kg][1]), "=f"(w[kg][2]), "=f"(w[kg][3])
                                         : "r"(rb + (uint32_t)q * RAW_ROW + (uint32_t)(TMA ? kg ^ (q & 7) : kg) * 16));
#pragma unroll
                        for (int kg = 0; kg < UM_KG; ++kg) {
                            uint32_t h[4], l[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) split2(w[kg][e], h[e], l[e]);
                            const uint32_t o = o0 + (uint32_t)kg * UM_LBO;
                            if constexpr (W == 1) {
                                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(hb + o), "r"(h[0]),
                                             "r"(h[1]), "r"(h[2]), "r"(h[3]));
                                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(lb + o), "r"(l[0]),
                                             "r"(l[1]), "r"(l[2]), "r"(l[3]));
                            } else {
                                // Re row (mr, -mi), Im row (mi, mr); conjugated blocks: (mr, mi), (mi, -mr)
                                const uint32_t oi = oi0 + (uint32_t)kg * UM_LBO;
                                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(hb + o), "r"(h[0]),
                                             "r"(h[1] ^ s_re), "r"(h[2]), "r"(h[3] ^ s_re));
                                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(lb + o), "r"(l[0]),
                                             "r"(l[1] ^ s_re), "r"(l[2]), "r"(l[3] ^ s_re));
                                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(hb + oi), "r"(h[1]),
                                             "r"(h[0] ^ s_im), "r"(h[3]), "r"(h[2] ^ s_im));
                                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(lb + oi), "r"(l[1]),
                                             "r"(l[0] ^ s_im), "r"(l[3]), "r"(l[2] ^ s_im));
                            }
                        }
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    mbar_arrive(&full[s]);
                    if constexpr (TMA) mbar_arrive(&br_empty[rs]);
                    else __syncwarp();  // the stage of this turn is copied into in the next one
                }
                c += nk;
                if (run) item_done(n);
            }
            if (!run) abort_s = 1;
            asm volatile("cp.async.wait_all;" ::: "memory");
        } else if (warp < UP_MMA) {
            // ---------------- copy warps: coupling columns UP_AR, moments UP_RS chunks ahead ----------------
            bool run = true;
            int c = 0;
            if (warp == UP_COPY) {
                for (int n = 0; run; ++n) {
                    if (!(run = item(n))) break;
                    const UpItem<NC> &it = rec[n % UP_IR];
                    const int nk = it.nk, snc = it.snc, col0 = it.col, x0 = it.m0 * W;
                    if (nk == 0) break;
                    // lane j: the columns 4 j .. 4 j + 3 of a chunk (past the block: its last one), loaded a
                    // chunk before they are used
                    const int *kmap = it.perm >= 0 ? m.perm + it.perm : nullptr;
                    auto columns = [&](int k) -> int4 {
                        int r[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const int kk = min(k * KQ + 4 * lane + e, snc - 1);
                            r[e] = kmap ? __ldg(kmap + kk) : kk;
                        }
                        return make_int4(r[0], r[1], r[2], r[3]);
                    };
                    int4 r = make_int4(0, 0, 0, 0), next = r;
                    if (lane < KQ / 4) r = columns(0);
                    for (int k = 0; k < nk; ++k, ++c) {
                        const int groups = (min(KQ, snc - k * KQ) + 3) / 4, st = c % UP_AR;
                        if (k + 1 < nk && lane < KQ / 4) next = columns(k + 1);
                        if (c >= UP_AR && !(run = wait(&ar_empty[st], ((c / UP_AR) - 1) & 1))) break;
                        if (lane == 0) mbar_expect_tx(&ar_full[st], (uint32_t)(4 * groups) * A_COL);
                        __syncwarp();
                        if (lane < groups)
                            tma_gather4(araw0 + (uint32_t)st * A_STAGE + (uint32_t)lane * (4 * A_COL), &blocks, x0,
                                        make_int4(r.x + col0, r.y + col0, r.z + col0, r.w + col0), &ar_full[st]);
                        __syncwarp();
                        r = next;
                    }
                    if (run) item_done(n);
                }
                // copies in flight write this CTA's shared memory: all have landed before the CTA can exit
                for (int cc = max(0, c - UP_AR); cc < c; ++cc) mbar_wait(&ar_full[cc % UP_AR], (cc / UP_AR) & 1, UM_SPIN_FINAL);
            } else {
                for (int n = 0; run; ++n) {
                    if (!(run = item(n))) break;
                    const UpItem<NC> &it = rec[n % UP_IR];
                    const int nk = it.nk, rb = TMA ? g.rowbox : 1, groups = (it.ncol + rb - 1) / rb;
                    if (nk == 0) break;
                    if constexpr (TMA) {
                        // lane j: rows j rb .. of the item's columns, in one box of rb rows (rb right-hand sides
                        // of a pair lie side by side) or, rb = 4, four rows named one by one
                        int4 r = make_int4(0, 0, 0, 0);
                        if (lane < groups) {
                            const int64_t *src = it.src + lane * rb;
                            r = make_int4((int)src[0], (int)src[1], (int)src[2], (int)src[3]);
                        }
                        const uint32_t dst = raw0 + (uint32_t)(lane * rb) * RAW_ROW, bytes = (uint32_t)(groups * rb) * RAW_ROW;
                        for (int k = 0; k < nk; ++k, ++c) {
                            const int st = c % UP_RS;
                            if (c >= UP_RS && !(run = wait(&br_empty[st], ((c / UP_RS) - 1) & 1))) break;
                            if (lane == 0) mbar_expect_tx(&br_full[st], bytes);
                            __syncwarp();
                            if (lane < groups) {
                                if (rb == 4) tma_gather4(dst + (uint32_t)st * RAW_STAGE, &moments, k * UM_KC, r, &br_full[st]);
                                else tma_box(dst + (uint32_t)st * RAW_STAGE, &moments, k * UM_KC, r.x, &br_full[st]);
                            }
                            __syncwarp();
                        }
                    }
                    if (run) item_done(n);
                }
                if constexpr (TMA)
                    for (int cc = max(0, c - UP_RS); cc < c; ++cc)
                        mbar_wait(&br_full[cc % UP_RS], (cc / UP_RS) & 1, UM_SPIN_FINAL);
            }
            if (!run) abort_s = 1;
        } else if (warp == UP_MMA) {
            // ---------------- MMA warp: converged, one lane issues ----------------
            int sg = 0;  // segments so far
            bool run = true;
            const uint32_t el = elect_one();
            const uint64_t desc0 = kmajor_desc(smem0);
            for (int n = 0; run; ++n) {
                if (!(run = item(n))) break;
                const int ns = rec[n % UP_IR].nk / UM_SEG;
                if (ns == 0) break;
                const uint32_t idesc = tf32_idesc(UM_M, W * up_part<W>(rec[n % UP_IR].ncol));
                for (int k = 0; k < ns; ++k, ++sg) {
                    const int s = sg % UP_NS, a = sg & 1;
                    if (sg >= 2 && !(run = wait(&acc_empty[a], ((sg >> 1) - 1) & 1))) break;
                    if (!(run = wait(&full[s], (sg / UP_NS) & 1))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t d = tmem + (uint32_t)(a * UP_N);
                    const uint32_t ta = tmem + COL_A + (uint32_t)s * (UM_SEG * 2u * UM_KC);
                    const uint64_t db = desc0 + (uint64_t)((uint32_t)s * (B_STAGE >> 4));
#pragma unroll
                    for (int j = 0; j < UM_SEG * UM_KC / 8; ++j) {
                        const int h = j / (UM_KC / 8), i = j % (UM_KC / 8);  // chunk of the segment, its k step
                        const uint64_t dbh = db + (uint64_t)((h * B_CHUNK + i * 2 * UM_LBO) >> 4);
                        const uint64_t dbl = dbh + (uint64_t)((UP_N * UM_KC * 4) >> 4);
                        const uint32_t ah = ta + (uint32_t)(h * 2 * UM_KC + 8 * i);
                        umma_ts_if(el, d, ah, dbh, idesc, j > 0 ? 1u : 0u);
                        umma_ts_if(el, d, ah, dbl, idesc, 1u);
                        umma_ts_if(el, d, ah + UM_KC, dbh, idesc, 1u);
                    }
                    umma_commit_if(el, &empty[s]);
                    umma_commit_if(el, &acc_full[a]);
                }
                item_done(n);
            }
            if (!run) abort_s = 1;
            umma_commit_if(el, &fin);  // products already issued may still read the operands (see the end)
        } else if (warp == UP_SCHED) {
            // ---------------- scheduler: item records ----------------
            // Column tile z of the tiles with more than z NC / qn pairs (they come first), row tile by row
            // tile: the grid's stride deals these out evenly. (z, its first item, its tiles) move along.
            int n = 0, z = 0, first = 0, nz = g.more[0];
            bool run = true;
            for (int id = blockIdx.x; run; id += gridDim.x) {
                while (nz > 0 && id - first >= nz * g.mt) {
                    first += nz * g.mt;
                    const int64_t least = (int64_t)++z * NC / g.qn;
                    nz = least < PAIR_TILE ? g.more[least] : 0;
                }
                const bool end = nz == 0;
                const int t = g.tile0 + (end ? 0 : (id - first) % nz), m0 = end ? 0 : (id - first) / nz * UM_M;
                int4 tl = make_int4(0, 0, 0, 0);
                if (!end) {
                    tl = __ldg(g.tile + t);
                    if (m0 >= tl.z) continue;
                }
                UpItem<NC> &it = rec[n % UP_IR];
                if (n >= UP_IR && !(run = wait(&it_empty[n % UP_IR], ((n / UP_IR) - 1) & 1))) break;
                if (!end) {
                    const int ncol = min(NC, tl.y * g.qn - z * NC);
                    for (int c = lane; c < NC; c += 32) {  // past the columns: the last one again
                        const int f = z * NC + min(c, ncol - 1), q = f % g.qn;
                        const int4 rc = __ldg(g.rec + tl.x + f / g.qn);
                        const int64_t src = (int64_t)rc.y << 32 | (uint32_t)rc.x;
                        it.src[c] = TMA ? src / tl.w * g.nrhs + g.q0 + q : src * g.nrhs + (int64_t)(g.q0 + q) * tl.w;
                        it.out[c] = ((int64_t)(rc.w - g.pbase) * g.qn + q) * g.pstride + m0;
                    }
                    if (lane == 0) {
                        it.ncol = ncol;
                        it.snc = tl.w;
                        it.rows = min(UM_M, tl.z - m0);
                        it.m0 = m0;
                        it.col = (int)(__ldg(g.tile_off + t) / g.ld);
                        // k -> stored column: the column permutation inverted forward, else the row permutation
                        const int ps = __ldg(g.rec + tl.x).z;
                        it.perm = ps < 0 ? -1 : ps + (fwd ? 3 * tl.w : tl.w);
                    }
                }
                if (lane == 0) it.nk = end ? 0 : (W * tl.w + UM_KC - 1) / UM_KC;
                __syncwarp();
                if (lane == 0) mbar_arrive(&it_full[n % UP_IR]);
                ++n;
                if (end) break;
            }
            if (!run) abort_s = 1;
        }
    } else {
        // ---------------- drain warps: FP64 sums of the segments, then the pairs' columns ----------------
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(UP_REG_D));
        const int row = 32 * (warp & 3) + lane, half = (warp - UP_D0) >> 2;
        const uint32_t tl = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
        constexpr int HC = NC / 2;  // columns of this warp: 16 complex or 32 real
        int gs = 0;  // segments so far
        bool run = true;
        for (int n = 0; run; ++n) {
            if (!(run = item(n))) break;
            const UpItem<NC> &it = rec[n % UP_IR];
            const int nk = it.nk, ncol = it.ncol;
            if (nk == 0) break;
            const bool mine = half * HC < ncol;
            // first part: the columns' real (or only) sums, second: the imaginary ones / columns 16-31
            const uint32_t part0 = (uint32_t)(half * HC);
            const uint32_t part1 = W == 2 ? (uint32_t)(up_part<W>(ncol) + half * HC) : part0 + 16u;
            double sum[2][16];
#pragma unroll
            for (int e = 0; e < 16; ++e) sum[0][e] = sum[1][e] = 0.0;
            for (int k = 0; k < nk; k += UM_SEG, ++gs) {
                const int a = gs & 1;
                if (!(run = wait(&acc_full[a], (gs >> 1) & 1))) break;
                if (mine) {
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    uint32_t f0[16], f1[16];
                    tmem_ld16(tl + (uint32_t)(a * UP_N) + part0, f0);
                    tmem_ld16(tl + (uint32_t)(a * UP_N) + part1, f1);
                    tmem_wait_ld();
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    mbar_arrive(&acc_empty[a]);
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        sum[0][e] += (double)__uint_as_float(f0[e]);
                        sum[1][e] += (double)__uint_as_float(f1[e]);
                    }
                } else {
                    mbar_arrive(&acc_empty[a]);
                }
            }
            if (!run) break;
            if (row < it.rows) {
#pragma unroll
                for (int e = 0; e < HC; ++e) {
                    const int c = half * HC + e;
                    if (c >= ncol) break;
                    if constexpr (W == 2) stv(prod + it.out[c] + row, cdouble{sum[0][e], sum[1][e]});
                    else prod[it.out[c] + row] = sum[e / 16][e % 16];
                }
            }
            item_done(n);
        }
        if (!run) abort_s = 1;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();  // every role has left its loop
    // products already issued may still read the operands and write tensor memory
    if (warp == UP_MMA && lane == 0) mbar_wait(&fin, 0, UM_SPIN_FINAL);
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

bool i2o_umma_eligible(bool cplx, int precision, const DMap &m, int nq) {
    // narrower blocks, and those of 4 FP32 columns whose pair products fit the buffer, have FP64 sums
    // (PAIR_MAX_COLS32); without a buffer 4 columns are the least that fill a quarter of the MMA tile
    return precision == H2B_FP32 && m.coupling_kind == H2B_COUPLING_DENSE && (cplx ? 2 : 1) * nq >= 4;
}

// A 2-D tensor map of `rows` rows of `inner` FP32 values, `stride` bytes apart, for boxes of `boxrows`
// rows of `box` values (1: gathers of four rows).
static cudaError_t up_map(CUtensorMap *map, const void *base, uint64_t inner, uint64_t rows, uint64_t stride,
                          uint32_t box, uint32_t boxrows, bool swizzle) {
    static const auto encode = []() -> PFN_cuTensorMapEncodeTiled_v12000 {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &found) != cudaSuccess ||
            found != cudaDriverEntryPointSuccess)
            return nullptr;
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }();
    if (!encode) return cudaErrorNotSupported;
    const cuuint64_t dims[2] = {inner, rows}, strides[1] = {stride};
    const cuuint32_t boxes[2] = {box, boxrows}, ones[2] = {1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void *>(base), dims, strides, boxes, ones,
                              CU_TENSOR_MAP_INTERLEAVE_NONE,
                              swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t launch_i2o_umma(bool cplx, const DMap &m, const DSide &recv, const DSide &src, const int *nodes,
                            int nnodes, const FarArgs &fa, int maxcoef, const PairTiles *pt, cudaStream_t st) {
    if (nnodes == 0) return cudaSuccess;
    const int nq = m.ncomp * fa.nrhs;
    const int ntmax = cplx ? UM_NT_MAX_CPLX : UM_NT_MAX_REAL;
    // right-hand sides per tile: at most ntmax, tiles of equal width
    const int ntiles = (nq + ntmax - 1) / ntmax;
    // a multiple of 8, so that the imaginary rows of a complex tile start on a 16-column boundary
    // of tensor memory; rows past the right-hand sides are zero
    const int qt_max = ((nq + ntiles - 1) / ntiles + 7) / 8 * 8;
    const int np = (((cplx ? 2 : 1) * qt_max + 15) / 16) * 16;
    // expanded moment stages (hi and lo), the raw moment ring and the coupling column stages
    const size_t eb = cplx ? 8 : 4, kq = cplx ? UM_KC / 2 : UM_KC;
    const size_t raw = ((size_t)UM_RS * qt_max * UM_RAWROW + 127) & ~(size_t)127;
    // whole columns of stored blocks, one shape, four to a gather: columns of at most 256 FP32 values,
    // multiples of 32 bytes apart
    const int W = cplx ? 2 : 1, ld = pt ? pt->nc32 : 0;
    const int pitch = (ld * W * 4 + 31) / 32 * 32;
    const bool tma = pt && pt->stored32 && pitch <= 1024;
    CUtensorMap blocks{};
    if (tma) {
        const cudaError_t em = up_map(&blocks, pt->blocks32, (uint64_t)ld * W, (uint64_t)pt->cols32, (uint64_t)ld * W * 4,
                                      pitch / 4, 1, false);
        if (em != cudaSuccess) return em;
    }
    const size_t acols = (size_t)UM_AR * ((kq * (tma ? (size_t)pitch : maxcoef * eb) + 127) & ~(size_t)127);
    size_t smem = (size_t)UM_NS * 2 * np * UM_KC * 4 + raw;
    // the coupling column stages grow with the block size; blocks whose stages do not fit beside
    // the moment stages are read by the register path instead
    int dev = 0, optin = 0;
    cudaError_t e0 = cudaGetDevice(&dev);
    if (e0 == cudaSuccess) e0 = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e0 != cudaSuccess) return e0;
    DMap mm = m;
    const bool fits = smem + acols + UM_STATIC <= (size_t)optin;
    if ((tma || mm.cpl_vec) && fits)
        smem += acols;
    else
        mm.cpl_vec = 0;
    const dim3 grid(nnodes, (maxcoef + UM_M - 1) / UM_M, ntiles);
    auto go = [&](auto kern, auto *am, auto *dm) {
        cudaError_t e = allow_most_smem(kern, UM_STATIC);
        if (e != cudaSuccess) return e;
        kern<<<grid, tma && fits ? UM_THREADS + 32 : UM_THREADS, smem, st>>>(mm, recv, src, nodes, fa.mode, fa.nrhs, qt_max,
                                                                            am, dm, blocks, pitch, std::max(ld, 1));
        return cudaGetLastError();
    };
    if (cplx) {
        const cfloat *am = static_cast<const cfloat *>(fa.am);
        cfloat *dm = static_cast<cfloat *>(fa.dm);
        return tma && fits ? go(&i2o_umma_kernel<cfloat, true>, am, dm) : go(&i2o_umma_kernel<cfloat, false>, am, dm);
    }
    const float *am = static_cast<const float *>(fa.am);
    float *dm = static_cast<float *>(fa.dm);
    return tma && fits ? go(&i2o_umma_kernel<float, true>, am, dm) : go(&i2o_umma_kernel<float, false>, am, dm);
}

bool i2o_umma_pairs_eligible(bool cplx, int precision, const DMap &m, int nq, const PairTiles &pt, size_t prod_bytes) {
    return i2o_umma_eligible(cplx, precision, m, nq) && pt.tile32 && !pt.units.empty() &&
           (int64_t)prod_bytes >= pt.unit_elems * (int64_t)(cplx ? sizeof(cdouble) : sizeof(double));
}

cudaError_t launch_i2o_umma_pairs(bool cplx, const DMap &m, const DSide &recv, const PairTiles &pt, const FarArgs &fa,
                                  int maxcoef, cudaStream_t st) {
    const int nq = m.ncomp * fa.nrhs;
    int dev = 0, nsm = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err == cudaSuccess) err = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (err != cudaSuccess) return err;
    const int W = cplx ? 2 : 1, cols = UP_N / W, nc = pt.nc32, snc = pt.snc32;
    const int ld = cplx ? up_ld<cfloat>(nc) : up_ld<float>(nc);
    // bytes of a copied block column: 128 rows, or the whole block's in multiples of 32 (four columns to a
    // gather, whose destination is 128-byte aligned)
    const int pitch = std::min(UM_M * W, (ld * W + 7) / 8 * 8) * 4;
    // moment columns of whole 16 bytes are gathered, others copied element by element
    const bool tma = (snc * W * 4) % 16 == 0;
    CUtensorMap blocks{}, moments{};
    err = up_map(&blocks, pt.blocks32, (uint64_t)ld * W, (uint64_t)pt.cols32, (uint64_t)ld * W * 4, pitch / 4, 1, false);
    // right-hand sides per pass, and how many of one pair's lie side by side in every tile's columns: they
    // are copied as one box of rows
    const int qc = (int)std::min<int64_t>(std::min(nq, 1024), (int64_t)fa.prod_bytes / (pt.unit_elems * (cplx ? 16 : 8)));
    int rowbox = 4;
    for (int b = cols; b >= 8 && rowbox == 4; b /= 2)
        if (qc % b == 0 && nq % b == 0) rowbox = b;
    if (err == cudaSuccess && tma)
        err = up_map(&moments, fa.am, (uint64_t)snc * W, (uint64_t)pt.src_cols * fa.nrhs, (uint64_t)snc * W * 4, UM_KC,
                     rowbox == 4 ? 1 : rowbox, true);
    if (err != cudaSuccess) return err;
    const size_t raw = ((size_t)UP_RS * cols * (tma ? up_raw_row<true>() : up_raw_row<false>()) + 1023) & ~(size_t)1023;
    const size_t smem = (size_t)UP_NS * UM_SEG * 2 * UP_N * UM_KC * 4 + raw +
                        (size_t)(cplx ? up_ar<2>() : up_ar<1>()) * UM_KC * 4 * UM_M + 1024;
    auto go = [&](auto kern, const auto *am, auto *prod) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        for (const PairUnit &u : pt.units)
            for (int q0 = 0; q0 < nq; q0 += qc) {
                const int qn = std::min(qc, nq - q0);
                UpArgs g{pt.rec, pt.tile32, pt.tile32_off, u.tile32_0, (nc + UM_M - 1) / UM_M, {}, fa.mode, fa.nrhs, q0, qn,
                         u.p0, pt.pstride, ld, pitch, rowbox};
                int64_t items = 0;
                std::copy(u.more32, u.more32 + PAIR_TILE, g.more);
                for (int64_t z = 0; z * cols / qn < PAIR_TILE; ++z) items += (int64_t)g.more[z * cols / qn] * g.mt;
                if (items > INT32_MAX) return cudaErrorInvalidValue;
                kern<<<(unsigned)std::min<int64_t>(nsm, items), UP_THREADS, smem, st>>>(m, g, blocks, moments, am, prod);
                e = launch_i2o_pairs_sum(cplx, H2B_FP32, m, recv, pt, u, fa, maxcoef, q0, qn, st);
                if (e != cudaSuccess) return e;
            }
        return cudaGetLastError();
    };
    if (cplx) {
        const cfloat *am = static_cast<const cfloat *>(fa.am);
        cdouble *prod = static_cast<cdouble *>(fa.prod);
        return tma ? go(&i2o_umma_pairs_kernel<cfloat, true>, am, prod) : go(&i2o_umma_pairs_kernel<cfloat, false>, am, prod);
    }
    const float *am = static_cast<const float *>(fa.am);
    double *prod = static_cast<double *>(fa.prod);
    return tma ? go(&i2o_umma_pairs_kernel<float, true>, am, prod) : go(&i2o_umma_pairs_kernel<float, false>, am, prod);
}

cudaError_t read_umma_timeouts(unsigned *count) {
    return cudaMemcpyFromSymbol(count, g_umma_timeouts, sizeof(unsigned));
}

cudaError_t copy_umma_timeouts_async(unsigned *host, cudaStream_t st) {
    return cudaMemcpyFromSymbolAsync(host, g_umma_timeouts, sizeof(unsigned), 0, cudaMemcpyDeviceToHost, st);
}

cudaError_t set_umma_wait_limit(unsigned limit) {
    const unsigned v = limit ? limit : UM_SPIN;
    return cudaMemcpyToSymbol(g_umma_wait_limit, &v, sizeof(unsigned));
}

}  // namespace h2b
