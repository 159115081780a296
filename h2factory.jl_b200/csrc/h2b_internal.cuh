// Internal definitions shared by the host orchestration (h2b_api.cu) and the kernels
// (h2b_kernels.cu): scalar types, the device-resident core layout, and kernel launchers.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>
#include <vector>

#include "../../include/h2b200.h"

namespace h2b {

// ---------------------------------------------------------------------------------------------
// Scalars. V is the field type of x, y and the near blocks (double or cdouble); T is the far-field
// arithmetic type (double, float, cdouble or cfloat); Toeplitz spectra are complex of T's real type.
// ---------------------------------------------------------------------------------------------
template <class R>
struct Cx {
    R x, y;
};
using cdouble = Cx<double>;
using cfloat = Cx<float>;

// Acc: the arithmetic type of every far-field sum. The FP32 form stores moments, spectra, collections,
// transfers and couplings in FP32 (half the bytes) but accumulates in FP64, so each stored
// intermediate is rounded once instead of once per operation.
template <class T> struct ScalarTraits;
template <> struct ScalarTraits<double> { using Real = double; using Complex = cdouble; using Acc = double; using CAcc = cdouble; static constexpr bool is_complex = false; };
template <> struct ScalarTraits<float> { using Real = float; using Complex = cfloat; using Acc = double; using CAcc = cdouble; static constexpr bool is_complex = false; };
template <> struct ScalarTraits<cdouble> { using Real = double; using Complex = cdouble; using Acc = cdouble; using CAcc = cdouble; static constexpr bool is_complex = true; };
template <> struct ScalarTraits<cfloat> { using Real = float; using Complex = cfloat; using Acc = cdouble; using CAcc = cdouble; static constexpr bool is_complex = true; };

template <class R> __host__ __device__ __forceinline__ Cx<R> operator+(Cx<R> a, Cx<R> b) { return {a.x + b.x, a.y + b.y}; }
template <class R> __host__ __device__ __forceinline__ Cx<R> operator-(Cx<R> a, Cx<R> b) { return {a.x - b.x, a.y - b.y}; }
template <class R> __host__ __device__ __forceinline__ Cx<R> operator*(Cx<R> a, Cx<R> b) {
    return {a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x};
}
template <class R> __host__ __device__ __forceinline__ Cx<R> operator*(R a, Cx<R> b) { return {a * b.x, a * b.y}; }
template <class R> __host__ __device__ __forceinline__ Cx<R> &operator+=(Cx<R> &a, Cx<R> b) { a.x += b.x; a.y += b.y; return a; }

__host__ __device__ __forceinline__ double conjg(double a) { return a; }
__host__ __device__ __forceinline__ float conjg(float a) { return a; }
template <class R> __host__ __device__ __forceinline__ Cx<R> conjg(Cx<R> a) { return {a.x, -a.y}; }

template <class T> __host__ __device__ __forceinline__ T sc_zero() { return T{}; }
template <class T> __host__ __device__ __forceinline__ bool is_zero(T a);
template <> __host__ __device__ __forceinline__ bool is_zero(double a) { return a == 0.0; }
template <> __host__ __device__ __forceinline__ bool is_zero(cdouble a) { return a.x == 0.0 && a.y == 0.0; }

// optional conjugation
template <class T> __host__ __device__ __forceinline__ T cj(T a, bool c) { return c ? conjg(a) : a; }

// conversions between the field type V and the far type T (same complexness)
__host__ __device__ __forceinline__ double to_t(double v, double) { return v; }
__host__ __device__ __forceinline__ float to_t(double v, float) { return (float)v; }
__host__ __device__ __forceinline__ cdouble to_t(cdouble v, cdouble) { return v; }
__host__ __device__ __forceinline__ cfloat to_t(cdouble v, cfloat) { return {(float)v.x, (float)v.y}; }
__host__ __device__ __forceinline__ double to_v(double t) { return t; }
__host__ __device__ __forceinline__ double to_v(float t) { return (double)t; }
__host__ __device__ __forceinline__ cdouble to_v(cdouble t) { return t; }
__host__ __device__ __forceinline__ cdouble to_v(cfloat t) { return {(double)t.x, (double)t.y}; }
// widening to the accumulation type and rounding back to the storage type
__host__ __device__ __forceinline__ double wide(double a) { return a; }
__host__ __device__ __forceinline__ double wide(float a) { return (double)a; }
__host__ __device__ __forceinline__ cdouble wide(cdouble a) { return a; }
__host__ __device__ __forceinline__ cdouble wide(cfloat a) { return {(double)a.x, (double)a.y}; }
__host__ __device__ __forceinline__ void narrow(double a, double &o) { o = a; }
__host__ __device__ __forceinline__ void narrow(double a, float &o) { o = (float)a; }
__host__ __device__ __forceinline__ void narrow(cdouble a, cdouble &o) { o = a; }
__host__ __device__ __forceinline__ void narrow(cdouble a, cfloat &o) { o = {(float)a.x, (float)a.y}; }
// moment <-> spectrum
template <class R> __host__ __device__ __forceinline__ Cx<R> to_cx(R a) { return {a, (R)0}; }
template <class R> __host__ __device__ __forceinline__ Cx<R> to_cx(Cx<R> a) { return a; }
template <class R> __host__ __device__ __forceinline__ void from_cx(Cx<R> s, R &out) { out = s.x; }
template <class R> __host__ __device__ __forceinline__ void from_cx(Cx<R> s, Cx<R> &out) { out = s; }
__host__ __device__ __forceinline__ void from_cx(cdouble s, float &out) { out = (float)s.x; }
__host__ __device__ __forceinline__ void from_cx(cdouble s, cfloat &out) { out = {(float)s.x, (float)s.y}; }

// One access per scalar for arrays of the library's own (a complex scalar's type only promises the
// alignment of its parts, since x and y come from the caller; ours start on 16 bytes)
template <class T> __device__ __forceinline__ T ldv(const T *p) { return *p; }
template <> __device__ __forceinline__ cdouble ldv(const cdouble *p) {
    const double2 v = *reinterpret_cast<const double2 *>(p);
    return {v.x, v.y};
}
template <> __device__ __forceinline__ cfloat ldv(const cfloat *p) {
    const float2 v = *reinterpret_cast<const float2 *>(p);
    return {v.x, v.y};
}
template <class T> __device__ __forceinline__ void stv(T *p, T v) { *p = v; }
template <> __device__ __forceinline__ void stv(cdouble *p, cdouble v) { *reinterpret_cast<double2 *>(p) = make_double2(v.x, v.y); }
template <> __device__ __forceinline__ void stv(cfloat *p, cfloat v) { *reinterpret_cast<float2 *>(p) = make_float2(v.x, v.y); }

// ---------------------------------------------------------------------------------------------
// The far passes of one column are a chain of short launches, each reading what the one before wrote.
// A kernel that calls chain_wait() before its first access to moments or pair products (reads and
// writes alike) may be launched ahead: its blocks then start, and read the map's own arrays, while the
// last blocks of the kernel before it in the stream still run. chain_wait() returns when that kernel
// has completed, and lets the next one start in turn; the pointers that it guards carry no
// __restrict__, so no load of theirs is an invariant one that could move above it. At least one
// thread of a launch must reach it. (After any other stream operation the launch is an ordinary one.)
//
// Which launches go ahead: those of one column, of dense and diagonal couplings, of up to 16 blocks
// an SM. Blocks that wait hold their places on the SMs, where the near field's kernels run meanwhile.
// Device time per product, us, ordinary -> ahead: Laplace maps of 2,048 points 36 -> 32, of 8,192 points
// 107 -> 95-97, Helmholtz ellipsoid of 20,011 points 420 -> 409, sphere of 65,536 points 1293 -> 1277 (no gain
// without the limit on blocks). Slower, so left out: Toeplitz maps (262,144 points, 1027 -> 1080) and several
// columns (12,289 points, three right-hand sides, 449 -> 456; 7,189 points, fourteen, 254 -> 266).
// ---------------------------------------------------------------------------------------------
constexpr int CHAIN_BLOCKS = 16 * 148;  // a B200 has 148 SMs

__device__ __forceinline__ void chain_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// The first kernel of a chain, launched the ordinary way, only lets the next one start.
__device__ __forceinline__ void chain_open() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---------------------------------------------------------------------------------------------
// Device-resident side of a core (all pointers device memory).
// ---------------------------------------------------------------------------------------------
struct DSide {
    int nnodes, nlevels, ndofs;
    int nvalues;             // value_ptr[nnodes]: dof entries held by the leaves
    const int *level, *parent, *sector, *child_ptr, *child, *value_ptr, *value;
    const int *shape;        // [(nlevels+1)*3]
    const int64_t *mom_off;  // [nnodes] moment offset per unit right-hand side (elements of T)
    const int64_t *spec_off; // [nnodes] spectrum offset per unit right-hand side (complex elements)
    const int64_t *coll_off; // [nnodes] leaf collection offsets (elements of T)
    const void *coll;        // T
    const int64_t *tr_off;   // [(nlevels+1)*nsectors] transfer offsets (elements of T)
    const void *tr;          // T
    const int *i2o_ptr, *i2o_src;
    const int64_t *i2o_cpl;   // coupling index of each pair
    const int64_t *pair_src;  // per pair: the source's moment / spectrum offset per unit rhs
    const int64_t *pair_cpl;  // per pair: the coupling's element offset in the coupling array
    const int64_t *pair_perm = nullptr;  // per pair: its permutation set in DMap::perm, -1 none
};

struct DMap {
    int ncomp, dim, nsectors;
    int transfer_kind, coupling_kind;
    int half_spectrum;       // Toeplitz spectra stored as half spectra (real maps, Hermitian couplings)
    int cube_ts;             // > 0: every level's padded Toeplitz arrays are cube_ts^3 (3-D cubes)
    const int64_t *cpl_off;  // [ncouplings] offsets in elements of T (dense/diag) or spectrum (Toeplitz)
    const void *cpl;
    // FP32 dense couplings for the tensor-core I2O: every block transposed, at the same offsets,
    // so that transposed / adjoint products read columns of a stored block like forward ones
    const void *cpl_t = nullptr;
    // every dense block starts on a 16-byte boundary and its columns are whole multiples of 16 bytes:
    // the tensor-core I2O then copies coupling columns with bulk (TMA) copies
    int cpl_vec = 0;
    // permuted dense couplings: sets [rowperm | rowperm^-1 | colperm | colperm^-1], n entries each
    const int *perm = nullptr;
};

// One oriented near operator: for every output leaf (group), the dense blocks that write its rows.
// Blocks are column-major, output rows x input columns, leading dimension near_padded_ld(rows).
struct NearOp {
    int ngroups = 0;
    const int *grp_leaf = nullptr;  // [ngroups] output leaf (every output leaf has a group)
    const int64_t *blk_off = nullptr;  // per block id: element offset in `data`
    // (block, 32-column chunk) work units of each group in block order: {first input value,
    // columns (<= 32), element offset of the chunk's first column in `data` (low, high 32 bits;
    // unused by the matrix-free kernels)}; one independent 16-byte load per unit instead of a
    // chain block -> input leaf -> values
    const int *unit_ptr = nullptr;  // [ngroups+1]
    const int4 *unit = nullptr;
    const void *data = nullptr;     // V
    // (group, 32-row slab) pairs covering every output row: the work items of the complex
    // tensor-core near kernel, one warp each
    int nslabs = 0;
    const int2 *slab = nullptr;
};

struct DNear {
    NearOp fwd;              // N: rows on the test side, columns on the trial side
    NearOp tr;               // N^T (unused when symmetric)
    bool symmetric = false;  // N^T == N: transposed products run on `fwd`
    // matrix-free near field (kind != H2B_NEAR_STORED): entries from the points, no block data
    int kind = 0;
    double wavenumber = 0.0;
    const double *test_pts = nullptr;   // [test ndofs * 3]
    const double *trial_pts = nullptr;  // [trial ndofs * 3]
};

// Sibling groups for the Toeplitz I2O (i2o_sibling_kernel): the receiving children of one parent.
// Record `msg` as the calling thread's error text (h2b_last_error) and return `st`.
h2b_status set_error_text(h2b_status st, const char *msg);

struct SibGroups {
    int ngroups = 0;
    const int *recv = nullptr;         // [ngroups*8] receiving node per child slot, -1 if none
    const int *slen = nullptr;         // [ngroups] stored spectrum length of the group's level
    const int *ptr = nullptr;          // [ngroups+1] into src_off / kof
    const int64_t *src_off = nullptr;  // spectrum offset (per unit rhs) of each source of the union
    const int *kof = nullptr;          // [nentries*8] coupling offset of (source, slot), -1 if no pair
};

// Dense I2O with FP64 sums (h2b_pairs.cu): the pairs of one receiving side in units of consecutive
// receiving nodes, sorted inside a unit by the stored coupling block that they read (then by its
// permutations), and cut into tiles of at most PAIR_TILE pairs of one block, most pairs first. A unit's products take
// unit_elems scalars at most per right-hand side: pair p's at (p - p0) pstride.
constexpr int PAIR_TILE = 64;
struct PairUnit {
    int tile0, ntiles;  // tiles of the unit
    int maxpairs;       // pairs of its largest tile
    int tile32_0;          // its first one of tile32
    int more32[PAIR_TILE]; // tiles of tile32 with more than c pairs
    int rcv0, nrcv;     // its receiving nodes
    int p0;             // its first pair
};
struct PairTiles {
    std::vector<PairUnit> units;  // host
    const int4 *rec = nullptr;    // pairs, tile by tile: {source's moment offset (low, high 32 bits) per
                                  // unit rhs, permutation set in DMap::perm or -1, pair}
    const int4 *tile = nullptr;   // {first record, pairs, rows, k}
    const int64_t *tile_off = nullptr;  // element offset of each tile's block in DMap::cpl
    const int *rcv = nullptr;     // receiving nodes, unit by unit
    // FP32 form on the tcgen05 tensor cores: tiles of pairs that read one block through one
    // permutation, the element offset of each one's block in `blocks32` (rows x k, column-major, columns
    // padded to whole 16 bytes: the stored blocks forward, their transposes for the other orientations)
    const int4 *tile32 = nullptr;
    const int64_t *tile32_off = nullptr;
    const void *blocks32 = nullptr;
    int nc32 = 0, snc32 = 0;      // rows and k of every block
    int64_t cols32 = 0;           // columns in blocks32
    bool stored32 = false;        // blocks32 is the stored array: a pair's block starts at its pair_cpl
    int64_t src_cols = 0;         // source moment columns per unit rhs
    int64_t unit_elems = 0;
    int pstride = 1;              // scalars per pair and right-hand side
};

// A launch that needs more than 48 KB of dynamic shared memory asks for it by an attribute of the kernel,
// one value per device that all host threads share. The value set here is the same in every call (all
// that a block may have beside `static_bytes` of static arrays), so that no thread can lower it between
// another thread's call and that thread's launch, as a value that follows the map could.
constexpr int SMEM_BLOCK_MAX = 227 * 1024;

template <class... P>
cudaError_t allow_most_smem(void (*kernel)(P...), int static_bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BLOCK_MAX - static_bytes);
}

inline bool chain_ahead(const DMap &m, int nq) { return nq == 1 && m.coupling_kind != H2B_COUPLING_TOEPLITZ; }

template <class... P, class... A>
cudaError_t launch_chain(bool ahead, void (*kernel)(P...), dim3 grid, unsigned block, size_t smem, cudaStream_t st,
                         A &&...args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = ahead && (int64_t)grid.x * grid.y * grid.z <= CHAIN_BLOCKS ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

// Per-call arguments of the far passes.
struct FarArgs {
    int mode;     // H2B_FORWARD / H2B_TRANSPOSE / H2B_ADJOINT
    int nrhs;
    void *am;     // aggregation moments (T)
    void *dm;     // disaggregation moments (T)
    void *as;     // aggregation spectra (complex of T's real)
    void *ds;     // disaggregation spectra
    void *prod = nullptr;   // pair products of the dense I2O
    size_t prod_bytes = 0;
};

// ---------------------------------------------------------------------------------------------
// Launchers (h2b_kernels.cu). Each enqueues on `st` and returns the launch error.
// `precision`: 0 = T is FP64, 1 = FP32; `cplx`: field is complex.
// ---------------------------------------------------------------------------------------------
cudaError_t launch_leaf_aggregate(bool cplx, int precision, const DMap &m, const DSide &s,
                                  const int *leaves, int nleaves, int maxcoef, bool conjc,
                                  const FarArgs &fa, const void *x, int64_t ldx, cudaStream_t st);
cudaError_t launch_transfer_up(bool cplx, int precision, const DMap &m, const DSide &s,
                               const int *nodes, int nnodes, bool conjt, const FarArgs &fa,
                               int maxcoef, int maxsep, cudaStream_t st);
cudaError_t launch_toeplitz_in(bool cplx, int precision, const DMap &m, const DSide &s,
                               const int *nodes, int nnodes, bool inverse, const FarArgs &fa,
                               int maxtsize, int maxaxis, cudaStream_t st);
cudaError_t launch_i2o(bool cplx, int precision, const DMap &m, const DSide &recv,
                       const DSide &src, const int *nodes, int nnodes, const FarArgs &fa,
                       int maxcoef, int maxtsize, int maxhalf, const PairTiles *pt, cudaStream_t st);
cudaError_t launch_toeplitz_out(bool cplx, int precision, const DMap &m, const DSide &s,
                                const int *nodes, int nnodes, bool inverse, const FarArgs &fa,
                                int maxtsize, int maxaxis, cudaStream_t st);
// Dense I2O of the FP32 form on the tcgen05 tensor cores (h2b_umma.cu): taken when the coupling
// storage is dense and the right-hand sides make at least 4 FP32 columns (MMA N padded to 16).
bool i2o_umma_eligible(bool cplx, int precision, const DMap &m, int nq);
cudaError_t launch_i2o_umma(bool cplx, const DMap &m, const DSide &recv, const DSide &src, const int *nodes,
                            int nnodes, const FarArgs &fa, int maxcoef, const PairTiles *pt, cudaStream_t st);
// The sums of one unit's pair products (right-hand sides [q0, q0 + qn)) into the receiving nodes' moments.
cudaError_t launch_i2o_pairs_sum(bool cplx, int precision, const DMap &m, const DSide &recv, const PairTiles &pt,
                                 const PairUnit &u, const FarArgs &fa, int maxcoef, int q0, int qn, cudaStream_t st);
// FP32 blocks (rows x cols, at element offsets `off` of `src`; stored transposed when `trans`) copied one after
// another to `dst` as columns of `ld` elements, zeros past the rows.
cudaError_t launch_pad_blocks(bool cplx, const void *src, const int64_t *off, int nblocks, int rows, int cols, bool trans,
                              int ld, void *dst, cudaStream_t st);
// The FP32 form's dense I2O by stored block on the tcgen05 tensor cores (PairTiles::tile32).
bool i2o_umma_pairs_eligible(bool cplx, int precision, const DMap &m, int nq, const PairTiles &pt, size_t prod_bytes);
cudaError_t launch_i2o_umma_pairs(bool cplx, const DMap &m, const DSide &recv, const PairTiles &pt, const FarArgs &fa,
                                  int maxcoef, cudaStream_t st);
// mbarrier waits of the tensor-core kernels that gave up on the current device (0 in a healthy run)
cudaError_t read_umma_timeouts(unsigned *count);
// the same count copied to host memory in order on `st`
cudaError_t copy_umma_timeouts_async(unsigned *host, cudaStream_t st);
// try_wait attempts of every bounded mbarrier wait on the current device (0: the default)
cudaError_t set_umma_wait_limit(unsigned limit);
cudaError_t launch_i2o_siblings(bool cplx, int precision, const DMap &m, const DSide &recv,
                                const SibGroups &g, int maxslen, const FarArgs &fa, cudaStream_t st);
// The dense I2O by stored block (PairTiles) with FP64 sums: every FP64 map whose pair products fit
// `prod_bytes`, and FP32 maps of at most PAIR_MAX_COLS32 field columns (W x nq, W = 2 complex).
//
// Why 4: a precision line, not a crossover. FP32 blocks of up to 4 field columns have FP64 sums, whose error
// is the smaller one; wider ones have the tcgen05 kernels' FP32 segments. Measured (I2O, ms, FP64 sums |
// tcgen05; p real or complex coefficients an axis):
//   columns                          4              6              8              16             32
//   12,289 points, p = 4 real    0.149 | 0.175  0.196 | 0.237  0.255 | 0.302  0.447 | 0.535  0.888 | 1.058
//   12,289 points, p = 5 real    0.380 | 0.255  0.536 | 0.355  0.691 | 0.443  1.361 | 0.863  2.716 | 1.693
//   12,289 points, p = 6 real    0.919 | 4.386  1.388 | 4.391  1.816 | 4.396  3.557 | 4.447  7.097 | 4.656
//   65,536 points, p = 6 complex 1.608 | 1.078  2.480 | 1.642  3.213 | 1.986  6.284 | 3.211  12.50 | 5.944
// So tcgen05 by stored block is the faster form from 125 coefficients on, and the FP64 sums are faster than
// what wider blocks get here at 64 real coefficients, and at 216 real ones (seven chunks, per receiving
// node) up to about 20 columns.
constexpr int PAIR_MAX_COLS32 = 4;
bool i2o_pairs_eligible(bool cplx, int precision, const DMap &m, int nq, const PairTiles &pt, size_t prod_bytes);
cudaError_t launch_i2o_pairs(bool cplx, int precision, const DMap &m, const DSide &recv, const PairTiles &pt,
                             const FarArgs &fa, int maxcoef, cudaStream_t st);
cudaError_t launch_transfer_down(bool cplx, int precision, const DMap &m, const DSide &s,
                                 const int *nodes, int nnodes, const uint8_t *received,
                                 const FarArgs &fa, int maxcoef, int maxsep, cudaStream_t st);
cudaError_t launch_leaf_disaggregate(bool cplx, int precision, const DMap &m, const DSide &s,
                                     const int *leaves, int nleaves, bool conjc, const FarArgs &fa,
                                     cdouble alpha, cdouble beta, void *y, int64_t ldy,
                                     cudaStream_t st);
cudaError_t launch_near(bool cplx, int mode, const DNear &n, const DSide &test, const DSide &trial,
                        int nrhs, const void *x, int64_t ldx, void *y, int64_t ldy, cdouble alpha,
                        cdouble beta, void *xp, cudaStream_t st);
int64_t near_padded_ld(bool cplx, int n);
// right-hand sides per pass of the complex tensor-core near kernel for a block of `nrhs`
int near_rhs_block(int nrhs);
cudaError_t launch_near_repack(bool cplx, const void *src, const int64_t *src_off, const int *blk_row,
                               const int *blk_col, const DSide &rows, const DSide &cols, void *dst,
                               const int64_t *dst_off, int nblocks, bool transpose, cudaStream_t st);
cudaError_t launch_near_symcheck(bool cplx, const void *src, const int64_t *off, const int *mirror,
                                 const int *blk_row, const DSide &rows, int nblocks, int *flag,
                                 cudaStream_t st);
cudaError_t launch_zero_columns(bool cplx, int nrhs, int64_t n, void *y, int64_t ldy,
                                cudaStream_t st);

}  // namespace h2b
