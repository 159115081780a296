// B1 dense I2O with FP64 sums: one matrix product per stored coupling block, then one sum per
// receiving node.
//
// l_r = sum over the pairs of r of op(B_pair) m_src (translateintonode!,
// src/farinteractions/traversalhelpers.jl:167-219, with applycouplingkernel! of
// src/farinteractions/i2otranslations/i2otranslationcollection.jl:367-409 and the orientation rule
// of i2oprotocol.jl:87-92). Many pairs read one stored block (a translation in a uniform tree, a
// symmetry orbit of translations when the couplings are symmetry-reduced), so the pairs are sorted
// by block when the core is built and the I2O runs as two launches:
//   * i2o_pairs_kernel: the moments of a run of pairs are the columns of one matrix product with
//     the block they share; every pair's product goes to its own column of a buffer;
//   * i2o_pairs_sum_kernel: every receiving node adds its pairs' columns in list order (the same
//     order on every call: no atomics) and writes its moments once.
// The permutations of a symmetry-reduced pair (symmetryreduceddense.jl:84-95) move to the gather of
// its moments (columns of the block) and to the row its sum reads (rows of the block), so pairs of
// one orbit share a tile whatever their permutations are.
//
// What bounds it: the FP64 tensor cores (37 TFLOP/s here, mma.sync m8n8k4 .f64). A product reads
// its block once per 64 columns and writes 16 bytes per complex sum (8 real) per row, read once by
// the sums: 8.5 % of the time at 216 complex coefficients, about half at 64 real ones. Measured
// (I2O per product, FP64): 65,536-point Helmholtz sphere, p = 6, 1 right-hand side 7.73 -> 0.91 ms;
// 262,144 points, 32 right-hand sides 211 -> 104 ms (28.5 TFLOP/s); 8,192-point Laplace cube, p = 4,
// unreduced blocks 2.56 -> 0.050 ms, against chunks of 16 receiving nodes that each staged every
// block they read (1-4 field columns) and one CTA per receiving node (wider blocks).
#include <algorithm>
#include <type_traits>

#include "h2b_internal.cuh"

namespace h2b {

namespace {

constexpr int PK_THREADS = 256;
constexpr int PK_WARPS = PK_THREADS / 32;
constexpr int PK_N = PAIR_TILE;  // columns per tile: eight 8-wide column blocks
// Rows per tile: at most 72, nine 8-row blocks, so that 216 coefficients (6^3) are three whole
// tiles and 125 (5^3) two of 64.
constexpr int PK_MB = 9;

// Stages in shared memory: 16 values of k each (two whole stages hid the copies as well as four of 8
// complex or three of 16 real values and halve the barriers: 262,144-point sphere, 32 right-hand sides
// 121 -> 112 ms, 30,011-point cube, 16 right-hand sides 3.05 -> 2.80 ms; FP32 values lost 5 %), and the
// row strides, which keep a fragment's 32 lanes (8 rows or columns x 4 k) on distinct banks: rows of
// KC + 4 elements where k is contiguous, columns of 72 + 4 (8-byte elements), 72 + 2 (16-byte) or 72
// (4-byte) elements where rows are. Real maps fit three CTAs on an SM (short products: a CTA's first
// loads cost as much as half its arithmetic at 64 coefficients), complex ones two.
template <class T> struct PkGeom {
    static constexpr bool CPLX = ScalarTraits<T>::is_complex;
    static constexpr int KC = 16;
    static constexpr int STAGES = !CPLX && sizeof(T) == 4 ? 3 : 2;
    static constexpr int CTAS = CPLX ? 2 : 3;
    static constexpr int LDK = KC + 4;                                          // k contiguous
    static constexpr int LDM = 8 * PK_MB + (sizeof(T) == 16 ? 2 : sizeof(T) == 8 ? 4 : 0);  // rows contiguous
    static constexpr int ASZ = 8 * PK_MB * LDK > KC * LDM ? 8 * PK_MB * LDK : KC * LDM;
    static constexpr int XSZ = PK_N * LDK;
    static constexpr size_t BYTES = (size_t)STAGES * (ASZ + XSZ) * sizeof(T);
};

__device__ __forceinline__ int pk_ncoef(const DSide &s, int lvl) {
    return s.shape[3 * lvl] * s.shape[3 * lvl + 1] * s.shape[3 * lvl + 2];
}

// element copy global -> shared; ok = false writes zeros and reads nothing
template <int EB>
__device__ __forceinline__ void pk_copy(uint32_t dst, const void *src, bool ok) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(EB), "r"(ok ? EB : 0)
                 : "memory");
}

__device__ __forceinline__ void pk_dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// One 8 x 8 block of sums: lane holds C[lane / 4][2 (lane % 4) + h]; complex blocks take four real
// products per step (re = ar br - ai bi, im = ar bi + ai br).
template <class A> struct PkAcc;
template <> struct PkAcc<double> {
    double c[2];
    __device__ __forceinline__ void zero() { c[0] = c[1] = 0.0; }
    __device__ __forceinline__ void step(double a, double b) { pk_dmma(c, a, b); }
    __device__ __forceinline__ double get(int h) const { return c[h]; }
};
template <> struct PkAcc<cdouble> {
    double re[2], im[2];
    __device__ __forceinline__ void zero() { re[0] = re[1] = im[0] = im[1] = 0.0; }
    __device__ __forceinline__ void step(cdouble a, cdouble b) {
        pk_dmma(re, a.x, b.x);
        pk_dmma(im, a.x, b.y);
        pk_dmma(re, -a.y, b.y);
        pk_dmma(im, a.y, b.x);
    }
    __device__ __forceinline__ cdouble get(int h) const { return {re[h], im[h]}; }
};

struct PkArgs {
    const int4 *rec;           // per pair: {moment offset (low, high), permutation set or -1, pair}
    const int4 *tile;          // {first record, pairs, rows, k}
    const int64_t *tile_off;   // element offset of the tile's block
    int tile0, nrhs, q0, qn, pbase, pstride;
    bool adj;
};

// The product of one CTA's tile with MW x NW 8 x 8 blocks per warp: warp w takes column blocks
// NW (w % WN) .. and row blocks w / WN, w / WN + WM, ... (past the tile: the last one again, never
// stored).
template <class T, bool FWD, int MW, int NW, int WN>
__device__ __forceinline__ void pk_tile(const DMap &m, const PkArgs &g, const T *__restrict__ B, int nc, int kk, int m0,
                                        int mt, int ncol, const int64_t *col_src, const int *col_perm,
                                        const int64_t *col_out, const T *__restrict__ am, unsigned char *pk_smem,
                                        typename ScalarTraits<T>::Acc *__restrict__ prod) {
    using A = typename ScalarTraits<T>::Acc;
    using G = PkGeom<T>;
    constexpr int KC = G::KC, EB = sizeof(T), ST = G::STAGES, WM = PK_WARPS / WN;
    constexpr uint32_t STAGE = (G::ASZ + G::XSZ) * EB;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nk = (kk + KC - 1) / KC;
    const uint32_t smem = (uint32_t)__cvta_generic_to_shared(pk_smem);

    // the block: rows contiguous, a warp takes every eighth k and its lanes the rows, or k contiguous,
    // a warp's lanes take KC k of 32 / KC rows
    constexpr int RL = 32 / KC;  // rows (or columns) per warp copy where lanes run along k
    constexpr int AJ = FWD ? (8 * PK_MB + 31) / 32 : (8 * PK_MB + RL * PK_WARPS - 1) / (RL * PK_WARPS);
    constexpr int AK = FWD ? KC / PK_WARPS : 1;
    const int kl = FWD ? warp : lane % KC, il = FWD ? lane : RL * warp + lane / KC;
    const T *pa = FWD ? B + m0 + il + (int64_t)kl * nc : B + kl + (int64_t)(m0 + il) * kk;
    const uint32_t da = smem + (uint32_t)((FWD ? kl * G::LDM + il : il * G::LDK + kl) * EB);
    // the columns: KC k of 32 / KC columns per warp copy, read through the column's permutation, whose
    // entries are loaded one stage ahead
    constexpr int XU = PK_N / (RL * PK_WARPS);
    const int xk = lane % KC;
    const T *px[XU];
    const int *pp[XU];
    int xi[XU];
    bool xok[XU];
    const uint32_t dx = smem + (uint32_t)((G::ASZ + (RL * warp + lane / KC) * G::LDK + xk) * EB);
#pragma unroll
    for (int u = 0; u < XU; ++u) {
        const int c = RL * (warp + PK_WARPS * u) + lane / KC;
        xok[u] = c < ncol;
        px[u] = am + (xok[u] ? col_src[c] : 0);
        pp[u] = xok[u] && col_perm[c] >= 0 ? m.perm + col_perm[c] : nullptr;
    }
    auto fetch = [&](int kc) {
        const int k = min(kc * KC + xk, kk - 1);
#pragma unroll
        for (int u = 0; u < XU; ++u) xi[u] = pp[u] ? __ldg(pp[u] + k) : k;
    };
    auto issue = [&](int kc) {
        const uint32_t so = (uint32_t)(kc % ST) * STAGE;
        const int k0 = kc * KC;
#pragma unroll
        for (int a = 0; a < AK; ++a) {
            const bool kin = k0 + kl + (FWD ? PK_WARPS * a : 0) < kk;
#pragma unroll
            for (int j = 0; j < AJ; ++j) {
                const int i = FWD ? il + 32 * j : il + RL * PK_WARPS * j;
                if (i < mt) {
                    if constexpr (FWD)
                        pk_copy<EB>(da + so + (uint32_t)((PK_WARPS * a * G::LDM + 32 * j) * EB),
                                    kin ? pa + 32 * j + (int64_t)(PK_WARPS * a) * nc : B, kin);
                    else
                        pk_copy<EB>(da + so + (uint32_t)(RL * PK_WARPS * j * G::LDK * EB),
                                    kin ? pa + (int64_t)(RL * PK_WARPS * j) * kk : B, kin);
                }
            }
        }
        pa += FWD ? (int64_t)KC * nc : KC;
        const bool xin = k0 + xk < kk;
#pragma unroll
        for (int u = 0; u < XU; ++u)
            if (xok[u]) pk_copy<EB>(dx + so + (uint32_t)(RL * PK_WARPS * u * G::LDK * EB), px[u] + xi[u], xin);
        fetch(kc + 1);
    };

    const int g4 = lane >> 2, t4 = lane & 3;
    const int nb0 = NW * (warp % WN), mb0 = warp / WN;
    const bool busy = 8 * nb0 < ncol;
    int aoff[MW];  // element offset of the lane's row in a stage
#pragma unroll
    for (int j = 0; j < MW; ++j) {
        const int i = 8 * min(mb0 + j * WM, PK_MB - 1) + g4;
        aoff[j] = FWD ? t4 * G::LDM + i : i * G::LDK + t4;
    }
    PkAcc<A> acc[MW][NW];
#pragma unroll
    for (int j = 0; j < MW; ++j)
#pragma unroll
        for (int n = 0; n < NW; ++n) acc[j][n].zero();
    fetch(0);
#pragma unroll
    for (int s = 0; s < ST - 1; ++s) {
        if (s < nk) issue(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int kc = 0; kc < nk; ++kc) {
        asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");  // this thread's stage kc
        __syncthreads();  // everyone's; and the stage issued next was read in the last step
        if (kc + ST - 1 < nk) issue(kc + ST - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (busy) {
            const T *as = reinterpret_cast<const T *>(pk_smem + (uint32_t)(kc % ST) * STAGE);
            const T *xs = as + G::ASZ + (8 * nb0 + g4) * G::LDK + t4;
#pragma unroll
            for (int k = 0; k < KC; k += 4) {
                A b[NW];
#pragma unroll
                for (int n = 0; n < NW; ++n) b[n] = wide(ldv(xs + 8 * n * G::LDK + k));
#pragma unroll
                for (int j = 0; j < MW; ++j) {
                    const A a = wide(cj(ldv(as + aoff[j] + (FWD ? k * G::LDM : k)), g.adj));
#pragma unroll
                    for (int n = 0; n < NW; ++n) acc[j][n].step(a, b[n]);
                }
            }
        }
    }
    if (!busy) return;
#pragma unroll
    for (int n = 0; n < NW; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c = 8 * (nb0 + n) + 2 * t4 + h;
            if (c >= ncol) continue;
            A *out = prod + col_out[c];
#pragma unroll
            for (int j = 0; j < MW; ++j) {
                const int i = 8 * (mb0 + j * WM) + g4;
                if (i < mt) stv(out + i, acc[j][n].get(h));
            }
        }
}

// Tile blockIdx.x of the unit, row tile blockIdx.y, columns [64 blockIdx.z, + 64) of the tile's
// pairs x qn right-hand sides (pair-major). FWD: the stored block is (receiver x source), rows
// contiguous; otherwise it is the (source x receiver) block of the mirrored pair, read transposed
// (conjugated for adjoint maps), k contiguous. Pair p's product for right-hand side q0 + q starts
// at prod[((p - pbase) qn + q) pstride].
template <class T, bool FWD>
__global__ void __launch_bounds__(PK_THREADS, PkGeom<T>::CTAS)
i2o_pairs_kernel(DMap m, PkArgs g, const T *am, typename ScalarTraits<T>::Acc *prod) {
    extern __shared__ __align__(16) unsigned char pk_smem[];
    __shared__ int64_t col_src[PK_N], col_out[PK_N];  // per column: its moments and its product
    __shared__ int col_perm[PK_N];                    // the permutation its moments are read through, -1: none
    const int4 tl = __ldg(g.tile + g.tile0 + blockIdx.x);
    const int64_t off = __ldg(g.tile_off + g.tile0 + blockIdx.x);
    const int c0 = blockIdx.z * PK_N;
    const int nc = tl.z, kk = tl.w;
    const int nmt = (nc + 8 * PK_MB - 1) / (8 * PK_MB);      // row tiles of equal 8-row blocks
    const int bm = 8 * ((nc + 8 * nmt - 1) / (8 * nmt));
    const int m0 = blockIdx.y * bm;
    if (c0 >= tl.y * g.qn || m0 >= nc) return;
    const int ncol = min(PK_N, tl.y * g.qn - c0), mt = min(bm, nc - m0);
    const T *B = static_cast<const T *>(m.cpl) + off;
    if (threadIdx.x < ncol) {
        const int c = threadIdx.x, q = (c0 + c) % g.qn;
        const int4 rc = __ldg(g.rec + tl.x + (c0 + c) / g.qn);
        col_src[c] = ((int64_t)rc.y << 32 | (uint32_t)rc.x) * g.nrhs + (int64_t)(g.q0 + q) * kk;
        col_out[c] = ((int64_t)(rc.w - g.pbase) * g.qn + q) * g.pstride + m0;
        // sets [rowperm | rowperm^-1 | colperm | colperm^-1] of n each: forward products run over the
        // block's columns (x read through colperm), transposed ones over its rows (rowperm)
        col_perm[c] = rc.z < 0 ? -1 : rc.z + (FWD ? 2 * kk : 0);
    }
    chain_wait();
    __syncthreads();
    // 8 x 8 blocks per warp: wide tiles one column block per warp with all row blocks, or, for real
    // tiles of 64 rows, two column blocks with half the row blocks (six loads for eight products
    // instead of nine); narrow tiles spread the row blocks of their few column blocks over the warps
    auto run = [&](auto mw, auto nw, auto wn) {
        pk_tile<T, FWD, decltype(mw)::value, decltype(nw)::value, decltype(wn)::value>(
            m, g, B, nc, kk, m0, mt, ncol, col_src, col_perm, col_out, am, pk_smem, prod);
    };
    using std::integral_constant;
    if (ncol > 32) {
        if (mt > 64) run(integral_constant<int, 9>{}, integral_constant<int, 1>{}, integral_constant<int, 8>{});
        else if (PkGeom<T>::CPLX) run(integral_constant<int, 8>{}, integral_constant<int, 1>{}, integral_constant<int, 8>{});
        else run(integral_constant<int, 4>{}, integral_constant<int, 2>{}, integral_constant<int, 4>{});
    } else if (ncol > 16) {
        run(integral_constant<int, 5>{}, integral_constant<int, 1>{}, integral_constant<int, 4>{});
    } else if (ncol > 8) {
        run(integral_constant<int, 3>{}, integral_constant<int, 1>{}, integral_constant<int, 2>{});
    } else {
        run(integral_constant<int, 2>{}, integral_constant<int, 1>{}, integral_constant<int, 1>{});
    }
}

// Padded copies of the FP32 form's blocks for the tcgen05 kernel, made once with the core. (On the host
// they took an eighth of the core's time, 12,289 points, p = 5: 31.6 -> 27.7 ms.)
template <class T>
__global__ void pad_blocks_kernel(const T *__restrict__ src, const int64_t *__restrict__ off, int rows, int cols, bool trans,
                                  int ld, T *__restrict__ dst) {
    const T *B = src + off[blockIdx.x];
    T *out = dst + (int64_t)blockIdx.x * ld * cols;
    for (int e = threadIdx.x; e < ld * cols; e += blockDim.x) {
        const int j = e / ld, i = e - j * ld;
        out[e] = i >= rows ? T{} : B[trans ? j + (int64_t)i * cols : i + (int64_t)j * rows];
    }
}

// Receiving node nodes[blockIdx.x]: its moments for right-hand sides [q0, q0 + qn) as the sum of
// its pairs' columns, read through each pair's row permutation. Loads of eight pairs are in flight
// per thread; the sum runs in list order. (Columns copied to shared memory as they lie and permuted on
// the reads from there were slower everywhere, 65,536-point sphere, 32 right-hand sides: 2.4 -> 5 ms.)
// Bound: the loads in flight, so the registers leave room for ten blocks an SM of complex maps (48
// each; 56 before: FP32 sphere, I2O of 32 right-hand sides 12.65 -> 12.30 ms, of 8 3.78 -> 3.72), twelve
// of real ones (40, what the compiler took by itself).
template <class T>
__global__ void __launch_bounds__(128, ScalarTraits<T>::is_complex ? 10 : 12)
i2o_pairs_sum_kernel(DMap m, DSide r, const int *__restrict__ nodes, bool fwd, int nrhs, int q0, int qn, int pbase,
                     int pstride, const typename ScalarTraits<T>::Acc *prod, T *dm) {
    using A = typename ScalarTraits<T>::Acc;
    constexpr int U = 8;
    const int node = nodes[blockIdx.x];
    const int nc = pk_ncoef(r, r.level[node]);
    const int e = blockIdx.y * 128 + threadIdx.x;
    if (e >= nc * qn) return;
    const int q = e / nc, i = e % nc;
    const int p0 = r.i2o_ptr[node], p1 = r.i2o_ptr[node + 1];
    // forward: out[i] += Y[rowperm^-1[i]]; transposed: out[j] += Y[colperm^-1[j]]
    const int set = fwd ? nc : 3 * nc;
    A sum = sc_zero<A>();
    chain_wait();
    for (int p = p0; p < p1; p += U) {
        A v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int pp = min(p + u, p1 - 1);
            const int64_t ps = r.pair_perm ? __ldg(r.pair_perm + pp) : -1;
            const int row = ps < 0 ? i : __ldg(m.perm + ps + set + i);
            v[u] = ldv(prod + ((int64_t)(pp - pbase) * qn + q) * pstride + row);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (p + u < p1) sum = sum + v[u];
    }
    T out;
    narrow(sum, out);
    stv(dm + r.mom_off[node] * nrhs + (int64_t)(q0 + q) * nc + i, out);
}

template <class T>
cudaError_t launch_sum_t(const DMap &m, const DSide &r, const PairTiles &pt, const PairUnit &u, const FarArgs &fa, int maxcoef,
                         int q0, int qn, cudaStream_t st) {
    using A = typename ScalarTraits<T>::Acc;
    const dim3 grid(u.nrcv, (unsigned)(((int64_t)maxcoef * qn + 127) / 128));
    return launch_chain(chain_ahead(m, m.ncomp * fa.nrhs), i2o_pairs_sum_kernel<T>, grid, 128, 0, st, m, r, pt.rcv + u.rcv0, fa.mode == H2B_FORWARD, fa.nrhs, q0,
                        qn, u.p0, pt.pstride, static_cast<const A *>(fa.prod), static_cast<T *>(fa.dm));
}

template <class T>
cudaError_t launch_pairs_t(const DMap &m, const DSide &r, const PairTiles &pt, const FarArgs &fa, int maxcoef,
                           cudaStream_t st) {
    using A = typename ScalarTraits<T>::Acc;
    const bool fwd = fa.mode == H2B_FORWARD, adj = fa.mode == H2B_ADJOINT;
    const int nq = m.ncomp * fa.nrhs;
    const size_t sm = PkGeom<T>::BYTES;
    auto kern = fwd ? &i2o_pairs_kernel<T, true> : &i2o_pairs_kernel<T, false>;
    cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (err != cudaSuccess) return err;
    // right-hand sides per pass: as many as the largest unit's products leave room for
    const int64_t unit = pt.unit_elems * (int64_t)sizeof(A);
    // (and as the grids' second and third extents allow)
    const int qc = (int)std::min<int64_t>(std::min(nq, 1024), (int64_t)fa.prod_bytes / unit);
    const int mtiles = (maxcoef + 8 * PK_MB - 1) / (8 * PK_MB);
    A *prod = static_cast<A *>(fa.prod);
    for (const PairUnit &u : pt.units)
        for (int q0 = 0; q0 < nq; q0 += qc) {
            const int qn = std::min(qc, nq - q0);
            const dim3 grid(u.ntiles, mtiles, (u.maxpairs * qn + PK_N - 1) / PK_N);
            const PkArgs g{pt.rec, pt.tile, pt.tile_off, u.tile0, fa.nrhs, q0, qn, u.p0, pt.pstride, adj};
            err = launch_chain(chain_ahead(m, nq), kern, grid, PK_THREADS, sm, st, m, g, static_cast<const T *>(fa.am), prod);
            if (err != cudaSuccess) return err;
            err = launch_sum_t<T>(m, r, pt, u, fa, maxcoef, q0, qn, st);
            if (err != cudaSuccess) return err;
        }
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_pad_blocks(bool cplx, const void *src, const int64_t *off, int nblocks, int rows, int cols, bool trans,
                              int ld, void *dst, cudaStream_t st) {
    if (cplx)
        pad_blocks_kernel<<<nblocks, 256, 0, st>>>(static_cast<const cfloat *>(src), off, rows, cols, trans, ld,
                                                   static_cast<cfloat *>(dst));
    else
        pad_blocks_kernel<<<nblocks, 256, 0, st>>>(static_cast<const float *>(src), off, rows, cols, trans, ld,
                                                   static_cast<float *>(dst));
    return cudaGetLastError();
}

bool i2o_pairs_eligible(bool cplx, int precision, const DMap &m, int nq, const PairTiles &pt, size_t prod_bytes) {
    if (pt.units.empty() || m.coupling_kind != H2B_COUPLING_DENSE) return false;
    // the FP32 form's products have FP64 sums up to PAIR_MAX_COLS32 field columns; wider blocks take
    // the tcgen05 kernel
    if (precision == H2B_FP32 && (cplx ? 2 : 1) * nq > PAIR_MAX_COLS32) return false;
    return (int64_t)prod_bytes >= pt.unit_elems * (int64_t)(cplx ? sizeof(cdouble) : sizeof(double));
}

cudaError_t launch_i2o_pairs(bool cplx, int precision, const DMap &m, const DSide &recv, const PairTiles &pt,
                             const FarArgs &fa, int maxcoef, cudaStream_t st) {
    if (!cplx)
        return precision == H2B_FP64 ? launch_pairs_t<double>(m, recv, pt, fa, maxcoef, st)
                                     : launch_pairs_t<float>(m, recv, pt, fa, maxcoef, st);
    return precision == H2B_FP64 ? launch_pairs_t<cdouble>(m, recv, pt, fa, maxcoef, st)
                                 : launch_pairs_t<cfloat>(m, recv, pt, fa, maxcoef, st);
}

cudaError_t launch_i2o_pairs_sum(bool cplx, int precision, const DMap &m, const DSide &recv, const PairTiles &pt,
                                 const PairUnit &u, const FarArgs &fa, int maxcoef, int q0, int qn, cudaStream_t st) {
    if (!cplx)
        return precision == H2B_FP64 ? launch_sum_t<double>(m, recv, pt, u, fa, maxcoef, q0, qn, st)
                                     : launch_sum_t<float>(m, recv, pt, u, fa, maxcoef, q0, qn, st);
    return precision == H2B_FP64 ? launch_sum_t<cdouble>(m, recv, pt, u, fa, maxcoef, q0, qn, st)
                                 : launch_sum_t<cfloat>(m, recv, pt, u, fa, maxcoef, q0, qn, st);
}

}  // namespace h2b
