// Inter-level transfers and block field operations of the FMM sweep and the
// Poisson level loop, FP64 (fields stay FP64 in every precision mode).
//
//   tp_kernel     tensor-product Lagrange transfers on Nb^3 blocks:
//                 FMM anterpolation / interpolation (include/iblgf/fmm/
//                 fmm_nli.hpp:101-247) and cell-centred interpolation /
//                 coarsification (interpolation/cell_center_nli_intrp.hpp:
//                 310-420, 557-674). One CTA per receiving block; the sending
//                 blocks of a group are applied in child order, so sums are
//                 deterministic without atomics. tp_antrp_kernel: anterpolation
//                 to few blocks, a cluster of eight CTAs each; tp_band2_kernel:
//                 coarsification by width-2 bands, a thread per node
//   halo_kernel   same-level buffer exchange (domain/mpi/haloCommunicator.hpp:
//                 63-107): each buffer cell takes the value of the neighbour
//                 interior cell that overlaps it
//   correction    add_source_correction (cell_center_nli_intrp.hpp:171-238)
//   zero / copy_interior / axpy over block lists (fmm.hpp:1029-1106,
//                 poisson.hpp:921-1013); solve_begin, sweep_begin: those that
//                 start a solve and a sweep, in one launch each
#include <cooperative_groups.h>

#include <algorithm>
#include <cstring>

#include "ctx.hpp"

namespace cg = cooperative_groups;

namespace iblgf_b200
{
namespace
{
// The Nb x Nb matrices of a transfer per set and child bit, passed by
// value: they sit in the constant bank, and with the dense passes fully
// unrolled every matrix entry is an FMA operand at a fixed offset (no
// shared-memory loads). Face and edge components use one of two sets per axis
// (their relative positions 0 and 1); set[c][a] is that of component c and
// axis a.
// lo: for the banded passes (W > 0), first column of row m's band of width W
// in summation order (the row's nonzeros all lie in [lo, lo + W)); w5: the
// entries of the bands of width 5
template<int NB, class T>
struct TpMats
{
    T m[2][2][NB * NB];
    T w5[2][2][NB][5];
    unsigned char lo[2][2][NB];
    unsigned char set[3][3];
};

// Pencils in shared memory: NB values at an odd row stride, so that the lanes
// of a warp, each in its own pencil, read without bank conflicts.
template<int NB>
constexpr int tp_stride()
{
    return NB | 1;
}
// bytes of one block there
template<int NB, class T>
constexpr size_t tp_bytes()
{
    return (size_t)NB * NB * tp_stride<NB>() * sizeof(T);
}
// place of entry m of the pass's output for pencil p = (z, y): with the axes
// rotated ([z][y][x] -> [x][z][y]) it is entry y of pencil (m, z)
template<int NB>
__device__ __forceinline__ int tp_out(int m, int p)
{
    return (m * NB + p / NB) * tp_stride<NB>() + p % NB;
}

// the component fields of one transfer (blockIdx.y = component)
struct TpFields
{
    const double* src[3];
    double* dst[3];
};

template<int NB>
constexpr int tp_threads()
{
    return (NB * NB + 31) / 32 * 32;
}

// One pass along the fastest axis of `in`: thread p owns pencil p and forms
// sum_n T(m,n) in[p][n] with T(m,n) = M_K(m,n) (anterpolation) or M_K(n,m)
// (interpolation). Writing the result with the axes rotated makes the next
// axis the fastest one, so all three passes read contiguous pencils; after
// three passes the layout is back to [z][y][x]. The last pass adds into the
// thread's accumulators instead of writing shared memory.
// W > 0: only the W entries of row m's band [lo, lo + W) are summed, in
// the same order; the skipped entries are zeros, whose FMAs leave the running
// sum unchanged, so the result equals the full row's. At W = 5 the bands move
// on by at most one column per row, so a window of five values in registers
// takes one shared-memory load per move instead of five per row (the
// cell-centred interpolation of three levels at extent 16: 760 -> 497 us).
// T: arithmetic and shared-memory type of the passes (the accumulators acc,
// which start from and end in the FP64 target block, stay FP64)
template<int NB, int K, bool TR, bool LAST, int W, class T, bool MULTI>
__device__ __forceinline__ void tp_pass(const T* __restrict__ in, T* __restrict__ out,
                                        const TpMats<NB, T>& mt, int set, int p, double* acc)
{
    if constexpr (W == 0)
    {
        T v[NB];
#pragma unroll
        for (int n = 0; n < NB; ++n) v[n] = in[p * tp_stride<NB>() + n];
#pragma unroll
        for (int m = 0; m < NB; ++m)
        {
            T s = 0;
#pragma unroll
            for (int n = 0; n < NB; ++n)
            {
                // one set: entries at fixed places of the constant bank
                const T* mat = mt.m[MULTI ? set : 0][K];
                s = fma(TR ? mat[n * NB + m] : mat[m * NB + n], v[n], s);
            }
            if (LAST) acc[m] += s;
            else out[tp_out<NB>(m, p)] = s;
        }
    }
    else if constexpr (W == 5)
    {
        const T* row = in + p * tp_stride<NB>();
        int cur = mt.lo[set][K][0];
        T v[5];
#pragma unroll
        for (int j = 0; j < 5; ++j) v[j] = row[cur + j];
#pragma unroll
        for (int m = 0; m < NB; ++m)
        {
            if (m && mt.lo[set][K][m] != cur)
            {
                ++cur;
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] = v[j + 1];
                v[4] = row[cur + 4];
            }
            T s = 0;
#pragma unroll
            for (int j = 0; j < 5; ++j) s = fma(mt.w5[set][K][m][j], v[j], s);
            if (LAST) acc[m] += s;
            else out[tp_out<NB>(m, p)] = s;
        }
    }
    else
    {
        const T* row = in + p * tp_stride<NB>();
        const T* mat = mt.m[set][K];
#pragma unroll
        for (int m = 0; m < NB; ++m)
        {
            const int lo = mt.lo[set][K][m];
            T s = 0;
#pragma unroll
            for (int j = 0; j < W; ++j)
            {
                const int n = lo + j;
                s = fma(TR ? mat[n * NB + m] : mat[m * NB + n], row[n], s);
            }
            if (LAST) acc[m] += s;
            else out[tp_out<NB>(m, p)] = s;
        }
    }
}

// a block into shared-memory pencils
template<int NB, class T>
__device__ __forceinline__ void tp_stage(const double* __restrict__ block, T* __restrict__ a)
{
    const double2* s2 = reinterpret_cast<const double2*>(block);
    for (int i = threadIdx.x; i < NB * NB * NB / 2; i += blockDim.x)
    {
        const double2 v = s2[i];
        const int at = 2 * i / NB * tp_stride<NB>() + 2 * i % NB;  // NB is even: both in one pencil
        a[at] = (T)v.x;
        a[at + 1] = (T)v.y;
    }
}

template<int NB, bool TR, bool LAST, int W, class T, bool MULTI = false>
__device__ __forceinline__ void tp_pass_bit(int bit, const T* in, T* out, const TpMats<NB, T>& mt, int set, int p,
                                            double* acc)
{
    if (bit) tp_pass<NB, 1, TR, LAST, W, T, MULTI>(in, out, mt, set, p, acc);
    else tp_pass<NB, 0, TR, LAST, W, T, MULTI>(in, out, mt, set, p, acc);
}

// mode 0: dst[group] += sum_tasks A(src)        (anterpolation / coarsify)
// mode 1: dst[group] += I(src)                  (FMM interpolation)
// mode 2: dst[group]  = I(src)                  (cell-centred interpolation)
// One CTA per receiving block, one thread per pencil; the sending blocks of
// a group are applied in child order into per-thread accumulators.
template<int NB, bool TR, int W, class T, bool MULTI = false>
__global__ void __launch_bounds__(tp_threads<NB>(), 2) tp_kernel(
    const int* __restrict__ gptr, const int* __restrict__ gdst, const int* __restrict__ tsrc,
    const int* __restrict__ tcid, const __grid_constant__ TpFields f, const __grid_constant__ TpMats<NB, T> mt, int mode)
{
    constexpr int N3 = NB * NB * NB;
    const double* src = f.src[blockIdx.y];
    double* dst = f.dst[blockIdx.y];
    const unsigned char* set = mt.set[blockIdx.y];
    extern __shared__ __align__(16) unsigned char tp_smem[];
    T* a = reinterpret_cast<T*>(tp_smem);
    T* b = a + NB * NB * tp_stride<NB>();
    const int g = blockIdx.x;
    const int p = threadIdx.x;
    const bool active = p < NB * NB;
    // accumulate onto the receiving block in task order (dst += r_0, += r_1, ...)
    double* d = dst + (size_t)gdst[g] * N3 + p;
    double acc[NB];
#pragma unroll
    for (int m = 0; m < NB; ++m) acc[m] = (active && mode != 2) ? d[m * NB * NB] : 0.0;
    for (int t = gptr[g]; t < gptr[g + 1]; ++t)
    {
        const int cid = tcid[t];
        tp_stage<NB, T>(src + (size_t)tsrc[t] * N3, a);
        __syncthreads();
        if (active) tp_pass_bit<NB, TR, false, W, T, MULTI>(cid & 1, a, b, mt, set[0], p, acc);
        __syncthreads();
        if (active) tp_pass_bit<NB, TR, false, W, T, MULTI>((cid >> 1) & 1, b, a, mt, set[1], p, acc);
        __syncthreads();
        if (active) tp_pass_bit<NB, TR, true, W, T, MULTI>((cid >> 2) & 1, a, (T*)nullptr, mt, set[2], p, acc);
        __syncthreads();
    }
    if (!active) return;
#pragma unroll
    for (int m = 0; m < NB; ++m) d[m * NB * NB] = acc[m];
}

// Dense anterpolation (mode 0): dst[group] += sum_tasks A(src). A cluster of
// eight CTAs per receiving block, one per sending child: each runs its three
// passes into its own shared memory, then takes an eighth of the receiving
// block and adds the children's results, read through distributed shared
// memory, in child order (the order and the roundings of one CTA that walks
// the children). For the coarse levels with few receiving blocks, where eight
// children in sequence are 24 barrier-separated passes on a few SMs: 22 against
// 45 us at 44 blocks of 18^3 in FP32, 16 against 28 at 8; with more blocks than
// kAntrpClusters the chip is full either way and the barriers of the cluster
// cost more (106 blocks: 44 / 46 us, 184: 73 / 67, 1161: 382 / 202; in FP64, 98 KB
// per CTA, 64 blocks 31 / 67, 216: 96 / 86). The line is that of 18^3 blocks; the
// clusters of smaller ones still win at 216 (extent 10, FP64 20 / 30 us, extent 4
// 8.5 / 11 us).
constexpr int kAntrpClusters = 120;

template<int NB, class T>
__global__ void __cluster_dims__(8, 1, 1) __launch_bounds__(tp_threads<NB>(), 2) tp_antrp_kernel(
    const int* __restrict__ gptr, const int* __restrict__ gdst, const int* __restrict__ tsrc,
    const int* __restrict__ tcid, const __grid_constant__ TpFields f, const __grid_constant__ TpMats<NB, T> mt)
{
    constexpr int N3 = NB * NB * NB;
    extern __shared__ __align__(16) unsigned char tp_smem[];
    T* a = reinterpret_cast<T*>(tp_smem);
    T* b = a + NB * NB * tp_stride<NB>();
    cg::cluster_group cluster = cg::this_cluster();
    const int g = blockIdx.x / 8, r = (int)cluster.block_rank();
    const int t0 = gptr[g], n = gptr[g + 1] - t0;
    const int p = threadIdx.x;
    const bool active = p < NB * NB;
    if (r < n)
    {
        const int cid = tcid[t0 + r];
        tp_stage<NB, T>(f.src[blockIdx.y] + (size_t)tsrc[t0 + r] * N3, a);
        __syncthreads();
        if (active) tp_pass_bit<NB, false, false, 0, T>(cid & 1, a, b, mt, 0, p, nullptr);
        __syncthreads();
        if (active) tp_pass_bit<NB, false, false, 0, T>((cid >> 1) & 1, b, a, mt, 0, p, nullptr);
        __syncthreads();
        if (active) tp_pass_bit<NB, false, false, 0, T>((cid >> 2) & 1, a, b, mt, 0, p, nullptr);
    }
    cluster.sync();
    double* d = f.dst[blockIdx.y] + (size_t)gdst[g] * N3;
    const T* part[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) part[k] = cluster.map_shared_rank(b, k);
    for (int i = N3 / 8 * r + threadIdx.x; i < N3 / 8 * (r + 1); i += blockDim.x)
    {
        double acc = d[i];
        const int at = i / NB * tp_stride<NB>() + i % NB;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (k < n) acc += (double)part[k][at];
        d[i] = acc;
    }
    cluster.sync();  // the others have read this CTA's result
}

// Width-2 band (mode 0, coarsening): each receiving node takes 2 x 2 x 2 nodes
// of the one sending block that covers it (per axis, the child bit whose row of
// this node is not zero; buffer nodes receive nothing). One thread per
// receiving node, so the 8 loads of a node and those of a thread's kBandNodes
// nodes are in flight together; the sums run in the order of the separable
// passes (x band, then y, then z, entries in summation order).
// Measured at Nb = 18 on the vortex ring's coarsening (40 to 248 receiving
// blocks): 55 us per component with one thread per receiving z pencil, whose
// sending blocks and planes followed one another.
constexpr int kBandNodes = 4;

template<int NB, class T>
__global__ void __launch_bounds__(256) tp_band2_kernel(const int* __restrict__ gptr, const int* __restrict__ gdst,
                                                       const int* __restrict__ tsrc, const int* __restrict__ tcid,
                                                       const __grid_constant__ TpFields f, const __grid_constant__ TpMats<NB, T> mt)
{
    constexpr int N3 = NB * NB * NB, E = NB - 2, E3 = E * E * E;
    __shared__ int child[8];           // sending block per child id, -1: none
    __shared__ unsigned char bit[3][NB], lo[3][NB];
    __shared__ T w0[3][NB], w1[3][NB];
    const double* __restrict__ src = f.src[blockIdx.y];
    const int g = blockIdx.x;
    if (threadIdx.x < 8) child[threadIdx.x] = -1;
    for (int i = threadIdx.x; i < 3 * NB; i += blockDim.x)
    {
        // the child bit whose row of node m is not zero, and its band
        const int a = i / NB, m = i % NB, s = mt.set[blockIdx.y][a];
        int k = 0, l = mt.lo[s][0][m];
        T u = mt.m[s][0][m * NB + l], v = mt.m[s][0][m * NB + l + 1];
        if (u == (T)0 && v == (T)0)
        {
            k = 1;
            l = mt.lo[s][1][m];
            u = mt.m[s][1][m * NB + l];
            v = mt.m[s][1][m * NB + l + 1];
        }
        bit[a][m] = (unsigned char)k;
        lo[a][m] = (unsigned char)l;
        w0[a][m] = u;
        w1[a][m] = v;
    }
    __syncthreads();
    for (int t = gptr[g] + threadIdx.x; t < gptr[g + 1]; t += blockDim.x) child[tcid[t]] = tsrc[t];
    __syncthreads();
    double* __restrict__ d = f.dst[blockIdx.y] + (size_t)gdst[g] * N3;
    const int i0 = blockIdx.z * (256 * kBandNodes) + threadIdx.x;
    double v[kBandNodes][8], old[kBandNodes];
    int at[kBandNodes];
#pragma unroll
    for (int k = 0; k < kBandNodes; ++k)
    {
        const int i = i0 + 256 * k;
        at[k] = -1;
        if (i >= E3) continue;
        const int x = 1 + i % E, y = 1 + (i / E) % E, z = 1 + i / (E * E);
        const int b = child[bit[0][x] + 2 * bit[1][y] + 4 * bit[2][z]];
        if (b < 0) continue;
        at[k] = (z * NB + y) * NB + x;
        const double* p = src + (size_t)b * N3 + (lo[2][z] * NB + lo[1][y]) * NB + lo[0][x];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[k][j] = p[(j >> 2) * NB * NB + ((j >> 1) & 1) * NB + (j & 1)];
        old[k] = d[at[k]];
    }
#pragma unroll
    for (int k = 0; k < kBandNodes; ++k)
    {
        if (at[k] < 0) continue;
        const int x = at[k] % NB, y = (at[k] / NB) % NB, z = at[k] / (NB * NB);
        const T x0 = w0[0][x], x1 = w1[0][x], y0 = w0[1][y], y1 = w1[1][y];
        T c[2];
#pragma unroll
        for (int j = 0; j < 2; ++j)
        {
            const T b0 = fma(x1, (T)v[k][4 * j + 1], fma(x0, (T)v[k][4 * j], (T)0));
            const T b1 = fma(x1, (T)v[k][4 * j + 3], fma(x0, (T)v[k][4 * j + 2], (T)0));
            c[j] = fma(y1, b1, fma(y0, b0, (T)0));
        }
        d[at[k]] = old[k] + fma(w1[2][z], c[1], fma(w0[2][z], c[0], (T)0));
    }
}

// threads walk the buffer shell only: the two z = 0, NB-1 planes, then per
// inner z plane its ring (rows y = 0, NB-1, columns x = 0, NB-1). The 27
// neighbours and their offsets are read once into shared memory, so that a
// node's copy is one load, all of a thread's nodes in flight.
template<int NB>
__global__ void __launch_bounds__(256) halo_kernel(const __grid_constant__ TpFields fs, const int* __restrict__ list,
                                                   const int* __restrict__ nbr, const int* __restrict__ bbase, int e)
{
    constexpr int N3 = NB * NB * NB;
    constexpr int P2 = NB * NB, RING = 4 * NB - 4, SHELL = 2 * P2 + (NB - 2) * RING;
    constexpr int K = (SHELL + 255) / 256;
    __shared__ int s_q[27], s_off[27][3];
    const int o = list[blockIdx.x];
    double* f = fs.dst[blockIdx.y];
    double* blk = f + (size_t)o * N3;
    if (threadIdx.x < 27)
    {
        const int q = nbr[27 * o + threadIdx.x];
        s_q[threadIdx.x] = q;
        for (int a = 0; a < 3; ++a) s_off[threadIdx.x][a] = q < 0 ? 0 : bbase[3 * o + a] - 1 - bbase[3 * q + a];
    }
    __syncthreads();
    double v[K];
    int at[K];
#pragma unroll
    for (int k = 0; k < K; ++k)
    {
        const int t = 256 * k + threadIdx.x;
        at[k] = -1;
        if (t >= SHELL) continue;
        int x, y, z;
        if (t < 2 * P2)
        {
            z = t < P2 ? 0 : NB - 1;
            x = (t % P2) % NB;
            y = (t % P2) / NB;
        }
        else
        {
            const int u = t - 2 * P2, r = u % RING;
            z = 1 + u / RING;
            if (r < 2 * NB)
            {
                y = r < NB ? 0 : NB - 1;
                x = r % NB;
            }
            else
            {
                const int w = r - 2 * NB;
                x = (w & 1) ? NB - 1 : 0;
                y = 1 + w / 2;
            }
        }
        const int dx = x == 0 ? 0 : (x == NB - 1 ? 2 : 1);
        const int dy = y == 0 ? 0 : (y == NB - 1 ? 2 : 1);
        const int dz = z == 0 ? 0 : (z == NB - 1 ? 2 : 1);
        const int d = dx + 3 * dy + 9 * dz, q = s_q[d];
        if (q < 0) continue;
        // global cell of this buffer node and its position in q's interior
        const int lx = s_off[d][0] + x, ly = s_off[d][1] + y, lz = s_off[d][2] + z;
        if (lx < 0 || ly < 0 || lz < 0 || lx >= e || ly >= e || lz >= e) continue;
        at[k] = x + NB * (y + NB * z);
        v[k] = f[(size_t)q * N3 + (lx + 1) + NB * ((ly + 1) + NB * (lz + 1))];
    }
#pragma unroll
    for (int k = 0; k < K; ++k)
        if (at[k] >= 0) blk[at[k]] = v[k];
}

// Block copies and sums are split over blockIdx.y in pieces of kPiece 16-byte
// pairs, kPairs per thread with all loads in flight before the first store: a
// block per CTA with one load after another took 15 us for 64 blocks of 18^3
// (uniform 64^3 solve), 3 us as a piece per CTA.
constexpr int kPairs = 4;
constexpr int kPiece = 256 * kPairs;
constexpr int pieces(int n3) { return (n3 / 2 + kPiece - 1) / kPiece; }

// add_source_correction on the listed (child) blocks: ct = c0 - laplace(tt) r
// on the interior, c0 = ct where the block is a correction block (flag bit 1:
// interpolated from its parent), 0 elsewhere; then st += ct
template<int NB>
__global__ void __launch_bounds__(256) correction_kernel(const double* __restrict__ tt, double* __restrict__ corr,
                                                         double* __restrict__ st, const int* __restrict__ list,
                                                         const int* __restrict__ flags, double r)
{
    constexpr int N3 = NB * NB * NB;
    const int o = list[blockIdx.x];
    const bool have = flags[o] & 2;
    const double* __restrict__ t = tt + (size_t)o * N3;
    double* __restrict__ c = corr + (size_t)o * N3;
    double* __restrict__ s = st + (size_t)o * N3;
#pragma unroll
    for (int k = 0; k < 2 * kPairs; ++k)
    {
        const int i = blockIdx.y * (2 * kPiece) + 256 * k + threadIdx.x;
        if (i >= N3) break;
        const int x = i % NB, y = (i / NB) % NB, z = i / (NB * NB);
        const bool in = x > 0 && y > 0 && z > 0 && x < NB - 1 && y < NB - 1 && z < NB - 1;
        double v = have ? c[i] : 0.0;
        if (in)
        {
            v += 6.0 * t[i] * r;
            v -= t[i - NB * NB] * r;
            v -= t[i + NB * NB] * r;
            v -= t[i - NB] * r;
            v -= t[i + NB] * r;
            v -= t[i + 1] * r;
            v -= t[i - 1] * r;
        }
        c[i] = v;
        if (in || have) s[i] += v;
    }
}

// f.dst[component] = 0 on the listed blocks
__global__ void __launch_bounds__(256) zero_kernel(const __grid_constant__ TpFields f, const int* __restrict__ list,
                                                   int half)
{
    double2* b = reinterpret_cast<double2*>(f.dst[blockIdx.z]) + (size_t)list[blockIdx.x] * half;
#pragma unroll
    for (int k = 0; k < kPairs; ++k)
    {
        const int i = blockIdx.y * kPiece + 256 * k + threadIdx.x;
        if (i < half) b[i] = make_double2(0.0, 0.0);
    }
}

// 1 if node i of a block is in its interior
template<int NB>
__device__ __forceinline__ bool interior(int i)
{
    const int x = i % NB, y = (i / NB) % NB, z = i / (NB * NB);
    return x > 0 && y > 0 && z > 0 && x < NB - 1 && y < NB - 1 && z < NB - 1;
}

// the interiors of the listed blocks of component blockIdx.z
template<int NB>
__global__ void __launch_bounds__(256) copy_interior_kernel(const __grid_constant__ TpFields f,
                                                            const int* __restrict__ list)
{
    constexpr int N3 = NB * NB * NB;
    const size_t off = (size_t)list[blockIdx.x] * N3;
    const double* __restrict__ s = f.src[blockIdx.z] + off;
    double* __restrict__ d = f.dst[blockIdx.z] + off;
    double v[2 * kPairs];
#pragma unroll
    for (int k = 0; k < 2 * kPairs; ++k)
    {
        const int i = blockIdx.y * (2 * kPiece) + 256 * k + threadIdx.x;
        v[k] = i < N3 ? s[i] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < 2 * kPairs; ++k)
    {
        const int i = blockIdx.y * (2 * kPiece) + 256 * k + threadIdx.x;
        if (i < N3 && interior<NB>(i)) d[i] = v[k];
    }
}

// start of a sweep: entry = block << 2 | op; op 0: fs = 0, 1: fs = interior of
// src and 0 around it, 2: ft = 0
template<int NB>
__global__ void __launch_bounds__(256) sweep_begin_kernel(const int* __restrict__ entries,
                                                          const double* __restrict__ src, double* __restrict__ fs,
                                                          double* __restrict__ ft)
{
    constexpr int N3 = NB * NB * NB;
    const int e = entries[blockIdx.x], op = e & 3;
    const size_t off = (size_t)(e >> 2) * (N3 / 2);
    double2* __restrict__ d = reinterpret_cast<double2*>(op == 2 ? ft : fs) + off;
    double2 v[kPairs];
#pragma unroll
    for (int k = 0; k < kPairs; ++k)
    {
        const int i = blockIdx.y * kPiece + 256 * k + threadIdx.x;
        v[k] = make_double2(0.0, 0.0);
        if (op == 1 && i < N3 / 2)
        {
            v[k] = reinterpret_cast<const double2*>(src)[off + i];
            if (!interior<NB>(2 * i)) v[k].x = 0.0;
            if (!interior<NB>(2 * i + 1)) v[k].y = 0.0;
        }
    }
#pragma unroll
    for (int k = 0; k < kPairs; ++k)
    {
        const int i = blockIdx.y * kPiece + 256 * k + threadIdx.x;
        if (i < N3 / 2) d[i] = v[k];
    }
}

// d = a s (assign) or d += a s on the listed blocks; leaf blocks' results also
// to leaf_out (if given)
__global__ void __launch_bounds__(256) axpy_kernel(const double2* __restrict__ s, double2* __restrict__ d,
                                                   const int* __restrict__ list, int half, double a, int assign,
                                                   const int* __restrict__ flags, double2* __restrict__ leaf_out)
{
    const size_t off = (size_t)list[blockIdx.x] * half;
    const bool leaf = leaf_out && (flags[list[blockIdx.x]] & 1);
    double2 v[kPairs], w[kPairs];
#pragma unroll
    for (int k = 0; k < kPairs; ++k)
    {
        const int i = blockIdx.y * kPiece + 256 * k + threadIdx.x;
        if (i < half) v[k] = s[off + i];
        if (i < half && !assign) w[k] = d[off + i];
    }
#pragma unroll
    for (int k = 0; k < kPairs; ++k)
    {
        const int i = blockIdx.y * kPiece + 256 * k + threadIdx.x;
        if (i >= half) break;
        const double2 r = assign ? make_double2(a * v[k].x, a * v[k].y)
                                 : make_double2(w[k].x + v[k].x * a, w[k].y + v[k].y * a);
        d[off + i] = r;
        if (leaf) leaf_out[off + i] = r;
    }
}

// start of a solve, one block per blockIdx.x: st = src on leaves (flag bit 0), 0
// elsewhere, and tt = ct = 0 where zero is set or the block's bit 2 is
__global__ void __launch_bounds__(256) solve_begin_kernel(const __grid_constant__ TpFields f,
                                                          const int* __restrict__ flags, int half, int zero)
{
    const int fl = flags[blockIdx.x];
    const size_t off = (size_t)blockIdx.x * half;
    const double2* __restrict__ src = reinterpret_cast<const double2*>(f.src[0]) + off;
    double2* __restrict__ st = reinterpret_cast<double2*>(f.dst[0]) + off;
    double2* __restrict__ tt = reinterpret_cast<double2*>(f.dst[1]) + off;
    double2* __restrict__ ct = reinterpret_cast<double2*>(f.dst[2]) + off;
    double2 v[kPairs];
#pragma unroll
    for (int k = 0; k < kPairs; ++k)
    {
        const int i = blockIdx.y * kPiece + 256 * k + threadIdx.x;
        v[k] = (fl & 1) && i < half ? src[i] : make_double2(0.0, 0.0);
    }
    const bool z = zero || (fl & 4);
#pragma unroll
    for (int k = 0; k < kPairs; ++k)
    {
        const int i = blockIdx.y * kPiece + 256 * k + threadIdx.x;
        if (i >= half) break;
        st[i] = v[k];
        if (z) tt[i] = ct[i] = make_double2(0.0, 0.0);
    }
}

template<class F>
void nb_dispatch(int Nb, F&& f)
{
    switch (Nb)
    {
        case 6: f(std::integral_constant<int, 6>{}); return;
        case 8: f(std::integral_constant<int, 8>{}); return;
        case 10: f(std::integral_constant<int, 10>{}); return;
        case 12: f(std::integral_constant<int, 12>{}); return;
        case 16: f(std::integral_constant<int, 16>{}); return;
        case 18: f(std::integral_constant<int, 18>{}); return;
        default: throw Error(IBLGF_EINVAL, "unsupported block size");
    }
}
}  // namespace

void launch_tp(Ctx& c, const TpTasks& t, const double* src, double* dst, int mat_base, int mode, bool fp32)
{
    const int bases[1][3] = {{mat_base, mat_base, mat_base}};
    launch_tp_vf(c, t, &src, &dst, 1, bases, mode, fp32);
}

namespace
{
template<int NB, class T>
void launch_tp_typed(Ctx& c, const TpTasks& t, const TpFields& f, int n, const int (*mat_base)[3], int mode)
{
    static_assert((NB * NB * NB) % 2 == 0, "blocks are copied as double2");
    TpMats<NB, T> mt{};
    const bool tr = mode != 0;
    int width = 0;  // widest band of any row, in summation order
    int base[2] = {-1, -1};
    for (int q = 0; q < n; ++q)
        for (int a = 0; a < 3; ++a)
        {
            int s = 0;
            while (s < 2 && base[s] >= 0 && base[s] != mat_base[q][a]) ++s;
            if (s == 2) throw Error(IBLGF_EINTERNAL, "a transfer takes two matrix sets at most");
            mt.set[q][a] = (unsigned char)s;
            if (base[s] >= 0) continue;
            base[s] = mat_base[q][a];
            const size_t off = (size_t)base[s] * NB * NB;
            if (c.h_mats.size() < off + 2 * NB * NB) throw Error(IBLGF_EINTERNAL, "transfer matrices missing");
            for (int k = 0; k < 2; ++k)
                for (int i = 0; i < NB * NB; ++i) mt.m[s][k][i] = (T)c.h_mats[off + (size_t)k * NB * NB + i];
            for (int k = 0; k < 2; ++k)
                for (int m = 0; m < NB; ++m)
                {
                    int lo = NB, hi = 0;
                    for (int i = 0; i < NB; ++i)
                        if ((tr ? mt.m[s][k][i * NB + m] : mt.m[s][k][m * NB + i]) != (T)0)
                        {
                            lo = std::min(lo, i);
                            hi = i + 1;
                        }
                    mt.lo[s][k][m] = (unsigned char)(lo < hi ? lo : 0);
                    width = std::max(width, lo < hi ? hi - lo : 0);
                }
        }
    int W = width <= 2 ? 2 : (width <= 5 ? 5 : 0);
    if (W == 2 && mode == 0)
        // tp_band2_kernel takes one sending child per receiving node and axis and
        // nothing on the buffer nodes; matrices that give more go another way
        for (int s = 0; s < 2 && base[s] >= 0; ++s)
            for (int m = 0; m < NB; ++m)
            {
                int children = 0;
                for (int k = 0; k < 2; ++k)
                    children += std::any_of(mt.m[s][k] + m * NB, mt.m[s][k] + (m + 1) * NB, [](T v) { return v != (T)0; });
                if (children > (m > 0 && m < NB - 1 ? 1 : 0)) W = 5;
            }
    if (W == 5)
    {
        // the smallest starts that never move back and cover the rows; they move
        // on by one column at most (checked, else the dense form)
        unsigned char start[2][2][NB] = {};
        for (int s = 0; s < 2 && base[s] >= 0; ++s)
            for (int k = 0; k < 2; ++k)
                for (int m = 0, st = 0; m < NB; ++m)
                {
                    int lo = NB, hi = 0;
                    for (int i = 0; i < NB; ++i)
                        if ((tr ? mt.m[s][k][i * NB + m] : mt.m[s][k][m * NB + i]) != (T)0)
                        {
                            lo = std::min(lo, i);
                            hi = i + 1;
                        }
                    const int prev = st;
                    st = std::max(st, hi - 5);
                    if (st > lo || (m && st > prev + 1)) W = 0;
                    start[s][k][m] = (unsigned char)st;
                    for (int j = 0; j < 5; ++j)
                        mt.w5[s][k][m][j] = tr ? mt.m[s][k][(st + j) * NB + m] : mt.m[s][k][m * NB + st + j];
                }
        if (W == 5) std::memcpy(mt.lo, start, sizeof(mt.lo));
    }
    if (W == 2)
        for (int s = 0; s < 2; ++s)
            for (int k = 0; k < 2; ++k)
                for (int m = 0; m < NB; ++m) mt.lo[s][k][m] = (unsigned char)std::min<int>(mt.lo[s][k][m], NB - W);
    const size_t smem = 2 * tp_bytes<NB, T>();
    auto launch = [&](auto kfn) {
        IBLGF_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kfn<<<dim3(t.n_groups, n), tp_threads<NB>(), smem, c.stream>>>(t.group_ptr.p, t.group_dst.p, t.task_src.p,
                                                                       t.task_cid.p, f, mt, mode);
    };
    if (mode == 0)
    {
        if (W == 2)
        {
            constexpr int per = 256 * kBandNodes, e3 = (NB - 2) * (NB - 2) * (NB - 2);
            auto kfn = tp_band2_kernel<NB, T>;
            kfn<<<dim3(t.n_groups, n, (e3 + per - 1) / per), 256, 0, c.stream>>>(
                t.group_ptr.p, t.group_dst.p, t.task_src.p, t.task_cid.p, f, mt);
        }
        else if (W == 5) launch(tp_kernel<NB, false, 5, T>);
        else if (base[1] >= 0) throw Error(IBLGF_EINTERNAL, "anterpolation has one matrix set");
        else if (t.n_groups * n > kAntrpClusters) launch(tp_kernel<NB, false, 0, T>);
        else
        {
            static_assert((NB * NB * NB) % 8 == 0, "eight CTAs share a receiving block");
            auto kfn = tp_antrp_kernel<NB, T>;
            IBLGF_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            kfn<<<dim3(8 * t.n_groups, n), tp_threads<NB>(), smem, c.stream>>>(
                t.group_ptr.p, t.group_dst.p, t.task_src.p, t.task_cid.p, f, mt);
        }
    }
    else
    {
        if (W == 2) launch(tp_kernel<NB, true, 2, T>);
        else if (W == 5) launch(tp_kernel<NB, true, 5, T>);
        else if (base[1] >= 0) launch(tp_kernel<NB, true, 0, T, true>);  // interpolation orders above 5
        else launch(tp_kernel<NB, true, 0, T>);
    }
}
}  // namespace

// fp32: the passes in FP32 (matrices rounded to FP32), the sums into the
// FP64 receiving blocks in FP64
void launch_tp_vf(Ctx& c, const TpTasks& t, const double* const* src, double* const* dst, int n,
                  const int (*mat_base)[3], int mode, bool fp32)
{
    if (!t.n_groups || n < 1) return;
    TpFields f{};
    for (int k = 0; k < n; ++k)
    {
        f.src[k] = src[k];
        f.dst[k] = dst[k];
    }
    nb_dispatch(c.Nb, [&](auto nbc) {
        constexpr int NB = decltype(nbc)::value;
        if (fp32) launch_tp_typed<NB, float>(c, t, f, n, mat_base, mode);
        else launch_tp_typed<NB, double>(c, t, f, n, mat_base, mode);
    });
    c.launches += 1;
    IBLGF_CUDA(cudaGetLastError());
}

void launch_tp_axes(Ctx& c, const TpTasks& t, const double* src, double* dst, const int* mat_base, int mode, bool fp32)
{
    const int bases[1][3] = {{mat_base[0], mat_base[1], mat_base[2]}};
    launch_tp_vf(c, t, &src, &dst, 1, bases, mode, fp32);
}

void launch_halo_vf(Ctx& c, double* const* f, int m, const int* list, int n)
{
    if (!n || m < 1) return;
    TpFields p{};
    for (int k = 0; k < m; ++k) p.dst[k] = f[k];
    nb_dispatch(c.Nb, [&](auto nbc) {
        constexpr int NB = decltype(nbc)::value;
        halo_kernel<NB><<<dim3(n, m), 256, 0, c.stream>>>(p, list, c.d_nbr.p, c.d_bbase.p, c.cfg.block_extent);
    });
    c.launches += 1;
    IBLGF_CUDA(cudaGetLastError());
}

void launch_halo(Ctx& c, double* f, const int* list, int n) { launch_halo_vf(c, &f, 1, list, n); }

void launch_source_correction(Ctx& c, const double* target_tmp, double* corr, double* source_tmp, const int* list,
                              int n, double inv_dx2)
{
    if (!n) return;
    nb_dispatch(c.Nb, [&](auto nbc) {
        constexpr int NB = decltype(nbc)::value;
        correction_kernel<NB><<<dim3(n, pieces(NB * NB * NB)), 256, 0, c.stream>>>(target_tmp, corr, source_tmp, list,
                                                                                  c.d_flags.p, inv_dx2);
    });
    c.launches += 1;
    IBLGF_CUDA(cudaGetLastError());
}

void launch_sweep_begin(Ctx& c, const int* entries, int n, const double* src, double* fs, double* ft)
{
    if (!n) return;
    nb_dispatch(c.Nb, [&](auto nbc) {
        constexpr int NB = decltype(nbc)::value;
        sweep_begin_kernel<NB><<<dim3(n, pieces(NB * NB * NB)), 256, 0, c.stream>>>(entries, src, fs, ft);
    });
    c.launches += 1;
    IBLGF_CUDA(cudaGetLastError());
}

void launch_solve_begin(Ctx& c, const double* src, double* st, double* tt, double* ct, bool zero)
{
    if (!c.n_oct) return;
    TpFields f{};
    f.src[0] = src;
    f.dst[0] = st;
    f.dst[1] = tt;
    f.dst[2] = ct;
    const int half = (int)(c.block_elems() / 2);  // Nb is even
    solve_begin_kernel<<<dim3(c.n_oct, pieces(2 * half)), 256, 0, c.stream>>>(f, c.d_flags.p, half, zero ? 1 : 0);
    c.launches += 1;
    IBLGF_CUDA(cudaGetLastError());
}

namespace
{
// n doubles from p set to zero (16-byte stores where p is aligned)
__global__ void fill_zero_kernel(double* __restrict__ p, size_t n)
{
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if ((reinterpret_cast<uintptr_t>(p) & 15) == 0)
    {
        double2* q = reinterpret_cast<double2*>(p);
        const double2 z = make_double2(0.0, 0.0);
        for (size_t j = i; j < n / 2; j += stride) q[j] = z;
        if (i == 0 && (n & 1)) p[n - 1] = 0.0;
    }
    else
        for (size_t j = i; j < n; j += stride) p[j] = 0.0;
}
// smallest index of a non-finite value (NaN or +-inf); *first starts at ~0
__global__ void nonfinite_kernel(const double* __restrict__ p, size_t n, unsigned long long* first)
{
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += stride)
        if (!isfinite(p[j]))
        {
            atomicMin(first, (unsigned long long)j);
            return;  // later indices of this thread are larger
        }
}
}  // namespace

long long first_nonfinite(Ctx& c, const double* p, size_t n)
{
    DevBuf<unsigned long long> d;
    d.alloc(1);
    IBLGF_CUDA(cudaMemsetAsync(d.p, 0xFF, sizeof(unsigned long long), c.stream));
    if (n)
    {
        const size_t blocks = std::min<size_t>((n + 255) / 256, 148 * 8);
        nonfinite_kernel<<<(unsigned)blocks, 256, 0, c.stream>>>(p, n, d.p);
        c.launches += 1;
        IBLGF_CUDA(cudaGetLastError());
    }
    unsigned long long h = 0;
    IBLGF_CUDA(cudaMemcpyAsync(&h, d.p, sizeof(h), cudaMemcpyDeviceToHost, c.stream));
    IBLGF_CUDA(cudaStreamSynchronize(c.stream));
    return h == ~0ull ? -1 : (long long)h;
}

// a plain kernel (not cudaMemsetAsync), so that the zeroing can sit in the
// body of a conditional graph node
void launch_fill_zero(Ctx& c, double* p, size_t n)
{
    if (!n) return;
    const size_t blocks = std::min<size_t>((n / 2 + 255) / 256, 148 * 8);
    fill_zero_kernel<<<(unsigned)std::max<size_t>(blocks, 1), 256, 0, c.stream>>>(p, n);
    c.launches += 1;
    IBLGF_CUDA(cudaGetLastError());
}

namespace
{
// component blockIdx.z of one block
__global__ void __launch_bounds__(256) masked_copy_kernel(const __grid_constant__ TpFields f,
                                                          const int* __restrict__ flags, int half)
{
    const size_t off = (size_t)blockIdx.x * half;
    const double2* __restrict__ s = reinterpret_cast<const double2*>(f.src[blockIdx.z]) + off;
    double2* __restrict__ d = reinterpret_cast<double2*>(f.dst[blockIdx.z]) + off;
    const bool leaf = flags[blockIdx.x] & 1;
    double2 v[kPairs];
#pragma unroll
    for (int k = 0; k < kPairs; ++k)
    {
        const int i = blockIdx.y * kPiece + 256 * k + threadIdx.x;
        v[k] = leaf && i < half ? s[i] : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int k = 0; k < kPairs; ++k)
    {
        const int i = blockIdx.y * kPiece + 256 * k + threadIdx.x;
        if (i < half) d[i] = v[k];
    }
}

TpFields tp_fields(const double* const* src, double* const* dst, int n)
{
    TpFields f{};
    for (int k = 0; k < n; ++k)
    {
        f.src[k] = src ? src[k] : nullptr;
        f.dst[k] = dst[k];
    }
    return f;
}
}  // namespace

void launch_leaf_copy_vf(Ctx& c, const double* const* src, double* const* dst, int n)
{
    if (!c.n_oct || n < 1) return;
    const int half = (int)(c.block_elems() / 2);  // Nb is even, so blocks are whole 16-byte pieces
    masked_copy_kernel<<<dim3(c.n_oct, pieces(2 * half), n), 256, 0, c.stream>>>(tp_fields(src, dst, n), c.d_flags.p,
                                                                                 half);
    c.launches += 1;
    IBLGF_CUDA(cudaGetLastError());
}

void launch_zero_blocks_vf(Ctx& c, double* const* f, int m, const int* list, int n)
{
    if (!n || m < 1) return;
    const int half = (int)(c.block_elems() / 2);
    zero_kernel<<<dim3(n, pieces(2 * half), m), 256, 0, c.stream>>>(tp_fields(nullptr, f, m), list, half);
    c.launches += 1;
    IBLGF_CUDA(cudaGetLastError());
}

void launch_zero_blocks(Ctx& c, double* f, const int* list, int n) { launch_zero_blocks_vf(c, &f, 1, list, n); }

// one CTA per leaf; host order: leaf i's interior e^3 values, x fastest
__global__ void leaves_scatter_kernel(const double* __restrict__ stage, double* __restrict__ f,
                                      const int* __restrict__ list, int e, int NB)
{
    const int e3 = e * e * e;
    const double* s = stage + (size_t)blockIdx.x * e3;
    double* b = f + (size_t)list[blockIdx.x] * NB * NB * NB;
    for (int i = threadIdx.x; i < e3; i += blockDim.x)
    {
        const int x = i % e, y = (i / e) % e, z = i / (e * e);
        b[((z + 1) * NB + y + 1) * NB + x + 1] = s[i];
    }
}

__global__ void leaves_gather_kernel(const double* __restrict__ f, double* __restrict__ stage,
                                     const int* __restrict__ list, int e, int NB)
{
    const int e3 = e * e * e;
    double* s = stage + (size_t)blockIdx.x * e3;
    const double* b = f + (size_t)list[blockIdx.x] * NB * NB * NB;
    for (int i = threadIdx.x; i < e3; i += blockDim.x)
    {
        const int x = i % e, y = (i / e) % e, z = i / (e * e);
        s[i] = b[((z + 1) * NB + y + 1) * NB + x + 1];
    }
}

void launch_leaves_scatter(Ctx& c, const double* stage, double* field, const int* list, int n)
{
    if (!n) return;
    leaves_scatter_kernel<<<n, 256, 0, c.stream>>>(stage, field, list, c.Nb - 2, c.Nb);
    c.launches += 1;
    IBLGF_CUDA(cudaGetLastError());
}

namespace
{
// one CTA per listed block: field block <-> buf[i]
__global__ void blocks_copy_kernel(const double* __restrict__ from, double* __restrict__ to,
                                   const int* __restrict__ list, int b3, int gather)
{
    const size_t o = (size_t)list[blockIdx.x] * b3, i0 = (size_t)blockIdx.x * b3;
    for (int i = threadIdx.x; i < b3; i += blockDim.x)
    {
        if (gather) to[i0 + i] = from[o + i];
        else to[o + i] = from[i0 + i];
    }
}
}  // namespace

void launch_blocks_gather(Ctx& c, const double* field, double* buf, const int* list, int n)
{
    if (!n) return;
    blocks_copy_kernel<<<n, 256, 0, c.stream>>>(field, buf, list, (int)c.block_elems(), 1);
    c.launches += 1;
    IBLGF_CUDA(cudaGetLastError());
}

void launch_blocks_scatter(Ctx& c, const double* buf, double* field, const int* list, int n)
{
    if (!n) return;
    blocks_copy_kernel<<<n, 256, 0, c.stream>>>(buf, field, list, (int)c.block_elems(), 0);
    c.launches += 1;
    IBLGF_CUDA(cudaGetLastError());
}

void launch_leaves_gather(Ctx& c, const double* field, double* stage, const int* list, int n)
{
    if (!n) return;
    leaves_gather_kernel<<<n, 256, 0, c.stream>>>(field, stage, list, c.Nb - 2, c.Nb);
    c.launches += 1;
    IBLGF_CUDA(cudaGetLastError());
}

namespace
{
// the leaf blocks (flag bit 0) in canonical order and a staging buffer for
// their interiors, built on first use after each domain (re)build
int leaf_blocks(Ctx& c)
{
    if (c.n_leaf_blocks < 0)
    {
        std::vector<int> l;
        for (int o = 0; o < c.n_oct; ++o)
            if (c.flags[o] & 1) l.push_back(o);
        c.d_leaf_blocks.upload(l, c.stream);
        c.n_leaf_blocks = (int)l.size();
        const size_t e = (size_t)c.Nb - 2;
        c.leaf_stage.alloc(std::max<size_t>(1, l.size() * e * e * e), c.cfg.device, c.stream);
    }
    return c.n_leaf_blocks;
}
}  // namespace

// DataField::update_device / update_host (datafield.hpp:211-226) restricted to
// the values a solve reads and produces: the interiors of the leaf blocks.
// The upload zeroes the whole field first (buffers and non-leaf blocks).
void field_upload_leaves(Ctx& c, int f, const double* host, size_t count)
{
    if (!c.finalized) throw Error(IBLGF_EINVAL, "domain not finalized");
    const int n = leaf_blocks(c);
    const size_t e = (size_t)c.Nb - 2;
    if (!host || count != (size_t)n * e * e * e) throw Error(IBLGF_EINVAL, "leaf field size mismatch");
    IBLGF_CUDA(cudaMemcpyAsync(c.leaf_stage.p, host, count * sizeof(double), cudaMemcpyHostToDevice, c.stream));
    IBLGF_CUDA(cudaMemsetAsync(c.field(f), 0, c.field_elems() * sizeof(double), c.stream));
    launch_leaves_scatter(c, c.leaf_stage.p, c.field(f), c.d_leaf_blocks.p, n);
}

void field_download_leaves(Ctx& c, int f, double* host, size_t count)
{
    if (!c.finalized) throw Error(IBLGF_EINVAL, "domain not finalized");
    const int n = leaf_blocks(c);
    const size_t e = (size_t)c.Nb - 2;
    if (!host || count != (size_t)n * e * e * e) throw Error(IBLGF_EINVAL, "leaf field size mismatch");
    launch_leaves_gather(c, c.field(f), c.leaf_stage.p, c.d_leaf_blocks.p, n);
    IBLGF_CUDA(cudaMemcpyAsync(host, c.leaf_stage.p, count * sizeof(double), cudaMemcpyDeviceToHost, c.stream));
    IBLGF_CUDA(cudaStreamSynchronize(c.stream));
}

namespace
{
void ensure_copy_stream(Ctx& c)
{
    if (c.copy_stream) return;
    IBLGF_CUDA(cudaStreamCreateWithFlags(&c.copy_stream, cudaStreamNonBlocking));
    IBLGF_CUDA(cudaEventCreateWithFlags(&c.ev_gathered, cudaEventDisableTiming));
    IBLGF_CUDA(cudaEventCreateWithFlags(&c.ev_copied, cudaEventDisableTiming));
    IBLGF_CUDA(cudaEventCreateWithFlags(&c.ev_in_copied, cudaEventDisableTiming));
    IBLGF_CUDA(cudaEventCreateWithFlags(&c.ev_scattered, cudaEventDisableTiming));
    IBLGF_CUDA(cudaEventRecord(c.ev_copied, c.copy_stream));
    IBLGF_CUDA(cudaEventRecord(c.ev_scattered, c.stream));
}
}  // namespace

// Gather on the context stream, host copy on a second stream, so that the
// copy overlaps whatever the context stream runs next (the next upload, the
// next solve). The gather waits for the previous asynchronous copy out of
// leaf_out; iblgf_synchronize waits for both streams.
void field_download_leaves_async(Ctx& c, int f, double* host, size_t count)
{
    if (!c.finalized) throw Error(IBLGF_EINVAL, "domain not finalized");
    const int n = leaf_blocks(c);
    const size_t e = (size_t)c.Nb - 2, vals = (size_t)n * e * e * e;
    if (!host || count != vals) throw Error(IBLGF_EINVAL, "leaf field size mismatch");
    ensure_copy_stream(c);
    IBLGF_CUDA(cudaStreamWaitEvent(c.stream, c.ev_copied, 0));
    if (c.leaf_out.n != std::max<size_t>(1, vals)) c.leaf_out.alloc(std::max<size_t>(1, vals), c.cfg.device, c.stream);
    launch_leaves_gather(c, c.field(f), c.leaf_out.p, c.d_leaf_blocks.p, n);
    IBLGF_CUDA(cudaEventRecord(c.ev_gathered, c.stream));
    IBLGF_CUDA(cudaStreamWaitEvent(c.copy_stream, c.ev_gathered, 0));
    IBLGF_CUDA(cudaMemcpyAsync(host, c.leaf_out.p, vals * sizeof(double), cudaMemcpyDeviceToHost, c.copy_stream));
    IBLGF_CUDA(cudaEventRecord(c.ev_copied, c.copy_stream));
}

// Host copy on the copy stream into leaf_in, then zeroing and scatter into
// the field on the context stream, which waits for the copy; the copy waits
// for the previous upload's scatter out of leaf_in. Issued right after a
// solve, the copy of the next input runs under that solve.
void field_upload_leaves_async(Ctx& c, int f, const double* host, size_t count)
{
    if (!c.finalized) throw Error(IBLGF_EINVAL, "domain not finalized");
    const int n = leaf_blocks(c);
    const size_t e = (size_t)c.Nb - 2, vals = (size_t)n * e * e * e;
    if (!host || count != vals) throw Error(IBLGF_EINVAL, "leaf field size mismatch");
    ensure_copy_stream(c);
    if (c.leaf_in.n != std::max<size_t>(1, vals))
    {
        // stream-ordered on the context stream; the copy stream waits for it
        IBLGF_CUDA(cudaStreamSynchronize(c.copy_stream));
        c.leaf_in.alloc(std::max<size_t>(1, vals), c.cfg.device, c.stream);
        IBLGF_CUDA(cudaEventRecord(c.ev_scattered, c.stream));
    }
    IBLGF_CUDA(cudaStreamWaitEvent(c.copy_stream, c.ev_scattered, 0));
    IBLGF_CUDA(cudaMemcpyAsync(c.leaf_in.p, host, vals * sizeof(double), cudaMemcpyHostToDevice, c.copy_stream));
    IBLGF_CUDA(cudaEventRecord(c.ev_in_copied, c.copy_stream));
    IBLGF_CUDA(cudaStreamWaitEvent(c.stream, c.ev_in_copied, 0));
    IBLGF_CUDA(cudaMemsetAsync(c.field(f), 0, c.field_elems() * sizeof(double), c.stream));
    launch_leaves_scatter(c, c.leaf_in.p, c.field(f), c.d_leaf_blocks.p, n);
    IBLGF_CUDA(cudaEventRecord(c.ev_scattered, c.stream));
}

void copy_stream_release(Ctx& c)
{
    if (!c.copy_stream) return;
    cudaStreamSynchronize(c.copy_stream);
    cudaStreamSynchronize(c.stream);
    c.leaf_out.release();
    c.leaf_in.release();
    cudaEventDestroy(c.ev_gathered);
    cudaEventDestroy(c.ev_copied);
    cudaEventDestroy(c.ev_in_copied);
    cudaEventDestroy(c.ev_scattered);
    cudaStreamDestroy(c.copy_stream);
    c.copy_stream = nullptr;
    c.ev_gathered = c.ev_copied = c.ev_in_copied = c.ev_scattered = nullptr;
}

void launch_copy_interior_vf(Ctx& c, const double* const* src, double* const* dst, int m, const int* list, int n)
{
    if (!n || m < 1) return;
    nb_dispatch(c.Nb, [&](auto nbc) {
        constexpr int NB = decltype(nbc)::value;
        copy_interior_kernel<NB><<<dim3(n, pieces(NB * NB * NB), m), 256, 0, c.stream>>>(tp_fields(src, dst, m), list);
    });
    c.launches += 1;
    IBLGF_CUDA(cudaGetLastError());
}

void launch_copy_interior(Ctx& c, const double* src, double* dst, const int* list, int n)
{
    launch_copy_interior_vf(c, &src, &dst, 1, list, n);
}

void launch_axpy_blocks(Ctx& c, const double* src, double* dst, const int* list, int n, double a, bool assign,
                        double* leaf_out)
{
    if (!n) return;
    const int half = (int)(c.block_elems() / 2);
    axpy_kernel<<<dim3(n, pieces(2 * half)), 256, 0, c.stream>>>(
        reinterpret_cast<const double2*>(src), reinterpret_cast<double2*>(dst), list, half, a, assign ? 1 : 0,
        c.d_flags.p, reinterpret_cast<double2*>(leaf_out));
    c.launches += 1;
    IBLGF_CUDA(cudaGetLastError());
}

// Adaptation: new block b takes old block src[b] (or zeros when src[b] < 0)
__global__ void remap_blocks_kernel(const double2* __restrict__ old, double2* __restrict__ nw,
                                    const int* __restrict__ src, int half_block)
{
    const int b = blockIdx.x;
    const int s = src[b];
    double2* d = nw + (size_t)b * half_block;
    if (s < 0)
        for (int i = threadIdx.x; i < half_block; i += blockDim.x) d[i] = make_double2(0.0, 0.0);
    else
    {
        const double2* o = old + (size_t)s * half_block;
        for (int i = threadIdx.x; i < half_block; i += blockDim.x) d[i] = o[i];
    }
}

void launch_remap_blocks(Ctx& c, const double* old, double* nw, const int* d_src, int n_new)
{
    if (!n_new) return;
    const int half = (int)(c.block_elems() / 2);  // Nb even: Nb^3 / 2 double2
    remap_blocks_kernel<<<n_new, 256, 0, c.stream>>>(reinterpret_cast<const double2*>(old),
                                                     reinterpret_cast<double2*>(nw), d_src, half);
    c.launches += 1;
    IBLGF_CUDA(cudaGetLastError());
}

// Operator::maxnorm / blockRootMeanSquare (operators.hpp:1149-1211) over the
// block's interior nodes: max over nodes of sqrt(sum_c v_c^2) and
// sqrt(sum_nodes sum_c v_c^2 / nodes)
__global__ void block_norms_kernel(const double* __restrict__ f0, const double* __restrict__ f1,
                                   const double* __restrict__ f2, int n_comp, int NB, double* __restrict__ out_max,
                                   double* __restrict__ out_rms)
{
    const int b = blockIdx.x;
    const int e = NB - 2;
    const size_t base = (size_t)b * NB * NB * NB;
    double mx = 0.0, sum = 0.0;
    for (int i = threadIdx.x; i < e * e * e; i += blockDim.x)
    {
        const int x = i % e + 1, y = (i / e) % e + 1, z = i / (e * e) + 1;
        const size_t at = base + x + (size_t)NB * (y + (size_t)NB * z);
        double v = f0[at] * f0[at];
        if (n_comp > 1) v += f1[at] * f1[at];
        if (n_comp > 2) v += f2[at] * f2[at];
        sum += v;
        mx = fmax(mx, sqrt(v));
    }
    __shared__ double smx[256], ssum[256];
    smx[threadIdx.x] = mx;
    ssum[threadIdx.x] = sum;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1)
    {
        if ((int)threadIdx.x < o)
        {
            smx[threadIdx.x] = fmax(smx[threadIdx.x], smx[threadIdx.x + o]);
            ssum[threadIdx.x] += ssum[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0)
    {
        out_max[b] = smx[0];
        out_rms[b] = sqrt(ssum[0] / ((double)e * e * e));
    }
}

void launch_block_norms(Ctx& c, const double* const* comps, int n_comp, double* d_max, double* d_rms)
{
    if (!c.n_oct) return;
    block_norms_kernel<<<c.n_oct, 256, 0, c.stream>>>(comps[0], n_comp > 1 ? comps[1] : comps[0],
                                                      n_comp > 2 ? comps[2] : comps[0], n_comp, c.Nb, d_max, d_rms);
    c.launches += 1;
    IBLGF_CUDA(cudaGetLastError());
}

}  // namespace iblgf_b200
