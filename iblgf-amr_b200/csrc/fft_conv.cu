// Batched per-block FFT convolution of the LGF-FMM sweep, hand-written for
// sm_100a (no cuFFT). Contract: include/iblgf/utilities/convolution.hpp:225-304
// and src/utilities/convolution.cpp — a zero-padded Nb^3 source and a
// (2Nb-1)^3 LGF block in a P^3 = (2Nb-1)^3 box, r2c, pointwise product
// accumulated per target, c2r, window [Nb-1, 2Nb-2]^3 scaled by dx^2 / P^3 into
// the target block.
//
// B200 structure (one sweep = all blocks of all tree levels at once):
//   forward      each source block once per sweep (the reference transforms it
//                once per (source, target) pair): one kernel for the extents
//                with a prime-factor split (inverse.cu), two for the others:
//     fwd_xy_rows  one CTA per source block: thread (z, y) transforms row y
//                  along x (real, Nb -> Nb half frequencies), thread (z, kx)
//                  then column kx along y (Nb -> P)
//     fwd_z        one thread per (ky,kx) pencil: z transform (Nb -> P)
//   bundle_mac   sibling-group spectral multiply-accumulate (mac_kernel:
//                general pair-list fallback)
//   inverse      assigned to the FP64 target block: one kernel for the extents
//                with a prime-factor split (inverse.cu), for the others
//                inv_fused, one CTA per (target, half of the output planes): z
//                inverse, y inverse and c2r along x of the extraction window,
//                in shared memory
// The half spectrum is laid out [kz][ky][kx], kx < Nb (= P/2 + 1), as in the
// reference's r2c output. Transforms are direct pruned DFTs (half of the
// inputs zero, half of the outputs discarded). The forward loops are unrolled
// over frequency and sample index so each twiddle is a compile-time constant
// operand; the FP64 inverse reads a per-CTA twiddle table instead.
#include <cmath>
#include <mutex>
#include <set>
#include <type_traits>
#include <vector>

#include <cuda_pipeline.h>

#include "cplx.cuh"
#include "ctx.hpp"
#include "lgf_dev.cuh"

namespace iblgf_b200
{
namespace
{
template<class R>
__device__ __forceinline__ void load_tw(cx<R>* s_tw, const R* tw, int P)
{
    for (int j = threadIdx.x; j < P; j += blockDim.x) s_tw[j] = mk<R>(tw[2 * j], tw[2 * j + 1]);
}

// Twiddles e^{-2 pi i j / P} of every supported P (Nb = 6, 8, 10, 12, 16, 18)
// in constant memory. The transform loops below are unrolled over both the
// frequency and the sample index, so (k * j) mod P is a compile-time constant
// and every twiddle is an immediate FMA operand: no shared-memory loads.
constexpr int kTwTotal = 11 + 15 + 19 + 23 + 31 + 35;
__host__ __device__ constexpr int tw_base(int P)
{
    return P == 11 ? 0 : P == 15 ? 11 : P == 19 ? 26 : P == 23 ? 45 : P == 31 ? 68 : 99;
}
__constant__ double c_tw64[2 * kTwTotal];
__constant__ float c_tw32[2 * kTwTotal];

template<class R, int P>
__device__ __forceinline__ cx<R> ctw(int j)
{
    if constexpr (std::is_same<R, double>::value)
        return mk<R>(c_tw64[2 * (tw_base(P) + j)], c_tw64[2 * (tw_base(P) + j) + 1]);
    else
        return mk<R>(c_tw32[2 * (tw_base(P) + j)], c_tw32[2 * (tw_base(P) + j) + 1]);
}

// x and y transforms of a whole field block: thread (z, y) takes row y of
// plane z along x (real NB -> NB half frequencies) into shared memory, then
// thread (z, kx) takes column kx of plane z along y (NB -> P) and writes
// W[item][z][ky][kx]. One CTA (NB^2 threads) per block; shared rows have an
// odd stride (NB + 1 complex), so both passes are free of bank conflicts.
template<class R, int NB>
__global__ void __launch_bounds__(NB * NB) fwd_xy_rows_kernel(const double* __restrict__ field,
                                                              const int* __restrict__ item_oct,
                                                              cx<R>* __restrict__ W)
{
    constexpr int P = 2 * NB - 1, S = NB + 1;
    extern __shared__ __align__(16) unsigned char smraw[];
    cx<R>* s_x1 = reinterpret_cast<cx<R>*>(smraw);  // [z][y][kx]
    const int item = blockIdx.x;
    const int z = threadIdx.x / NB, r = threadIdx.x % NB;
    {
        const double* row = field + (size_t)item_oct[item] * (NB * NB * NB) + (size_t)threadIdx.x * NB;
        R in[NB];
#pragma unroll
        for (int x = 0; x < NB; ++x) in[x] = (R)row[x];
        cx<R>* dst = s_x1 + (size_t)threadIdx.x * S;
#pragma unroll
        for (int kx = 0; kx < NB; ++kx)
        {
            cx<R> s = mk<R>(0, 0);
#pragma unroll
            for (int x = 0; x < NB; ++x) rmac<R>(s, in[x], ctw<R, P>((kx * x) % P));
            dst[kx] = s;
        }
    }
    __syncthreads();
    cx<R> v[NB];
#pragma unroll
    for (int y = 0; y < NB; ++y) v[y] = s_x1[(z * NB + y) * S + r];
    cx<R>* out = W + ((size_t)item * NB + z) * (P * NB) + r;
#pragma unroll
    for (int ky = 0; ky < P; ++ky)
    {
        cx<R> s = mk<R>(0, 0);
#pragma unroll
        for (int y = 0; y < NB; ++y) cmac<R>(s, v[y], ctw<R, P>((ky * y) % P));
        out[(size_t)ky * NB] = s;
    }
}

// x and y transforms of one staged z plane s_in[y][x] (NIN rows of NIN) into
// out[ky][kx]
template<class R, int NB, int NIN>
__device__ __forceinline__ void plane_xy(const cx<R>* s_tw, const R* s_in, cx<R>* s_x1, cx<R>* __restrict__ out)
{
    constexpr int P = 2 * NB - 1;
    // x: real NIN -> NB half frequencies
    for (int i = threadIdx.x; i < NIN * NB; i += blockDim.x)
    {
        const int y = i / NB, kx = i % NB;
        cx<R> s = mk<R>(0, 0);
        int j = 0;
#pragma unroll 6
        for (int x = 0; x < NIN; ++x)
        {
            rmac<R>(s, s_in[y * NIN + x], s_tw[j]);
            j += kx;
            if (j >= P) j -= P;
        }
        s_x1[y * NB + kx] = s;
    }
    __syncthreads();
    // y: NIN -> P
    for (int i = threadIdx.x; i < P * NB; i += blockDim.x)
    {
        const int ky = i / NB, kx = i % NB;
        cx<R> s = mk<R>(0, 0);
        int j = 0;
#pragma unroll 6
        for (int y = 0; y < NIN; ++y)
        {
            cmac<R>(s, s_x1[y * NB + kx], s_tw[j]);
            j += ky;
            if (j >= P) j -= P;
        }
        out[i] = s;
    }
}

// fwd_xy: x and y transforms of one z plane of one LGF block, in FP64:
//   desc[4*item] = {ld, bx, by, bz}: G((b + i) * 2^ld), ld < 0: table -ld-1 of
//   the integrating factor
// W: [item][z < P][ky < P][kx < NB]
template<int NB>
__global__ void __launch_bounds__(256) fwd_xy_kernel(const int* __restrict__ desc, const double* __restrict__ table,
                                                     const double* __restrict__ tw, double2* __restrict__ W,
                                                     const double* __restrict__ ge, int ge_stride)
{
    constexpr int P = 2 * NB - 1, NIN = P;
    __shared__ double2 s_tw[P];
    __shared__ double s_in[NIN * NIN];
    __shared__ double2 s_x1[NIN * NB];
    const int item = blockIdx.x;
    const int z = blockIdx.y;
    load_tw<double>(s_tw, tw, P);
    // desc[0] >= 0: LGF_GL at stride 2^level_diff (lgf.hpp:222-262);
    // desc[0] < 0: LGF_GE table -desc[0]-1, E(n) = f[|n1|] f[|n2|] f[|n3|]
    const int ld = desc[4 * item];
    const int bx = desc[4 * item + 1], by = desc[4 * item + 2], bz = desc[4 * item + 3];
    if (ld >= 0)
    {
        const int st = 1 << ld;
        for (int i = threadIdx.x; i < NIN * NIN; i += blockDim.x)
        {
            const int x = i % NIN, y = i / NIN;
            s_in[i] = lgf_get_dev((bx + x) * st, (by + y) * st, (bz + z) * st, table);
        }
    }
    else
    {
        const double* f = ge + (size_t)(-ld - 1) * ge_stride;
        const double fz = f[abs(bz + z)];
        for (int i = threadIdx.x; i < NIN * NIN; i += blockDim.x)
        {
            const int x = i % NIN, y = i / NIN;
            s_in[i] = f[abs(bx + x)] * f[abs(by + y)] * fz;
        }
    }
    __syncthreads();
    plane_xy<double, NB, NIN>(s_tw, s_in, s_x1, W + ((size_t)item * NIN + z) * (P * NB));
}

// Single-block convolution (fft::Convolution, convolution.hpp:141-328): out +=
// scale * window of source * kernel, in three launches that spread the one
// block over the chip (one CTA per block left 147 SMs idle: 82 us in six
// launches at Nb = 18 FP64).
//   conv_xy   CTA per z plane of the kernel (P, FP64) and of the source (NB)
//   conv_z    CTA per ky: z transforms of both, their product (kernel spectrum
//             rounded to R first, as the sweeps keep it) and the inverse z
//             transform to the NB window planes, in shared memory
//   conv_out  CTA per window plane: inverse y, c2r along x, added to out
// The inverse runs in FP64 in both precisions. Where P = N1 N2 (pfa_extent) its z
// and y passes take the prime-factor form in two stages, a thread per value of
// each: N2 sums of N1 terms, then the window outputs as sums of N2 terms. Sums of
// 5 and 7 instead of 35 terms round less: relative 2-norm error of the whole
// convolution in FP64 against extended precision 7.2e-16 instead of 8.3e-16 at extent
// 16, 7.5e-16 instead of 8.3e-16 at extent 6.
template<int NB>
struct ConvSplit
{
    static constexpr int P = 2 * NB - 1, N1 = P == 35 ? 5 : 3, N2 = P / N1;
};

// first stage: T[n2][k1][kx] = sum_n1 in[(N2 n1 + N1 n2) mod P][kx] e^{2 pi i n1 k1 / N1}
// of item = (n2 N1 + k1) NB + kx; tw[j] = e^{-2 pi i j / P}
template<int NB>
__device__ __forceinline__ void conv_stage1(const double2* in, double2* T, const double2* tw, int item)
{
    using S = ConvSplit<NB>;
    constexpr int P = S::P, N1 = S::N1, N2 = S::N2;
    const int kx = item % NB, r = item / NB, n2 = r / N1, k1 = r % N1;
    int n = N1 * n2 % P, j = 0;
    double2 v = make_double2(0.0, 0.0);
#pragma unroll
    for (int n1 = 0; n1 < N1; ++n1)
    {
        cmac_conj<double>(v, in[n * NB + kx], tw[j * N2]);
        n = n + N2 >= P ? n + N2 - P : n + N2;
        j = j + k1 >= N1 ? j + k1 - N1 : j + k1;
    }
    T[item] = v;
}

// second stage: output o = sum_n2 T[n2][o mod N1][kx] e^{2 pi i n2 o / N2}
template<int NB>
__device__ __forceinline__ double2 conv_stage2(const double2* T, const double2* tw, int o, int kx)
{
    using S = ConvSplit<NB>;
    constexpr int N1 = S::N1, N2 = S::N2;
    const int k1 = o % N1, k2 = o % N2;
    int j = 0;
    double2 v = make_double2(0.0, 0.0);
#pragma unroll
    for (int n2 = 0; n2 < N2; ++n2)
    {
        cmac_conj<double>(v, T[(n2 * N1 + k1) * NB + kx], tw[j * N1]);
        j = j + k2 >= N2 ? j + k2 - N2 : j + k2;
    }
    return v;
}

template<class R, int NB>
__global__ void __launch_bounds__(256) conv_xy_kernel(const double* __restrict__ kernel,
                                                      const double* __restrict__ source,
                                                      const double* __restrict__ tw, double2* __restrict__ WK,
                                                      cx<R>* __restrict__ WS)
{
    constexpr int P = 2 * NB - 1;
    __shared__ double2 s_tw[P];
    __shared__ double s_in[P * P];
    __shared__ double2 s_x1[P * NB];
    const int z = blockIdx.x;
    if (z < P)
    {
        load_tw<double>(s_tw, tw, P);
        for (int i = threadIdx.x; i < P * P; i += blockDim.x) s_in[i] = kernel[(size_t)z * P * P + i];
        __syncthreads();
        plane_xy<double, NB, P>(s_tw, s_in, s_x1, WK + (size_t)z * P * NB);
    }
    else
    {
        cx<R>* t = reinterpret_cast<cx<R>*>(s_tw);
        R* in = reinterpret_cast<R*>(s_in);
        for (int j = threadIdx.x; j < P; j += blockDim.x) t[j] = mk<R>((R)tw[2 * j], (R)tw[2 * j + 1]);
        for (int i = threadIdx.x; i < NB * NB; i += blockDim.x) in[i] = (R)source[(size_t)(z - P) * NB * NB + i];
        __syncthreads();
        plane_xy<R, NB, NB>(t, in, reinterpret_cast<cx<R>*>(s_x1), WS + (size_t)(z - P) * P * NB);
    }
}

template<class R, int NB>
__global__ void __launch_bounds__((2 * NB - 1) * NB) conv_z_kernel(const double2* __restrict__ WK,
                                                                   const cx<R>* __restrict__ WS,
                                                                   const double* __restrict__ tw,
                                                                   double2* __restrict__ V)
{
    constexpr int P = 2 * NB - 1, NP = P * NB;
    __shared__ double2 s_tw[P];
    __shared__ cx<R> s_twr[P];
    __shared__ double2 s_k[P * NB];
    __shared__ cx<R> s_s[NB * NB];
    __shared__ double2 s_p[P * NB];
    const int ky = blockIdx.x, kx = threadIdx.x % NB, kz = threadIdx.x / NB;
    for (int j = threadIdx.x; j < P; j += blockDim.x)
    {
        s_tw[j] = make_double2(tw[2 * j], tw[2 * j + 1]);
        s_twr[j] = mk<R>((R)tw[2 * j], (R)tw[2 * j + 1]);
    }
    s_k[threadIdx.x] = WK[(size_t)kz * NP + ky * NB + kx];
    if (kz < NB) s_s[threadIdx.x] = WS[(size_t)kz * NP + ky * NB + kx];
    __syncthreads();
    double2 g = make_double2(0.0, 0.0);
    cx<R> s = mk<R>(0, 0);
    int j = 0;
#pragma unroll 5
    for (int z = 0; z < P; ++z)
    {
        cmac<double>(g, s_k[z * NB + kx], s_tw[j]);
        if (z < NB) cmac<R>(s, s_s[z * NB + kx], s_twr[j]);
        j += kz;
        if (j >= P) j -= P;
    }
    cx<R> p = mk<R>(0, 0);
    cmac<R>(p, mk<R>((R)g.x, (R)g.y), s);
    s_p[threadIdx.x] = make_double2((double)p.x, (double)p.y);
    __syncthreads();
    // window plane zo = kz
    double2 v = make_double2(0.0, 0.0);
    if constexpr (pfa_extent(NB))
    {
        conv_stage1<NB>(s_p, s_k, s_tw, threadIdx.x);
        __syncthreads();
        if (kz >= NB) return;
        v = conv_stage2<NB>(s_k, s_tw, kz + NB - 1, kx);
    }
    else
    {
        if (kz >= NB) return;
        j = 0;
#pragma unroll 5
        for (int k = 0; k < P; ++k)
        {
            cmac_conj<double>(v, s_p[k * NB + kx], s_tw[j]);
            j += kz + NB - 1;
            if (j >= P) j -= P;
        }
    }
    V[((size_t)kz * P + ky) * NB + kx] = v;
}

template<int NB>
__global__ void __launch_bounds__(NB* NB) conv_out_kernel(const double2* __restrict__ V,
                                                          const double* __restrict__ tw, double scale,
                                                          double* __restrict__ out)
{
    constexpr int P = 2 * NB - 1;
    __shared__ double2 s_tw[P];
    __shared__ double2 s_v[P * NB];
    __shared__ double2 s_y[NB * (NB + 1)];
    __shared__ double2 s_t[pfa_extent(NB) ? P * NB : 1];
    const int zo = blockIdx.x, a = threadIdx.x % NB, yo = threadIdx.x / NB;
    for (int j = threadIdx.x; j < P; j += blockDim.x) s_tw[j] = make_double2(tw[2 * j], tw[2 * j + 1]);
    for (int i = threadIdx.x; i < P * NB; i += blockDim.x) s_v[i] = V[(size_t)zo * P * NB + i];
    __syncthreads();
    double2 v = make_double2(0.0, 0.0);
    int j = 0;
    if constexpr (pfa_extent(NB))
    {
        for (int i = threadIdx.x; i < P * NB; i += NB * NB) conv_stage1<NB>(s_v, s_t, s_tw, i);
        __syncthreads();
        v = conv_stage2<NB>(s_t, s_tw, yo + NB - 1, a);
    }
    else
    {
#pragma unroll 5
        for (int k = 0; k < P; ++k)
        {
            cmac_conj<double>(v, s_v[k * NB + a], s_tw[j]);
            j += yo + NB - 1;
            if (j >= P) j -= P;
        }
    }
    s_y[yo * (NB + 1) + a] = v;
    __syncthreads();
    // c2r: Re y_0 + 2 sum_{k >= 1} Re(y_k e^{+2 pi i k (xo + NB - 1) / P}), xo = a,
    // in two sums of half the terms each
    double sx[2] = {0.5 * s_y[yo * (NB + 1)].x, 0.0};
    j = 0;
#pragma unroll
    for (int k = 1; k < NB; ++k)
    {
        j += a + NB - 1;
        if (j >= P) j -= P;
        const double2 y = s_y[yo * (NB + 1) + k], t = s_tw[j];
        double& s = sx[k < NB / 2 ? 0 : 1];
        s = fma(y.x, t.x, fma(y.y, t.y, s));
    }
    out[((size_t)zo * NB + yo) * NB + a] += scale * (2.0 * (sx[0] + sx[1]));
}

// fwd_z: per (ky,kx) pencil, NIN -> P; spectrum slot = item_slot[item] (or item)
template<class R, class RO, int NB, int NIN>
__global__ void __launch_bounds__(128) fwd_z_kernel(const cx<R>* __restrict__ W, const int* __restrict__ item_slot,
                                                    cx<RO>* __restrict__ spec)
{
    constexpr int P = 2 * NB - 1;
    constexpr int NP = P * NB;
    const int item = blockIdx.x;
    const int p = blockIdx.y * blockDim.x + threadIdx.x;
    if (p >= NP) return;
    const cx<R>* w = W + (size_t)item * NIN * NP + p;
    cx<R> v[NIN];
#pragma unroll
    for (int z = 0; z < NIN; ++z) v[z] = w[(size_t)z * NP];
    const int slot = item_slot ? item_slot[item] : item;
    cx<RO>* out = spec + (size_t)slot * P * NP + p;
    if constexpr (NIN > NB)
    {
        // dense P-point input (LGF spectra, cache fill only): kz rolled
#pragma unroll 1
        for (int kz = 0; kz < P; ++kz)
        {
            cx<R> s = mk<R>(0, 0);
            int j = 0;
#pragma unroll
            for (int z = 0; z < NIN; ++z)
            {
                cmac<R>(s, v[z], ctw<R, P>(j));
                j += kz;
                if (j >= P) j -= P;
            }
            out[(size_t)kz * NP] = mk<RO>((RO)s.x, (RO)s.y);
        }
    }
    else
    {
#pragma unroll
        for (int kz = 0; kz < P; ++kz)
        {
            cx<R> s = mk<R>(0, 0);
#pragma unroll
            for (int z = 0; z < NIN; ++z) cmac<R>(s, v[z], ctw<R, P>((kz * z) % P));
            out[(size_t)kz * NP] = mk<RO>((RO)s.x, (RO)s.y);
        }
    }
}

// mac: ACC[t][f] = sum_pairs G[spec][f] * S[src][f]
template<class R>
__global__ void __launch_bounds__(128) mac_kernel(const cx<R>* __restrict__ G, const cx<R>* __restrict__ S,
                                                  const int* __restrict__ pair_ptr,
                                                  const int* __restrict__ pair_src,
                                                  const int* __restrict__ pair_spec, long long NC,
                                                  cx<R>* __restrict__ ACC)
{
    const long long f = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const int t = blockIdx.y;
    if (f >= NC) return;
    cx<R> acc = mk<R>(0, 0);
    const int j0 = pair_ptr[t], j1 = pair_ptr[t + 1];
    for (int j = j0; j < j1; ++j)
    {
        const cx<R> g = G[(size_t)pair_spec[j] * NC + f];
        const cx<R> s = S[(size_t)pair_src[j] * NC + f];
        cmac<R>(acc, g, s);
    }
    ACC[(size_t)t * NC + f] = acc;
}

// Sibling-group MAC. At a sweep's base level the neighbours and the influence
// list of a target together are exactly the children of its parent's 27
// neighbours; coarser targets see the non-adjacent ones. The 8 siblings of a
// parent therefore share one candidate source set (216 = 27 x 8 candidates
// k = (n, c')), and the offset of (child c, candidate (n, c')) is
// u = c - c' - 2n in [-3,3]^3. For one neighbour parent n the 64 (c, c') pairs
// use only the 27 offsets u = d - 2n, d = c - c' in [-1,1]^3.
//
// One warp = NG = 2 sibling groups of one LGF table (a bundle) at 32
// consecutive frequencies. It walks the bundle's half parents (n, c'z): the 18
// LGF values of one go from shared memory into registers once and serve both
// groups, whose 16 accumulators stay in registers for the whole walk; the
// source values are read straight from their rows (256-byte row segments in
// FP32), one group ahead of their use. The CTA stages the table's 343 rows at
// its 32 frequencies in shared memory and its warps take the tile's bundles
// from a counter.
// A half parent with all 4 candidates, seen from a group with all 4 target
// rows (pairs along x), runs its 32 products without a branch; elsewhere
// absent candidates, target rows without a target and rows beyond the adjacent
// ones (neighbour-only plans) are skipped. Offsets that a plan excludes
// altogether (adjacent ones of coarse targets, the others of neighbour-only
// plans) are zero rows of the staged table.
template<class R, int CY, int CZ, int Q>
__device__ __forceinline__ void mac_row(const cx<R> (&gv)[9], const cx<R>& s, cx<R>* acc)
{
    // targets c = (0, CY, CZ) and (1, CY, CZ) of source child Q + 4 c'z;
    // gv[(dx + 1) + 3 (dy + 1)] with d = c - c', of the plane dz = CZ - c'z
    constexpr int d0 = (0 - (Q & 1) + 1) + 3 * (CY - (Q >> 1) + 1);
    cmac<R>(acc[2 * CY + 4 * CZ], gv[d0], s);
    cmac<R>(acc[2 * CY + 4 * CZ + 1], gv[d0 + 1], s);
}

template<class R, int CZ, int Q>
__device__ __forceinline__ void mac_source(const cx<R> (&gv)[9], const cx<R>& s, cx<R>* acc)
{
    mac_row<R, 0, CZ, Q>(gv, s, acc);
    mac_row<R, 1, CZ, Q>(gv, s, acc);
}

// the products of one half parent with the target rows cz = CZ of one group;
// mask: bit 4 q + cy + 2 cz of each candidate and target row to take (all 16
// set also where the few absent candidates read the zero row)
template<class R, int CZ>
__device__ __forceinline__ void mac_half(const cx<R> (&gv)[9], const cx<R> (&s)[4], cx<R>* acc, unsigned mask)
{
    if (mask == 0xFFFFu)
    {
        mac_source<R, CZ, 0>(gv, s[0], acc);
        mac_source<R, CZ, 1>(gv, s[1], acc);
        mac_source<R, CZ, 2>(gv, s[2], acc);
        mac_source<R, CZ, 3>(gv, s[3], acc);
    }
    else if (mask & (0x3333u << (2 * CZ)))
    {
        constexpr unsigned b = 1u << (2 * CZ);
        if (mask & b) mac_row<R, 0, CZ, 0>(gv, s[0], acc);
        if (mask & (b << 1)) mac_row<R, 1, CZ, 0>(gv, s[0], acc);
        if (mask & (b << 4)) mac_row<R, 0, CZ, 1>(gv, s[1], acc);
        if (mask & (b << 5)) mac_row<R, 1, CZ, 1>(gv, s[1], acc);
        if (mask & (b << 8)) mac_row<R, 0, CZ, 2>(gv, s[2], acc);
        if (mask & (b << 9)) mac_row<R, 1, CZ, 2>(gv, s[2], acc);
        if (mask & (b << 12)) mac_row<R, 0, CZ, 3>(gv, s[3], acc);
        if (mask & (b << 13)) mac_row<R, 1, CZ, 3>(gv, s[3], acc);
    }
}

template<class R, int NB>
__device__ __forceinline__ void mac_load(cx<R> (&s)[4], const cx<R>* Sf, const uint4& r)
{
    constexpr unsigned NC = (unsigned)NB * (2 * NB - 1) * (2 * NB - 1);
    s[0] = __ldg(Sf + (unsigned long long)r.x * NC);
    s[1] = __ldg(Sf + (unsigned long long)r.y * NC);
    s[2] = __ldg(Sf + (unsigned long long)r.z * NC);
    s[3] = __ldg(Sf + (unsigned long long)r.w * NC);
}

// Bound by instruction issue (FP32: 72% of the issue slots, three quarters of
// them FFMAs; FP64: the DFMA pipe and the LGF rows' shared-memory reads), with
// DRAM at a tenth. Against one group per warp, 64 frequencies per CTA and tiles
// of 32 groups, each of one problem of a batch: the MAC of a batch of 256
// problems 6.06 -> 1.88 ms (one staged table for 192 groups of any problem
// instead of one for the few groups of each), amr_3level FP32 7.53 -> 7.08 ms,
// vortex ring FP32 1.12 -> 1.04 ms, amr_2level FP64 3.45 -> 3.41 ms. In FP32
// the source values are loaded one half parent ahead, at 16 warps (122
// registers), instead of 20 warps without: solves of amr_3level 11.21 -> 11.05
// ms, of 256 problems 2.86 -> 2.83 ms, vortex ring step 11.92 -> 11.64 ms. Not
// kept: all 27 LGF values of a parent in registers without shared memory (10.0
// ms on amr_3level), LGF rows read through L1 by small warps (25 ms), two CTAs
// of 10 warps per SM (less L1 for the source rows: +0.7 ms), packed FP32 FMAs
// with their accumulators doubled (+0.7 ms).
// In a split tile (bit 2 of its mode) a warp takes one group of a bundle and one
// half (cz) of its targets: tables of at most kMacSplit bundles. ALL: every tile is split, and the kernel keeps the registers
// of that path only (FP32: two CTAs per SM), for plans with few groups (8
// groups of a uniform 64^3 solve: 52 against 73 us).
template<class R, int NB, int NT, int MINB, bool ALL>
__global__ void __launch_bounds__(NT, MINB) bundle_mac_kernel(
    const cx<R>* __restrict__ G, const cx<R>* __restrict__ S, const int4* __restrict__ tiles,
    const int* __restrict__ spec_u, const int* __restrict__ bundle_ptr, const int2* __restrict__ bundle_grp,
    const uint2* __restrict__ head, const uint4* __restrict__ rows, const int* __restrict__ tgt,
    cx<R>* __restrict__ ACC)
{
    constexpr int P = 2 * NB - 1, F = 32;
    constexpr long long NC = (long long)NB * P * P;
    constexpr int per = 16 / sizeof(cx<R>), parts = F / per;  // 16-byte pieces of a staged row
    extern __shared__ __align__(16) unsigned char smraw[];
    cx<R>* Gs = reinterpret_cast<cx<R>*>(smraw);  // [343][F]
    int* Sl = reinterpret_cast<int*>(Gs + 343 * F);
    int* next = Sl + 343;
    const int4 tile = tiles[blockIdx.x];  // first bundle, end, table, mode: 0 all, 1 non-adjacent, 2 adjacent
    const int mode = tile.w & 3;
    const bool split = ALL || (tile.w & 4);
    const long long f0 = (long long)blockIdx.y * F;
    const cx<R> zero = mk<R>(0, 0);
    for (int r = threadIdx.x; r < 343; r += NT)
    {
        const int ux = r % 7 - 3, uy = (r / 7) % 7 - 3, uz = r / 49 - 3;
        const bool adj = ux >= -1 && ux <= 1 && uy >= -1 && uy <= 1 && uz >= -1 && uz <= 1;
        Sl[r] = (mode == 1 && adj) || (mode == 2 && !adj) ? -1 : spec_u[343 * tile.z + r];
    }
    if (threadIdx.x == 0) *next = split ? 4 * tile.x : tile.x;
    __syncthreads();
    const bool full = f0 + F <= NC;
    for (int q = threadIdx.x; q < 343 * parts; q += NT)
    {
        const int r = q / parts, part = q % parts, slot = Sl[r];
        cx<R>* dst = Gs + r * F + part * per;
        const cx<R>* src = G + (size_t)max(slot, 0) * NC + f0 + part * per;
        if (slot >= 0 && full) __pipeline_memcpy_async(dst, src, 16);
        else
            for (int e = 0; e < per; ++e) dst[e] = (slot >= 0 && f0 + part * per + e < NC) ? src[e] : zero;
    }
    __pipeline_commit();
    __pipeline_wait_prior(0);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const long long f = f0 + lane;
    const cx<R>* Sf = S + (f < NC ? f : NC - 1);  // clamped column for the tail
    for (;;)
    {
        int item = 0;
        if (lane == 0) item = atomicAdd(next, 1);
        item = __shfl_sync(0xffffffffu, item, 0);
        const int b = split ? item >> 2 : item;
        if (b >= tile.y) return;
        const int2 bg = bundle_grp[b];
        const int e0 = bundle_ptr[b], e1 = bundle_ptr[b + 1];
        const uint2* hp = head + e0;
        if (split)
        {
            const int i = (item >> 1) & 1, cz = item & 1, g = i ? bg.y : bg.x;
            if (g < 0) continue;
            cx<R> acc[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[c] = zero;
            // source values one half parent ahead, their rows two (the lists end
            // with spare entries)
            const uint4* rp = rows + 2 * (size_t)e0 + i;
            cx<R> s[4], sn[4];
            mac_load<R, NB>(s, Sf, rp[0]);
            uint4 rn = rp[2];
            uint2 h = *hp;
            for (int e = e0; e < e1; ++e)
            {
                mac_load<R, NB>(sn, Sf, rn);
                rn = rp[4];
                rp += 2;
                const uint2 hn = *++hp;
                // the target row bits of this cz, as those of cz = 0
                unsigned m = i ? h.y >> 16 : h.y & 0xFFFFu;
                if (m != 0xFFFFu) m = (m >> (2 * cz)) & 0x3333u;
                if (m)
                {
                    cx<R> gv[9];
                    const cx<R>* g9 = Gs + (h.x + 49u * cz) * F + lane;
#pragma unroll
                    for (int d = 0; d < 9; ++d) gv[d] = g9[((d % 3) + 7 * (d / 3)) * F];
                    mac_half<R, 0>(gv, s, acc, m == 0x3333u ? 0xFFFFu : m);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) s[q] = sn[q];
                h = hn;
            }
            if (f < NC)
#pragma unroll
                for (int c = 0; c < 4; ++c)
                {
                    const int t = tgt[8 * (size_t)g + 4 * cz + c];
                    if (t >= 0) ACC[(size_t)t * NC + f] = acc[c];
                }
        }
        else if constexpr (!ALL)
        {
            cx<R> acc0[8], acc1[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) acc0[c] = acc1[c] = zero;
            // the lists end with spare entries, so the reads ahead stay inside
            const uint4* rp = rows + 2 * (size_t)e0;
            uint4 ra = rp[0], rb = rp[1];
            uint2 h = *hp;
            if constexpr (sizeof(R) == 4)
            {
                // source values one half parent ahead, their rows two
                cx<R> s0[4], s1[4];
                mac_load<R, NB>(s0, Sf, ra);
                mac_load<R, NB>(s1, Sf, rb);
                ra = rp[2];
                rb = rp[3];
#pragma unroll 2
                for (int e = e0; e < e1; ++e)
                {
                    cx<R> n0[4], n1[4], gv[9];
                    mac_load<R, NB>(n0, Sf, ra);
                    mac_load<R, NB>(n1, Sf, rb);
                    const cx<R>* g = Gs + h.x * F + lane;
                    const unsigned m0 = h.y & 0xFFFFu, m1 = h.y >> 16;
                    ra = rp[4];
                    rb = rp[5];
                    rp += 2;
                    h = *++hp;
#pragma unroll
                    for (int d = 0; d < 9; ++d) gv[d] = g[((d % 3) + 7 * (d / 3)) * F];
                    mac_half<R, 0>(gv, s0, acc0, m0);
                    mac_half<R, 0>(gv, s1, acc1, m1);
#pragma unroll
                    for (int d = 0; d < 9; ++d) gv[d] = g[((d % 3) + 7 * (d / 3) + 49) * F];
                    mac_half<R, 1>(gv, s0, acc0, m0);
                    mac_half<R, 1>(gv, s1, acc1, m1);
#pragma unroll
                    for (int q = 0; q < 4; ++q) s0[q] = n0[q], s1[q] = n1[q];
                }
            }
            else  // rows one half parent ahead; no registers for more
                for (int e = e0; e < e1; ++e)
                {
                    cx<R> s0[4], s1[4], gv[9];
                    mac_load<R, NB>(s0, Sf, ra);
                    mac_load<R, NB>(s1, Sf, rb);
                    const cx<R>* g = Gs + h.x * F + lane;
                    const unsigned m0 = h.y & 0xFFFFu, m1 = h.y >> 16;
                    rp += 2;
                    ra = rp[0];
                    rb = rp[1];
                    h = *++hp;
#pragma unroll
                    for (int d = 0; d < 9; ++d) gv[d] = g[((d % 3) + 7 * (d / 3)) * F];
                    mac_half<R, 0>(gv, s0, acc0, m0);
                    mac_half<R, 0>(gv, s1, acc1, m1);
#pragma unroll
                    for (int d = 0; d < 9; ++d) gv[d] = g[((d % 3) + 7 * (d / 3) + 49) * F];
                    mac_half<R, 1>(gv, s0, acc0, m0);
                    mac_half<R, 1>(gv, s1, acc1, m1);
                }
            if (f < NC)
#pragma unroll
                for (int c = 0; c < 8; ++c)
                {
                    const int t0 = tgt[8 * (size_t)bg.x + c], t1 = bg.y >= 0 ? tgt[8 * (size_t)bg.y + c] : -1;
                    if (t0 >= 0) ACC[(size_t)t0 * NC + f] = acc0[c];
                    if (t1 >= 0) ACC[(size_t)t1 * NC + f] = acc1[c];
                }
        }
    }
}

// Fused inverse of one target block: z inverse, y inverse, c2r along x and
// target[oct] = scale * window, with every intermediate in shared memory.
// One CTA per (target, half of the NB output z-planes), NB^2 threads:
//   z  thread per pencil (ky, kx): the P accumulators (working precision RA,
//      widened to FP64) -> the NB/2 output planes of this half, into sV
//   y  thread (kx, plane, half of yo): P -> NB/2 outputs yo
//   x  thread (yo, plane, half of xo): c2r NB -> NB/2 outputs xo
// All three passes use one FP64 table sT[k][o] = e^{-2 pi i k (o + NB - 1) / P}
// (conjugated): each pass loops over its input index k and reads row k of
// the table at compile-time offsets, a uniform broadcast read. The inverse
// runs in FP64 on both paths: cancellation in the c2r amplifies FP32
// rounding of the twiddled sums far more than in the forward transforms.
// The summation order per output is the reference order k = 0, 1, ...
template<class RA, int NB>
__global__ void __launch_bounds__(NB * NB, 2) inv_fused_kernel(const cx<RA>* __restrict__ ACC,
                                                               const int* __restrict__ tgt_oct, double scale,
                                                               double* __restrict__ target)
{
    constexpr int P = 2 * NB - 1, NP = P * NB, ZH = NB / 2, S = NB + 1;
    static_assert(NB % 2 == 0, "the block splits into two halves of output planes");
    extern __shared__ __align__(16) unsigned char smraw[];
    double2* sT = reinterpret_cast<double2*>(smraw);  // [k < P][o < NB]
    double2* sV = sT + P * NB;                        // [plane][ky][kx], then [plane][yo][kx] (stride S)
    const int t = blockIdx.x, h = blockIdx.y;
    for (int i = threadIdx.x; i < P * NB; i += blockDim.x)
        sT[i] = ctw<double, P>(((i / NB) * (i % NB + NB - 1)) % P);
    __syncthreads();
    // z: P -> the ZH planes zo = h ZH + i
    const cx<RA>* a = ACC + (size_t)t * P * NP;
    for (int p = threadIdx.x; p < NP; p += blockDim.x)
    {
        double2 acc[ZH];
#pragma unroll
        for (int i = 0; i < ZH; ++i) acc[i] = mk<double>(0, 0);
#pragma unroll 5
        for (int kz = 0; kz < P; ++kz)
        {
            const cx<RA> x0 = a[(size_t)kz * NP + p];
            const double2 x = mk<double>((double)x0.x, (double)x0.y);
            const double2* tr = sT + kz * NB + h * ZH;
#pragma unroll
            for (int i = 0; i < ZH; ++i) cmac_conj<double>(acc[i], x, tr[i]);
        }
#pragma unroll
        for (int i = 0; i < ZH; ++i) sV[i * NP + p] = acc[i];
    }
    __syncthreads();
    // y: thread (kx, plane zl, half yh of the outputs yo)
    const int kx = threadIdx.x % NB, rest = threadIdx.x / NB, zl = rest % ZH, yh = rest / ZH;
    double2 acc[ZH];
#pragma unroll
    for (int i = 0; i < ZH; ++i) acc[i] = mk<double>(0, 0);
#pragma unroll 5
    for (int ky = 0; ky < P; ++ky)
    {
        const double2 x = sV[zl * NP + ky * NB + kx];
        const double2* tr = sT + ky * NB + yh * ZH;
#pragma unroll
        for (int i = 0; i < ZH; ++i) cmac_conj<double>(acc[i], x, tr[i]);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ZH; ++i) sV[(zl * NB + yh * ZH + i) * S + kx] = acc[i];
    __syncthreads();
    // x: thread (yo, plane zl2, half xh of the outputs xo); c2r of the half
    // spectrum: v = Re y_0 + 2 sum_{k >= 1} Re(y_k e^{+2 pi i k (xo + NB - 1) / P})
    const int xh = threadIdx.x / (ZH * NB), r2 = threadIdx.x % (ZH * NB), zl2 = r2 / NB, yo = r2 % NB;
    const double2* yrow = sV + (size_t)(zl2 * NB + yo) * S;
    double sx[ZH];
#pragma unroll
    for (int i = 0; i < ZH; ++i) sx[i] = 0;
#pragma unroll 6
    for (int k = 1; k < NB; ++k)
    {
        const double2 y = yrow[k];
        const double2* tr = sT + k * NB + xh * ZH;
#pragma unroll
        for (int i = 0; i < ZH; ++i) sx[i] = fma(y.x, tr[i].x, fma(y.y, tr[i].y, sx[i]));
    }
    const double y0 = yrow[0].x;
    double* out = target + (size_t)tgt_oct[t] * NB * NB * NB + ((size_t)(h * ZH + zl2) * NB + yo) * NB + xh * ZH;
#pragma unroll
    for (int i = 0; i < ZH; ++i) out[i] = scale * (y0 + 2.0 * sx[i]);
}

template<class R, int NB>
struct Conv
{
    using Real = R;
    static constexpr int Nb = NB;
    static constexpr int P = 2 * NB - 1;
    static constexpr int NP = P * NB;

    static void launch_fwd_xy_rows(Ctx& c, const double* field, const int* d_item_oct, int n, cx<R>* W)
    {
        const int smem = NB * NB * (NB + 1) * (int)sizeof(cx<R>);
        auto kfn = fwd_xy_rows_kernel<R, NB>;
        IBLGF_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        kfn<<<n, NB * NB, smem, c.stream>>>(field, d_item_oct, W);
    }

    static void launch_inverse(Ctx& c, const cx<R>* acc, const int* d_tgt_oct, int n, double scale, double* target)
    {
        const int smem = (P * NB + NB / 2 * NP) * (int)sizeof(double2);
        auto kfn = inv_fused_kernel<R, NB>;
        IBLGF_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        kfn<<<dim3(n, 2), NB * NB, smem, c.stream>>>(acc, d_tgt_oct, scale, target);
    }

    static void forward_field(Ctx& c, const double* field, const int* d_item_oct, int n, void* spec)
    {
        if (!n) return;
        if constexpr (pfa_extent(NB)) forward_pfa(c, field, d_item_oct, n, spec);
        else
        {
            c.grow(c.d_w, (size_t)n * NB * NP * sizeof(cx<R>));
            cx<R>* W = (cx<R>*)c.d_w.p;
            launch_fwd_xy_rows(c, field, d_item_oct, n, W);
            fwd_z_kernel<R, R, NB, NB><<<dim3(n, (NP + 127) / 128), 128, 0, c.stream>>>(W, nullptr, (cx<R>*)spec);
            c.launches += 2;
        }
    }

    // LGF blocks are transformed in FP64 and stored in R
    static void forward_lgf(Ctx& c, const int* d_desc, const int* d_slot, int n, void* spec)
    {
        if (!n) return;
        double2* W = (double2*)c.d_w.p;
        fwd_xy_kernel<NB><<<dim3(n, P), 256, 0, c.stream>>>(d_desc, c.d_lgf_table.p, c.d_tw64.p, W, c.d_ge.p,
                                                            c.ge_stride);
        fwd_z_kernel<double, R, NB, P><<<dim3(n, (NP + 127) / 128), 128, 0, c.stream>>>(W, d_slot,
                                                                                      (cx<R>*)spec);
        c.launches += 2;
    }

    // bytes of a single-block convolution's work buffer
    static constexpr size_t conv_bytes = (size_t)(P + 2 * NB) * NP * sizeof(double2);

    static void conv_block(Ctx& c, const double* src, const double* kernel, double* out, double scale, void* work)
    {
        double2* WK = (double2*)work;
        double2* V = WK + (size_t)P * NP;
        cx<R>* WS = (cx<R>*)(V + (size_t)NB * NP);
        conv_xy_kernel<R, NB><<<P + NB, 256, 0, c.stream>>>(kernel, src, c.d_tw64.p, WK, WS);
        conv_z_kernel<R, NB><<<P, P * NB, 0, c.stream>>>(WK, WS, c.d_tw64.p, V);
        conv_out_kernel<NB><<<NB, NB * NB, 0, c.stream>>>(V, c.d_tw64.p, scale, out);
        c.launches += 3;
    }

    static void mac(Ctx& c, const void* G, const void* S, const int* ptr, const int* src, const int* spec,
                    int n_tgt, void* acc)
    {
        if (!n_tgt) return;
        dim3 grid((unsigned)((c.NC + 127) / 128), n_tgt);
        mac_kernel<R><<<grid, 128, 0, c.stream>>>((const cx<R>*)G, (const cx<R>*)S, ptr, src, spec, c.NC,
                                                  (cx<R>*)acc);
        c.launches += 1;
    }

    static constexpr bool kF32 = std::is_same<R, float>::value;

    template<int NT, int MINB, bool ALL>
    static void group_mac_shape(Ctx& c, const FmmPlan& p, const void* S, void* acc)
    {
        const size_t smem = (size_t)343 * 32 * sizeof(cx<R>) + 344 * sizeof(int);
        auto kfn = bundle_mac_kernel<R, NB, NT, MINB, ALL>;
        IBLGF_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kfn<<<dim3(p.n_mac_tiles, (unsigned)((c.NC + 31) / 32)), NT, smem, c.stream>>>(
            (const cx<R>*)c.d_spec.p, (const cx<R>*)S, (const int4*)p.mac_tile.p, p.spec_u.p, p.mac_ptr.p,
            (const int2*)p.mac_grp.p, (const uint2*)p.mac_head.p, (const uint4*)p.mac_rows.p, p.grp_tgt.p,
            (cx<R>*)acc);
        c.launches += 1;
    }

    // the direct sibling-group MAC: variant 0 = two groups per warp, 1 = half a
    // group per warp
    static void group_mac(Ctx& c, const FmmPlan& p, const void* S, void* acc, int variant)
    {
        if (!p.n_mac_tiles) return;
        if (c.NC != (long long)NB * (2 * NB - 1) * (2 * NB - 1))
            throw Error(IBLGF_EINTERNAL, "spectrum row length differs from the kernel's");
        if (variant == 1)
        {
            if constexpr (kF32) group_mac_shape<512, 2, true>(c, p, S, acc);
            else group_mac_shape<512, 1, true>(c, p, S, acc);
        }
        else
        {
            if constexpr (kF32) group_mac_shape<512, 1, false>(c, p, S, acc);
            else group_mac_shape<384, 1, false>(c, p, S, acc);
        }
    }

    static void inverse(Ctx& c, const void* acc, const int* d_tgt_oct, int n_tgt, double scale, double* target)
    {
        if (!n_tgt) return;
        if constexpr (pfa_extent(NB)) inverse_pfa(c, acc, d_tgt_oct, n_tgt, scale, target);
        else
        {
            launch_inverse(c, (const cx<R>*)acc, d_tgt_oct, n_tgt, scale, target);
            c.launches += 1;
        }
    }
};

template<class F>
void dispatch(Ctx& c, F&& f)
{
    const bool fp32 = c.cfg.precision == IBLGF_FP32;
#define IBLGF_CASE(NBV)                                  \
    case NBV:                                            \
        if (fp32) f(Conv<float, NBV>{});                 \
        else f(Conv<double, NBV>{});                     \
        return;
    switch (c.Nb)
    {
        IBLGF_CASE(6)
        IBLGF_CASE(8)
        IBLGF_CASE(10)
        IBLGF_CASE(12)
        IBLGF_CASE(16)
        IBLGF_CASE(18)
        default: throw Error(IBLGF_EINVAL, "unsupported block_extent (supported: 4,6,8,10,14,16)");
    }
#undef IBLGF_CASE
}

}  // namespace

bool nb_supported(int Nb) { return Nb == 6 || Nb == 8 || Nb == 10 || Nb == 12 || Nb == 16 || Nb == 18; }

void init_twiddle_constants(int device)
{
    static std::mutex m;
    static std::set<int> done;
    std::lock_guard<std::mutex> lock(m);
    if (done.count(device)) return;
    std::vector<double> t64(2 * kTwTotal);
    std::vector<float> t32(2 * kTwTotal);
    for (int P : {11, 15, 19, 23, 31, 35})
        for (int j = 0; j < P; ++j)
        {
            const double a = 2.0 * M_PI * j / P;
            const int k = 2 * (tw_base(P) + j);
            t64[k] = std::cos(a);
            t64[k + 1] = -std::sin(a);
            t32[k] = (float)t64[k];
            t32[k + 1] = (float)t64[k + 1];
        }
    IBLGF_CUDA(cudaMemcpyToSymbol(c_tw64, t64.data(), t64.size() * sizeof(double)));
    IBLGF_CUDA(cudaMemcpyToSymbol(c_tw32, t32.data(), t32.size() * sizeof(float)));
    done.insert(device);
}

void launch_spectra(Ctx& c, const std::vector<std::array<int, 5>>& new_slots)
{
    // new_slots: {slot, ld, bx, by, bz}; processed in batches of 64
    const int P = c.P;
    const size_t wbytes = (size_t)64 * P * P * c.Nb * 16;
    c.grow(c.d_w, wbytes);
    for (size_t b0 = 0; b0 < new_slots.size(); b0 += 64)
    {
        const size_t nb = std::min<size_t>(64, new_slots.size() - b0);
        std::vector<int> desc(4 * nb), slot(nb);
        for (size_t i = 0; i < nb; ++i)
        {
            const auto& s = new_slots[b0 + i];
            slot[i] = s[0];
            desc[4 * i] = s[1];
            desc[4 * i + 1] = s[2];
            desc[4 * i + 2] = s[3];
            desc[4 * i + 3] = s[4];
        }
        DevBuf<int> d_desc, d_slot;
        d_desc.upload(desc, c.stream);
        d_slot.upload(slot, c.stream);
        dispatch(c, [&](auto cv) {
            using CV = decltype(cv);
            CV::forward_lgf(c, d_desc.p, d_slot.p, (int)nb, c.d_spec.p);
        });
        IBLGF_CUDA(cudaGetLastError());
        IBLGF_CUDA(cudaStreamSynchronize(c.stream));  // d_desc / d_slot go out of scope
    }
}

void launch_forward_sources(Ctx& c, const double* fmm_s, const int* d_src_oct, int n_src, void* src_spec)
{
    dispatch(c, [&](auto cv) {
        using CV = decltype(cv);
        CV::forward_field(c, fmm_s, d_src_oct, n_src, src_spec);
    });
    IBLGF_CUDA(cudaGetLastError());
}

// one run of the sibling-group MAC in the given variant: 0, 1 the direct
// kernel with two groups or half a group per warp, 2 the block-Toeplitz kernel,
// 3 the tensor-core kernel
void group_mac_variant(Ctx& c, const FmmPlan& p, const void* src_spec, void* acc, int variant)
{
    if (variant == 2 && toeplitz_mac(c, p, src_spec, acc)) return;
    if (variant == 3 && tc_mac(c, p, src_spec, acc)) return;
    dispatch(c, [&](auto cv) {
        using CV = decltype(cv);
        CV::group_mac(c, p, src_spec, acc, variant);
    });
}

// The MAC autotuner: on a plan's first sweep (outside stream capture) every
// applicable group-MAC variant runs twice on the sweep's real data, the
// second run timed with CUDA events on the context stream; the fastest one
// is kept for the plan (and run last, so that the accumulators hold its
// result). A plan rebuilt for the same (level, mask index) sweep, after an
// adaptation, takes the choice made for its predecessor without re-timing.
// iblgf_mac_variant() can pin a variant instead; a pinned variant that does
// not apply to a plan runs variant 0.
void launch_mac(Ctx& c, const FmmPlan& p, const void* src_spec, void* acc)
{
    dispatch(c, [&](auto cv) {
        using CV = decltype(cv);
        // targets outside sibling groups: general pair-list MAC
        CV::mac(c, c.d_spec.p, src_spec, p.pair_ptr.p, p.pair_src.p, p.pair_spec.p, p.n_csr_tgt, acc);
    });
    if (p.n_tiles)
    {
        const bool ok[4] = {true, true, !p.adj_only && p.tile_combo.p && c.cfg.precision == IBLGF_FP32,
                            tc_mac_ok(c, p)};
        int v = c.mac_variant_forced;
        if (v >= 0 && !ok[v]) v = 0;
        if (v < 0) v = p.mac_variant;
        if (v < 0)
        {
            auto it = c.mac_choice.find({p.level, p.mask_idx});
            if (it != c.mac_choice.end() && ok[it->second]) v = p.mac_variant = it->second;
        }
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        IBLGF_CUDA(cudaStreamIsCapturing(c.stream, &cs));
        if (v < 0 && cs != cudaStreamCaptureStatusNone) v = 0;
        if (v < 0)
        {
            constexpr int nv = 4;
            double ms[nv] = {-1.0, -1.0, -1.0, -1.0};
            cudaEvent_t e0, e1;
            IBLGF_CUDA(cudaEventCreate(&e0));
            IBLGF_CUDA(cudaEventCreate(&e1));
            for (int k = 0; k < nv; ++k)
            {
                if (!ok[k]) continue;
                group_mac_variant(c, p, src_spec, acc, k);
                IBLGF_CUDA(cudaEventRecord(e0, c.stream));
                group_mac_variant(c, p, src_spec, acc, k);
                IBLGF_CUDA(cudaEventRecord(e1, c.stream));
                IBLGF_CUDA(cudaEventSynchronize(e1));
                float t = 0.0f;
                IBLGF_CUDA(cudaEventElapsedTime(&t, e0, e1));
                ms[k] = t;
            }
            cudaEventDestroy(e0);
            cudaEventDestroy(e1);
            int best = 0;
            for (int k = 1; k < nv; ++k)
                if (ok[k] && ms[k] < ms[best]) best = k;
            p.mac_variant = best;
            c.mac_choice[{p.level, p.mask_idx}] = best;
            c.mac_tuning.push_back({(double)p.level, (double)p.mask_idx, (double)p.n_tgt, ms[0], ms[1], ms[2], ms[3],
                                    (double)best});
            v = best;
        }
        group_mac_variant(c, p, src_spec, acc, v);
    }
    IBLGF_CUDA(cudaGetLastError());
}

void launch_inverse_targets(Ctx& c, const FmmPlan& p, const void* acc, double* fmm_t, double scale)
{
    dispatch(c, [&](auto cv) {
        using CV = decltype(cv);
        CV::inverse(c, acc, p.tgt_oct.p, p.n_tgt, scale, fmm_t);
    });
    IBLGF_CUDA(cudaGetLastError());
}

// the work buffer is kept with the context
void launch_conv_block(Ctx& c, const double* src, const double* kernel, double* out, double scale)
{
    const double s = scale / ((double)c.P * c.P * c.P);
    dispatch(c, [&](auto cv) {
        using CV = decltype(cv);
        if (c.conv_work.n < CV::conv_bytes) c.conv_work.alloc(CV::conv_bytes);
        CV::conv_block(c, src, kernel, out, s, c.conv_work.p);
    });
    IBLGF_CUDA(cudaGetLastError());
    IBLGF_CUDA(cudaStreamSynchronize(c.stream));
}

// ---------------------------------------------------------------------------
// Single-block convolution without any device allocation. The work buffer of
// launch_conv_block lives instead in one file-scope device array of
// kNoAllocScratchBytes (2 MiB); the largest supported block (Nb = 18) needs
// 0.72 MB of it.
//
// Who needs it: a host application that has already reserved the device
// memory for its own block pool, or that calls the solve from a section in
// which it must not allocate — cudaMalloc can fail there, and cudaFree
// synchronises the whole device, which stalls every other stream the
// application keeps busy. The context (twiddles) is created beforehand as
// usual; this call itself performs no cudaMalloc, cudaFree or library
// allocation, and it enqueues on the context stream without synchronising.
//
// Limits: the scratch is one array per device, shared by every context and
// stream of that device, so calls that overlap in time on different streams
// race on it; serialise them (one stream, or a host lock). The first call on a
// device looks up the symbol's address, so make it before any stream capture
// begins. No scratch byte needs to start at zero: every byte a kernel reads is
// written earlier in the same call.
constexpr size_t kNoAllocScratchBytes = size_t(2) << 20;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

namespace
{
constexpr int kNoAllocMaxDevices = 64;
unsigned char* g_noalloc_ptr[kNoAllocMaxDevices] = {};
std::mutex g_noalloc_mutex;

// Makes the context's device current for the scope of a call and restores
// the caller's current device on every way out (return or exception).
struct DeviceScope
{
    int prev = -1;
    explicit DeviceScope(int device)
    {
        IBLGF_CUDA(cudaGetDevice(&prev));
        if (prev != device) IBLGF_CUDA(cudaSetDevice(device));
    }
    ~DeviceScope()
    {
        int cur = -1;
        if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev);
    }
};

// the static scratch's device address on the current device (set up once
// per device); the caller holds a DeviceScope for the context's device
unsigned char* noalloc_scratch()
{
    int dev = -1;
    IBLGF_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kNoAllocMaxDevices) throw Error(IBLGF_EINVAL, "device ordinal beyond the scratch table");
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev])
    {
        void* ptr = nullptr;
        IBLGF_CUDA(cudaGetSymbolAddress(&ptr, g_noalloc_scratch));
        if (!ptr) throw Error(IBLGF_ECUDA, "cudaGetSymbolAddress returned a null scratch address");
        g_noalloc_ptr[dev] = static_cast<unsigned char*>(ptr);
    }
    return g_noalloc_ptr[dev];
}
}  // namespace

void launch_conv_block_noalloc(Ctx& c, const double* src, const double* kernel, double* out, double scale)
{
    DeviceScope on_device(c.cfg.device);
    unsigned char* work = noalloc_scratch();
    const double s = scale / ((double)c.P * c.P * c.P);
    dispatch(c, [&](auto cv) {
        using CV = decltype(cv);
        static_assert(CV::conv_bytes <= kNoAllocScratchBytes, "every supported block fits the static scratch");
        CV::conv_block(c, src, kernel, out, s, work);
    });
    IBLGF_CUDA(cudaGetLastError());
}

}  // namespace iblgf_b200
