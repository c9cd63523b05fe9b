// Inverse transform of the accumulated spectra of one FMM sweep, assigned to
// the targets (Convolution::apply_backward + dfft_c2r::execute + add_solution,
// include/iblgf/utilities/convolution.hpp:232-304, src/utilities/
// convolution.cpp:151-238): per target, c2r of the P^3 half spectrum,
// window [Nb-1, 2Nb-2]^3 scaled into the Nb^3 target block (each target has one
// inverse per sweep).
//
// B200 structure: a cluster of two CTAs per target. CTA h owns the kx half
// [h Nb/2, (h+1) Nb/2) of the half spectrum, so every accumulated value is
// read from HBM once:
//   z  thread per (ky, kx) pencil: P frequencies -> the Nb window planes
//   y  thread per (plane, kx) column: P -> the Nb window rows
//   x  thread per (plane, row): this CTA's kx half of the c2r sum, all Nb
//      outputs (a partial sum)
// then each CTA adds its half of the planes, own partial plus the peer's
// read through distributed shared memory (always rank 0's partial first, so
// the result does not depend on timing), into the target.
// The forward transform of the source blocks (dfft_r2c::execute of the
// zero-padded block, convolution.cpp:107-119) runs in one kernel, a cluster of
// two CTAs per source. CTA h owns the kx half in the x and y passes and half of
// the (ky, kx) pencils, in their order in memory, in the z pass:
//   x  thread per (z, y) row: real Nb inputs -> the half's Nb/2 frequencies
//   y  thread per (z, kx) column: Nb -> P, in shared memory
//   z  thread per pencil, its inputs from the shared memory of the CTA that
//      owns its kx: Nb -> P, to the spectrum in full rows
// so that only the block and its spectrum cross HBM (two kernels with the x/y
// intermediate in between moved half as much again), and every store of a warp
// is contiguous. Bound by the FP32 (FP64) pipe and shared memory. The 11649
// sources of an FP32 solve on three levels (extent 16) take 0.78 ms; two kernels
// with prime-factor passes took 1.14, one kernel that keeps the kx halves in the
// z pass 1.9 (its stores cover 72 of each 144 bytes). The inverse of as many
// targets: 1.02 -> 0.74 ms with the short transforms' symmetry (below).
//
// The z and y passes use the prime-factor (Good-Thomas) algorithm for
// P = N1 N2 with coprime N1, N2 (35 = 5 x 7, 15 = 3 x 5): with input
// n = (N2 n1 + N1 n2) mod P and output k, e^{2 pi i n k / P} =
// e^{2 pi i n1 (k mod N1) / N1} e^{2 pi i n2 (k mod N2) / N2}, so
//     X[k] = sum_n2 W_N2^{n2 (k mod N2)} T_n2[k mod N1],
//     T_n2[k1] = sum_n1 W_N1^{n1 k1} x[N2 n1 + N1 n2 mod P],
// N2 short DFTs of length N1 and N1 of length N2, with no twiddle
// multiplications. The short DFTs of odd length N pair inputs j and N - j and
// outputs k and N - k,
//     C_k = x_0 + sum_j (x_j + x_{N-j}) cos(2 pi j k / N),
//     S_k =       sum_j (x_j - x_{N-j}) sin(2 pi j k / N),
//     X_k = C_k +- i S_k, X_{N-k} = C_k -+ i S_k,
// half the multiplications of the direct sums. Zero inputs (forward: n >= Nb)
// and outputs outside the window (inverse) are left out. A forward pencil takes
// about 500 FMAs or additions instead of 2520, an inverse one about 560 instead
// of 960, and sums of 5 and 7 terms round less than sums of 18 and 35. All loops
// are unrolled, so every root of unity is a compile-time-indexed constant-bank
// operand.
#include <cooperative_groups.h>

#include <type_traits>

#include "cplx.cuh"
#include "ctx.hpp"

namespace cg = cooperative_groups;

namespace iblgf_b200
{
namespace
{
// roots of unity e^{+2 pi i j / N} for N in {3, 5, 7} and the c2r roots
// e^{+2 pi i j / P} for P in {15, 35}
constexpr int kPfaTw = 3 + 5 + 7;
__constant__ double c_pfa64[2 * kPfaTw];
__constant__ float c_pfa32[2 * kPfaTw];
__constant__ double c_c2r64[2 * (15 + 35)];
__constant__ float c_c2r32[2 * (15 + 35)];

__host__ __device__ constexpr int pfa_base(int N) { return N == 3 ? 0 : (N == 5 ? 3 : 8); }
__host__ __device__ constexpr int c2r_base(int P) { return P == 15 ? 0 : 15; }

template<class R, int N>
__device__ __forceinline__ cx<R> wroot(int j)
{
    if constexpr (std::is_same<R, double>::value)
        return mk<R>(c_pfa64[2 * (pfa_base(N) + j)], c_pfa64[2 * (pfa_base(N) + j) + 1]);
    else
        return mk<R>(c_pfa32[2 * (pfa_base(N) + j)], c_pfa32[2 * (pfa_base(N) + j) + 1]);
}

// e^{+2 pi i j / P}
template<class R, int P>
__device__ __forceinline__ cx<R> c2r_root(int j)
{
    const int i = 2 * (c2r_base(P) + j);
    if constexpr (std::is_same<R, double>::value) return mk<R>(c_c2r64[i], c_c2r64[i + 1]);
    else return mk<R>(c_c2r32[i], c_c2r32[i + 1]);
}

template<int NB>
struct Pfa
{
    static constexpr int P = 2 * NB - 1;
    static constexpr int N1 = P == 35 ? 5 : 3;
    static constexpr int N2 = P == 35 ? 7 : 5;
    static_assert(P == 35 || P == 15, "prime-factor split of 15 or 35");
};

template<class R>
__device__ __forceinline__ cx<R> cadd(const cx<R>& a, const cx<R>& b)
{
    return mk<R>(a.x + b.x, a.y + b.y);
}
template<class R>
__device__ __forceinline__ cx<R> csub(const cx<R>& a, const cx<R>& b)
{
    return mk<R>(a.x - b.x, a.y - b.y);
}
// c + s i d for s = +1 or -1
template<class R, int SGN>
__device__ __forceinline__ cx<R> cadd_i(const cx<R>& c, const cx<R>& d)
{
    return SGN > 0 ? mk<R>(c.x - d.y, c.y + d.x) : mk<R>(c.x + d.y, c.y - d.x);
}

// short DFT of odd length N, X_k = sum_j v_j e^{SGN 2 pi i j k / N}; only the
// outputs of the bit set NEED are formed and handed to put(k, X_k)
template<class R, int N, int SGN, unsigned NEED, class Put>
__device__ __forceinline__ void short_dft(const cx<R> (&v)[N], Put&& put)
{
    constexpr int H = N / 2;
    cx<R> a[H], b[H];
#pragma unroll
    for (int j = 0; j < H; ++j)
    {
        a[j] = cadd<R>(v[j + 1], v[N - 1 - j]);
        b[j] = csub<R>(v[j + 1], v[N - 1 - j]);
    }
    if (NEED & 1u)
    {
        cx<R> s = v[0];
#pragma unroll
        for (int j = 0; j < H; ++j) s = cadd<R>(s, a[j]);
        put(0, s);
    }
#pragma unroll
    for (int k = 1; k <= H; ++k)
    {
        if (!((NEED >> k | NEED >> (N - k)) & 1u)) continue;
        cx<R> C = v[0], S = mk<R>(0, 0);
#pragma unroll
        for (int j = 1; j <= H; ++j)
        {
            const cx<R> w = wroot<R, N>((j * k) % N);
            C.x = fma(a[j - 1].x, w.x, C.x);
            C.y = fma(a[j - 1].y, w.x, C.y);
            S.x = fma(b[j - 1].x, w.y, S.x);
            S.y = fma(b[j - 1].y, w.y, S.y);
        }
        if (NEED >> k & 1u) put(k, cadd_i<R, SGN>(C, S));
        if (NEED >> (N - k) & 1u) put(N - k, cadd_i<R, -SGN>(C, S));
    }
}

// output k of P = N1 N2 with k mod N1 = k1, k mod N2 = k2
template<int NB>
__host__ __device__ constexpr int pfa_k(int k1, int k2)
{
    using PF = Pfa<NB>;
    int k = k1;
    while (k % PF::N2 != k2) k += PF::N1;
    return k;
}
// k2 of the window outputs k in [NB - 1, 2 NB - 2] with k mod N1 = k1
template<int NB>
__host__ __device__ constexpr unsigned pfa_window(int k1)
{
    unsigned m = 0;
    for (int k2 = 0; k2 < Pfa<NB>::N2; ++k2)
    {
        const int k = pfa_k<NB>(k1, k2);
        if (k >= NB - 1 && k <= 2 * NB - 2) m |= 1u << k2;
    }
    return m;
}

// inverse pencil: x(i) loads input i (i < P), put(o, value) takes the window
// output k = o + NB - 1
template<class R, int NB, int K1, class Put>
__device__ __forceinline__ void pfa_inverse_k1(const cx<R> (&T)[Pfa<NB>::N1][Pfa<NB>::N2], Put&& put)
{
    short_dft<R, Pfa<NB>::N2, 1, pfa_window<NB>(K1)>(
        T[K1], [&](int k2, const cx<R>& v) { put(pfa_k<NB>(K1, k2) - (NB - 1), v); });
    if constexpr (K1 + 1 < Pfa<NB>::N1) pfa_inverse_k1<R, NB, K1 + 1>(T, put);
}

template<class R, int NB, class Load, class Put>
__device__ __forceinline__ void pfa_inverse(Load&& x, Put&& put)
{
    using PF = Pfa<NB>;
    constexpr int P = PF::P, N1 = PF::N1, N2 = PF::N2;
    cx<R> T[N1][N2];
#pragma unroll
    for (int n2 = 0; n2 < N2; ++n2)
    {
        cx<R> v[N1];
#pragma unroll
        for (int n1 = 0; n1 < N1; ++n1) v[n1] = x((N2 * n1 + N1 * n2) % P);
        short_dft<R, N1, 1, (1u << N1) - 1>(v, [&](int k1, const cx<R>& t) { T[k1][n2] = t; });
    }
    pfa_inverse_k1<R, NB, 0>(T, put);
}

// forward pencil of the NB inputs v (the other P - NB are zero): put(k, X_k) for
// every k < P. The residues k1 and N1 - k1 are formed together: T = C +- i S as
// in short_dft, over the inputs that are there.
template<class R, int NB, class Put>
__device__ __forceinline__ void pfa_forward(const cx<R> (&v)[NB], Put&& put)
{
    using PF = Pfa<NB>;
    constexpr int P = PF::P, N1 = PF::N1, N2 = PF::N2;
#pragma unroll
    for (int k1 = 0; k1 <= N1 / 2; ++k1)
    {
        cx<R> T[N2], U[N2];  // residues k1 and N1 - k1
#pragma unroll
        for (int n2 = 0; n2 < N2; ++n2)
        {
            cx<R> C = mk<R>(0, 0), S = mk<R>(0, 0);
#pragma unroll
            for (int n1 = 0; n1 < N1; ++n1)
            {
                const int n = (N2 * n1 + N1 * n2) % P;
                if (n >= NB) continue;
                const int j = (n1 * k1) % N1;
                if (j == 0)
                {
                    C = cadd<R>(C, v[n]);
                    continue;
                }
                const cx<R> w = wroot<R, N1>(j);
                C.x = fma(v[n].x, w.x, C.x);
                C.y = fma(v[n].y, w.x, C.y);
                S.x = fma(v[n].x, w.y, S.x);
                S.y = fma(v[n].y, w.y, S.y);
            }
            T[n2] = k1 ? cadd_i<R, -1>(C, S) : C;
            U[n2] = cadd_i<R, 1>(C, S);
        }
        short_dft<R, N2, -1, (1u << N2) - 1>(T, [&](int k2, const cx<R>& x) { put(pfa_k<NB>(k1, k2), x); });
        if (k1)
            short_dft<R, N2, -1, (1u << N2) - 1>(U, [&](int k2, const cx<R>& x) { put(pfa_k<NB>(N1 - k1, k2), x); });
    }
}

// x pass of CTA half H: partial c2r over kx in [H NB/2, (H+1) NB/2) of one
// row y[kx] (local index), v(xo) = sum w_kx Re(y e^{+2 pi i kx (xo+NB-1)/P}),
// w = 1 for kx = 0, 2 otherwise
template<class R, int NB, int H>
__device__ __forceinline__ void c2r_half(const cx<R>* yrow, double (&out)[NB])
{
    constexpr int P = 2 * NB - 1, KH = NB / 2;
#pragma unroll
    for (int o = 0; o < NB; ++o) out[o] = 0.0;
#pragma unroll
    for (int j = 0; j < KH; ++j)
    {
        const int kx = H * KH + j;
        const cx<R> yv = yrow[j];
        const double yr = (double)yv.x * (kx ? 2.0 : 1.0), yi = (double)yv.y * (kx ? 2.0 : 1.0);
#pragma unroll
        for (int o = 0; o < NB; ++o)
        {
            const int idx = (kx * (o + NB - 1)) % P;
            const double c = c_c2r64[2 * (c2r_base(P) + idx)], s = c_c2r64[2 * (c2r_base(P) + idx) + 1];
            out[o] = fma(yr, c, fma(-yi, s, out[o]));
        }
    }
}

// shared memory: V [NB planes][P][KH] complex (z output, then y output in
// the first NB rows of each plane) and the x-pass partials [NB][NB][NB]
template<class R, int NB>
struct InvSmem
{
    static constexpr int P = 2 * NB - 1, KH = NB / 2;
    static constexpr size_t v = (size_t)NB * P * KH * sizeof(cx<R>);
    static constexpr size_t part = (size_t)NB * NB * NB * sizeof(double);
    static constexpr size_t total = v + part;
};

template<class R, int NB>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NB* NB)
    inv_pfa_kernel(const cx<R>* __restrict__ ACC, const int* __restrict__ tgt_oct, double scale,
                   double* __restrict__ target)
{
    constexpr int P = 2 * NB - 1, KH = NB / 2, NP = P * NB;
    using SM = InvSmem<R, NB>;
    extern __shared__ __align__(16) unsigned char smraw[];
    cx<R>* V = reinterpret_cast<cx<R>*>(smraw);                    // [zo][ky][kxl]
    double* part = reinterpret_cast<double*>(smraw + SM::v);         // [zo][yo][xo]
    cg::cluster_group cluster = cg::this_cluster();
    const int h = (int)cluster.block_rank();
    const int t = blockIdx.x / 2;

    // z: pencil (ky, kxl); the accumulator is [kz][ky][kx]
    {
        const int p = threadIdx.x;
        if (p < P * KH)
        {
            const int ky = p / KH, kxl = p % KH;
            const cx<R>* a = ACC + (size_t)t * P * NP + (size_t)ky * NB + h * KH + kxl;
            pfa_inverse<R, NB>([&](int kz) { return a[(size_t)kz * NP]; },
                               [&](int o, const cx<R>& v) { V[(o * P + ky) * KH + kxl] = v; });
        }
    }
    __syncthreads();
    // y: column (zo, kxl), outputs written over the column's first NB rows
    {
        const int q = threadIdx.x;
        if (q < NB * KH)
        {
            const int zo = q / KH, kxl = q % KH;
            cx<R>* col = V + (size_t)zo * P * KH + kxl;
            cx<R> out[NB];
            pfa_inverse<R, NB>([&](int ky) { return col[(size_t)ky * KH]; },
                               [&](int o, const cx<R>& v) { out[o] = v; });
#pragma unroll
            for (int o = 0; o < NB; ++o) col[(size_t)o * KH] = out[o];
        }
    }
    __syncthreads();
    // x: row (zo, yo), partial c2r over this CTA's kx half
    {
        const int zo = threadIdx.x / NB, yo = threadIdx.x % NB;
        const cx<R>* yrow = V + ((size_t)zo * P + yo) * KH;
        double out[NB];
        if (h == 0) c2r_half<R, NB, 0>(yrow, out);
        else c2r_half<R, NB, 1>(yrow, out);
        double* prow = part + ((size_t)zo * NB + yo) * NB;
#pragma unroll
        for (int o = 0; o < NB; ++o) prow[o] = out[o];
    }
    cluster.sync();  // both partials complete
    {
        const double* p0 = h == 0 ? part : cluster.map_shared_rank(part, 0);
        const double* p1 = h == 1 ? part : cluster.map_shared_rank(part, 1);
        double* out = target + (size_t)tgt_oct[t] * NB * NB * NB;
        const int base = h * (NB / 2) * NB * NB;
        for (int i = threadIdx.x; i < (NB / 2) * NB * NB; i += blockDim.x)
            out[base + i] = scale * (p0[base + i] + p1[base + i]);
    }
    cluster.sync();  // the peer has read this CTA's partials
}

// half spectra of the listed field blocks (item i -> spectrum row i)
template<class R, int NB>
struct FwdSmem
{
    static constexpr int P = 2 * NB - 1, KH = NB / 2, S = KH | 1;  // odd row stride: no bank conflicts
    static constexpr size_t x1 = (size_t)NB * NB * S * sizeof(cx<R>);  // [z][y][kxl]
    static constexpr size_t w = (size_t)NB * P * KH * sizeof(cx<R>);   // [z][ky][kxl]
    static constexpr size_t total = x1 + w;
    static_assert(NB % 2 == 0 && (size_t)NB * NB * (NB + 1) * sizeof(R) <= w, "the block is staged in W");
};

template<class R, int NB, int H>
__device__ __forceinline__ void fwd_row(const R* row, cx<R>* dst)
{
    constexpr int P = 2 * NB - 1, KH = NB / 2;
    R in[NB];
#pragma unroll
    for (int x = 0; x < NB; ++x) in[x] = row[x];
#pragma unroll
    for (int j = 0; j < KH; ++j)
    {
        cx<R> s = mk<R>(0, 0);
#pragma unroll
        for (int x = 0; x < NB; ++x)
        {
            const int idx = ((H * KH + j) * x) % P;
            const cx<R> w = c2r_root<R, P>(idx);
            s.x = fma(in[x], w.x, s.x);
            s.y = fma(in[x], -w.y, s.y);
        }
        dst[j] = s;
    }
}

template<class R, int NB>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NB* NB)
    fwd_pfa_kernel(const double* __restrict__ field, const int* __restrict__ item_oct, cx<R>* __restrict__ spec)
{
    constexpr int P = 2 * NB - 1, KH = NB / 2, NP = P * NB;
    using SM = FwdSmem<R, NB>;
    extern __shared__ __align__(16) unsigned char smraw[];
    cx<R>* X = reinterpret_cast<cx<R>*>(smraw);
    cx<R>* W = reinterpret_cast<cx<R>*>(smraw + SM::x1);
    cg::cluster_group cluster = cg::this_cluster();
    const int item = blockIdx.x / 2, h = (int)cluster.block_rank(), t = threadIdx.x;
    {
        // the block in rows of odd stride, in the memory of W
        R* in = reinterpret_cast<R*>(W);
        const double2* blk = reinterpret_cast<const double2*>(field + (size_t)item_oct[item] * (NB * NB * NB));
#pragma unroll
        for (int k = 0; k < NB / 2; ++k)
        {
            const int i = k * NB * NB + t;
            const double2 v = blk[i];
            const int at = 2 * i / NB * (NB + 1) + 2 * i % NB;
            in[at] = (R)v.x;
            in[at + 1] = (R)v.y;
        }
        __syncthreads();
        const R* row = in + (size_t)t * (NB + 1);
        if (h == 0) fwd_row<R, NB, 0>(row, X + (size_t)t * SM::S);
        else fwd_row<R, NB, 1>(row, X + (size_t)t * SM::S);
    }
    __syncthreads();
    if (t < NB * KH)
    {
        const int z = t / KH, kxl = t % KH;
        cx<R> v[NB];
#pragma unroll
        for (int y = 0; y < NB; ++y) v[y] = X[(z * NB + y) * SM::S + kxl];
        cx<R>* out = W + (size_t)z * P * KH + kxl;
        pfa_forward<R, NB>(v, [&](int k, const cx<R>& x) { out[(size_t)k * KH] = x; });
    }
    cluster.sync();  // both halves of W are there
    if (t < P * KH)
    {
        const int p = h * P * KH + t, ky = p / NB, kx = p % NB;
        const cx<R>* w = cluster.map_shared_rank(W, kx / KH) + (size_t)ky * KH + kx % KH;
        cx<R> v[NB];
#pragma unroll
        for (int z = 0; z < NB; ++z) v[z] = w[(size_t)z * P * KH];
        cx<R>* out = spec + (size_t)item * P * NP + p;
        pfa_forward<R, NB>(v, [&](int k, const cx<R>& x) { out[(size_t)k * NP] = x; });
    }
    cluster.sync();  // the peer has read this CTA's half
}

template<class R, int NB>
void launch_fwd_pfa(Ctx& c, const double* field, const int* d_item_oct, int n, void* spec)
{
    using SM = FwdSmem<R, NB>;
    auto kfn = fwd_pfa_kernel<R, NB>;
    IBLGF_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SM::total));
    kfn<<<2 * n, NB * NB, SM::total, c.stream>>>(field, d_item_oct, (cx<R>*)spec);
    c.launches += 1;
}

template<class R, int NB>
void launch_inv_pfa(Ctx& c, const void* acc, const int* d_tgt_oct, int n, double scale, double* target)
{
    using SM = InvSmem<R, NB>;
    auto kfn = inv_pfa_kernel<R, NB>;
    IBLGF_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SM::total));
    kfn<<<2 * n, NB * NB, SM::total, c.stream>>>((const cx<R>*)acc, d_tgt_oct, scale, target);
    c.launches += 1;
}
}  // namespace

void init_pfa_constants(int device)
{
    (void)device;
    double t64[2 * kPfaTw];
    float t32[2 * kPfaTw];
    for (int N : {3, 5, 7})
        for (int j = 0; j < N; ++j)
        {
            const double a = 2.0 * M_PI * j / N;
            t64[2 * (pfa_base(N) + j)] = std::cos(a);
            t64[2 * (pfa_base(N) + j) + 1] = std::sin(a);
        }
    for (int i = 0; i < 2 * kPfaTw; ++i) t32[i] = (float)t64[i];
    double c2r[2 * (15 + 35)];
    for (int P : {15, 35})
        for (int j = 0; j < P; ++j)
        {
            const double a = 2.0 * M_PI * j / P;
            c2r[2 * (c2r_base(P) + j)] = std::cos(a);
            c2r[2 * (c2r_base(P) + j) + 1] = std::sin(a);
        }
    IBLGF_CUDA(cudaMemcpyToSymbol(c_pfa64, t64, sizeof(t64)));
    IBLGF_CUDA(cudaMemcpyToSymbol(c_pfa32, t32, sizeof(t32)));
    float c2r32[2 * (15 + 35)];
    for (int i = 0; i < 2 * (15 + 35); ++i) c2r32[i] = (float)c2r[i];
    IBLGF_CUDA(cudaMemcpyToSymbol(c_c2r64, c2r, sizeof(c2r)));
    IBLGF_CUDA(cudaMemcpyToSymbol(c_c2r32, c2r32, sizeof(c2r32)));
}

// The z and y passes run in the sweep's precision; the c2r stage and the sum over
// the two kx halves are FP64. On the 3-level Gaussian workload the FP32 path is
// 2.15e-6 (relative L-inf) from the FP64 oracle; when the passes' type was chosen,
// FP32 passes gave 4.8e-6 and 1.89 ms of inverse per solve, FP64 passes 1.4e-7 and
// 2.53 ms, direct 35-term FP32 sums 1.16e-5.
void inverse_pfa(Ctx& c, const void* acc, const int* d_tgt_oct, int n, double scale, double* target)
{
    const bool f32 = c.cfg.precision == IBLGF_FP32;
    if (c.Nb == 18 && f32) launch_inv_pfa<float, 18>(c, acc, d_tgt_oct, n, scale, target);
    else if (c.Nb == 18) launch_inv_pfa<double, 18>(c, acc, d_tgt_oct, n, scale, target);
    else if (f32) launch_inv_pfa<float, 8>(c, acc, d_tgt_oct, n, scale, target);
    else launch_inv_pfa<double, 8>(c, acc, d_tgt_oct, n, scale, target);
}

void forward_pfa(Ctx& c, const double* field, const int* d_item_oct, int n, void* spec)
{
    const bool f32 = c.cfg.precision == IBLGF_FP32;
    if (c.Nb == 18 && f32) launch_fwd_pfa<float, 18>(c, field, d_item_oct, n, spec);
    else if (c.Nb == 18) launch_fwd_pfa<double, 18>(c, field, d_item_oct, n, spec);
    else if (f32) launch_fwd_pfa<float, 8>(c, field, d_item_oct, n, spec);
    else launch_fwd_pfa<double, 8>(c, field, d_item_oct, n, spec);
}

}  // namespace iblgf_b200
