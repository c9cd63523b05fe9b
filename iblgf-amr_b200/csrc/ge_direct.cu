// Direct evaluation of the integrating factor's neighbour sweep.
//
// Contract: the neighbour-only FMM sweep with the LGF_GE kernel
// (fmm.hpp:754-770, poisson.hpp:436-494) gives every target block T
//     out_T(i) = sum over the source blocks S among T's 27 neighbours,
//                sum over the interior nodes j of S:  E(x_i - x_j) f_S(j),
// E(n) = e^{-6a} I_n1(2a) I_n2(2a) I_n3(2a) = g(n1) g(n2) g(n3) with
// g(m) = e^{-2a} I_m(2a) (lgf_ge.hpp:158-175). The reference forms it with
// block FFT convolutions; here it is summed directly, which is exact up to
// the terms with some |n_k| > R: the host takes the smallest R in kGeRs
// with g(m) <= 2^-56 g(0) for every m > R, i.e. every dropped term lies
// below FP64 rounding of the result (g(m) / g(0) ~ a^m / m!: the IF-HERK
// steps' integrating factors, a ~ 5e-4 .. 2e-2, take R = 4 .. 8), or no term
// is dropped at all (2 Nb - 4 is the largest distance from a target node to a
// neighbour's interior), and the transform path when none qualifies.
//
// A cell of the 27-neighbourhood lies in the interior of one block only, so a
// source position s in [-R, Nb - 1 + R] per axis (target node 0 at s = 0)
// names one block and one of its interior nodes. Two CTAs per target block,
// halves of its z planes:
//   z  thread per (qy, qx) column: the half's H + 2R values, read from the up
//      to 3 blocks they lie in (consecutive lanes read consecutive x), to H
//      outputs in shared memory [z][qy][qx]
//   x  thread per (z, qy, half of x): in the rows, both halves read before
//      either is written
//   y  thread per (z, half of y, x): columns, written to the target with
//      consecutive lanes along x
// All arithmetic FP64 (both precision paths).
#include <algorithm>

#include "ctx.hpp"

namespace iblgf_b200
{
namespace
{
constexpr int kGeRs[5] = {4, 6, 8, 12, 16};

template<int NB, int R>
struct GeShape
{
    static constexpr int Q = NB + 2 * R;  // region extent per axis
    static constexpr int H = NB / 2;      // output planes per CTA, outputs per thread
    static constexpr int S = Q | 1;       // row stride in shared memory (odd: no bank conflicts)
    static constexpr int W = 2 * R + 1;
    static constexpr int K = H + 2 * R;   // inputs of H outputs
    static constexpr size_t smem = (size_t)H * Q * S * sizeof(double);
};

struct GeFields
{
    const double* src[3];
    double* dst[3];
};

// mode 0: dst += scale * out, 1: dst = scale * out (blocks without a source: 0)
template<int NB, int R>
__global__ void __launch_bounds__(256) ge_direct_kernel(const __grid_constant__ GeFields f, const int* __restrict__ ge_tgt,
                                                        const int* __restrict__ ge_src,
                                                        const double* __restrict__ gtab, double scale, int assign)
{
    using G = GeShape<NB, R>;
    constexpr int Q = G::Q, H = G::H, S = G::S, W = G::W, K = G::K, E = NB - 2;
    extern __shared__ double sb[];  // [H][Q][S]
    __shared__ int src[27];
    const int tid = threadIdx.x;
    const double* __restrict__ fs = f.src[blockIdx.z];
    double* __restrict__ out = f.dst[blockIdx.z] + (size_t)ge_tgt[blockIdx.x] * NB * NB * NB;
    const int z0 = blockIdx.y * H;
    int any = 0;
    if (tid < 27)
    {
        src[tid] = ge_src[(size_t)blockIdx.x * 27 + tid];
        any = src[tid] >= 0;
    }
    double e[R + 1];  // e[|m|]
#pragma unroll
    for (int m = 0; m <= R; ++m) e[m] = gtab[m];
    if (!__syncthreads_or(any))
    {
        if (assign)
            for (int i = tid; i < H * NB * NB; i += blockDim.x) out[z0 * NB * NB + i] = 0.0;
        return;
    }
    // z: region cell s - 1 of an axis relative to the target's interior; the
    // neighbour it lies in is o, its node there s - E o, in 1 .. E
    for (int c = tid; c < Q * Q; c += blockDim.x)
    {
        const int qy = c / Q, qx = c % Q, sy = qy - R, sx = qx - R;
        const int oy = sy < 1 ? -1 : (sy > E ? 1 : 0), ox = sx < 1 ? -1 : (sx > E ? 1 : 0);
        const int jy = sy - E * oy, jx = sx - E * ox;
        const bool in = jy >= 1 && jy <= E && jx >= 1 && jx <= E;
        const double* col[3];
#pragma unroll
        for (int o = 0; o < 3; ++o)
        {
            const int b = src[(ox + 1) + 3 * (oy + 1) + 9 * o];
            col[o] = in && b >= 0 ? fs + (size_t)b * NB * NB * NB + jy * NB + jx : nullptr;
        }
        double a[K];
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
            const int sz = z0 + k - R;
            const int oz = sz < 1 ? -1 : (sz > E ? 1 : 0), jz = sz - E * oz;
            const double* p = oz < 0 ? col[0] : (oz > 0 ? col[2] : col[1]);
            a[k] = p && jz >= 1 && jz <= E ? __ldg(p + jz * NB * NB) : 0.0;
        }
#pragma unroll
        for (int z = 0; z < H; ++z)
        {
            double b = 0.0;
#pragma unroll
            for (int m = 0; m < W; ++m) b = fma(e[m < R ? R - m : m - R], a[z + m], b);
            sb[(z * Q + qy) * S + qx] = b;
        }
    }
    __syncthreads();
    // x: all inputs of a pass are read before any output of the rows is written
    for (int it0 = 0; it0 < H * Q * 2; it0 += blockDim.x)
    {
        // a row's two halves are neighbouring work items: an even number of
        // threads keeps both in the same pass
        const int it = it0 + tid, row = it >> 1, h = it & 1;
        double b[H];
        if (it < H * Q * 2)
        {
            double a[K];
#pragma unroll
            for (int k = 0; k < K; ++k) a[k] = sb[row * S + h * H + k];
#pragma unroll
            for (int x = 0; x < H; ++x)
            {
                b[x] = 0.0;
#pragma unroll
                for (int m = 0; m < W; ++m) b[x] = fma(e[m < R ? R - m : m - R], a[x + m], b[x]);
            }
        }
        __syncwarp();
        if (it < H * Q * 2)
#pragma unroll
            for (int x = 0; x < H; ++x) sb[row * S + h * H + x] = b[x];
    }
    __syncthreads();
    // y, into the target
    for (int it = tid; it < H * 2 * NB; it += blockDim.x)
    {
        const int x = it % NB, h = (it / NB) & 1, z = it / (2 * NB);
        double a[K];
#pragma unroll
        for (int k = 0; k < K; ++k) a[k] = sb[(z * Q + h * H + k) * S + x];
        double* o = out + ((size_t)(z0 + z) * NB + h * H) * NB + x;
#pragma unroll
        for (int y = 0; y < H; ++y)
        {
            double b = 0.0;
#pragma unroll
            for (int m = 0; m < W; ++m) b = fma(e[m < R ? R - m : m - R], a[y + m], b);
            if (assign) o[y * NB] = scale * b;
            else o[y * NB] += scale * b;
        }
    }
}
template<int NB, int R>
void launch_ge_nb(Ctx& c, const GeFields& f, int n, const int* tgt, const int* src, int n_tgt, const double* gtab,
                  double scale, bool assign)
{
    using G = GeShape<NB, R>;
    auto kfn = ge_direct_kernel<NB, R>;
    IBLGF_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::smem));
    kfn<<<dim3((unsigned)n_tgt, 2, n), 256, G::smem, c.stream>>>(f, tgt, src, gtab, scale, assign ? 1 : 0);
    c.launches += 1;
    IBLGF_CUDA(cudaGetLastError());
}

template<int NB>
void launch_ge_r(Ctx& c, const GeFields& f, int n, const int* tgt, const int* src, int n_tgt, const double* gtab,
                 double scale, bool assign, int R)
{
    switch (R)
    {
        case 4: launch_ge_nb<NB, 4>(c, f, n, tgt, src, n_tgt, gtab, scale, assign); return;
        case 6: launch_ge_nb<NB, 6>(c, f, n, tgt, src, n_tgt, gtab, scale, assign); return;
        case 8: launch_ge_nb<NB, 8>(c, f, n, tgt, src, n_tgt, gtab, scale, assign); return;
        case 12: launch_ge_nb<NB, 12>(c, f, n, tgt, src, n_tgt, gtab, scale, assign); return;
        default: launch_ge_nb<NB, 16>(c, f, n, tgt, src, n_tgt, gtab, scale, assign); return;
    }
}

// the truncation radius of table ge: the smallest R in kGeRs beyond which
// the 1-D factor is negligible or no neighbour node lies, 0 if none
int ge_direct_radius(const Ctx& c, int ge)
{
    if (ge < 0) return 0;
    if (c.Nb != 6 && c.Nb != 8 && c.Nb != 10 && c.Nb != 12 && c.Nb != 16 && c.Nb != 18) return 0;
    const double* f = c.ge_host.data() + (size_t)ge * c.ge_stride;
    for (int R : kGeRs)
    {
        if (R >= 2 * c.Nb - 4) return R;
        if (c.ge_stride <= R + 1) return 0;
        bool ok = true;
        for (int m = R + 1; m < c.ge_stride && ok; ++m) ok = std::fabs(f[m]) <= std::ldexp(std::fabs(f[0]), -56);
        if (ok) return R;
    }
    return 0;
}
}  // namespace

bool ge_direct_ok(const Ctx& c, int ge) { return ge_direct_radius(c, ge) > 0; }

void launch_ge_direct(Ctx& c, const int* tgt, const int* src, int n_tgt, const double* const* from, double* const* to,
                      int n, int ge, double scale, bool assign)
{
    if (!n_tgt || n < 1) return;
    const int R = ge_direct_radius(c, ge);
    if (!R) throw Error(IBLGF_EINTERNAL, "the integrating factor does not allow the direct sweep");
    const double* gtab = c.d_ge.p + (size_t)ge * c.ge_stride;
    GeFields f{};
    for (int k = 0; k < n; ++k)
    {
        f.src[k] = from[k];
        f.dst[k] = to[k];
    }
#define IBLGF_GE(NBV)                                                             \
    case NBV:                                                                     \
        launch_ge_r<NBV>(c, f, n, tgt, src, n_tgt, gtab, scale, assign, R);       \
        return;
    switch (c.Nb)
    {
        IBLGF_GE(6)
        IBLGF_GE(8)
        IBLGF_GE(10)
        IBLGF_GE(12)
        IBLGF_GE(16)
        IBLGF_GE(18)
        default: throw Error(IBLGF_EINVAL, "unsupported block size");
    }
#undef IBLGF_GE
}
}  // namespace iblgf_b200
