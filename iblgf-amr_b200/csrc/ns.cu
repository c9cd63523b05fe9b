// Field kernels of the IF-HERK time step (FP64, whole component fields):
//   clean3_kernel    Ifherk::clean (ifherk.hpp:1309-1352): zero whole blocks,
//                    or with non_leaf_only only the outer `width` planes of
//                    leaves and all of every other block
//   axpby3_kernel    Ifherk::copy / add (ifherk.hpp:1878-1960), over every
//                    node including buffers
//   lincomb_kernel   the sums of two fields that the stages form by a copy and
//                    an add, in one pass (3 field passes instead of 5)
//   smooth_kernel    Operator::smooth2zero (operators.hpp:653-760) as called
//                    by clean_leaf_correction_boundary (ifherk.hpp:1383-1404):
//                    each listed (block, neighbour direction) multiplies the
//                    block by the tanh taper towards that face / edge / corner,
//                    `reps` times in a row (once per component of the field)
#include <algorithm>
#include <cmath>

#include "ctx.hpp"

namespace iblgf_b200
{
namespace
{
// up to three component fields per launch (blockIdx.y = component)
struct Fields3
{
    double* to[3];
    const double* from[3];
};

template<int NB>
__global__ void clean3_kernel(const __grid_constant__ Fields3 f, const int* __restrict__ leaf, int non_leaf_only, int w)
{
    constexpr int N3 = NB * NB * NB;
    const int o = blockIdx.x;
    double* b = f.to[blockIdx.y] + (size_t)o * N3;
    const bool shell = non_leaf_only && leaf[o];
    for (int i = threadIdx.x; i < N3; i += blockDim.x)
    {
        if (shell)
        {
            const int x = i % NB, y = (i / NB) % NB, z = i / (NB * NB);
            if (x >= w && y >= w && z >= w && x < NB - w && y < NB - w && z < NB - w) continue;
        }
        b[i] = 0.0;
    }
}

// mode 0: to = a * from; 1: to += a * from (per component); n16 16-byte pairs
__global__ void axpby3_kernel(const __grid_constant__ Fields3 f, double a, size_t n16, int mode)
{
    double2* __restrict__ to = reinterpret_cast<double2*>(f.to[blockIdx.y]);
    const double2* __restrict__ from = reinterpret_cast<const double2*>(f.from[blockIdx.y]);
#pragma unroll 4
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n16; i += (size_t)gridDim.x * blockDim.x)
    {
        const double2 v = from[i];
        if (mode == 0) to[i] = make_double2(v.x * a, v.y * a);
        else
        {
            const double2 w = to[i];
            to[i] = make_double2(w.x + v.x * a, w.y + v.y * a);
        }
    }
}

// mode 0: to = x + y * a; 1: to = (x - y) * a. to may be x.
struct LinComb3
{
    double* to[3];
    const double* x[3];
    const double* y[3];
};
__global__ void lincomb_kernel(const __grid_constant__ LinComb3 f, double a, size_t n16, int mode)
{
    double2* to = reinterpret_cast<double2*>(f.to[blockIdx.y]);
    const double2* x = reinterpret_cast<const double2*>(f.x[blockIdx.y]);
    const double2* __restrict__ y = reinterpret_cast<const double2*>(f.y[blockIdx.y]);
#pragma unroll 4
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n16; i += (size_t)gridDim.x * blockDim.x)
    {
        const double2 u = x[i], v = y[i];
        if (mode == 0) to[i] = make_double2(u.x + v.x * a, u.y + v.y * a);
        else to[i] = make_double2((u.x - v.x) * a, (u.y - v.y) * a);
    }
}

double taper(double x)
{
    const double fac = 10.0, shift = 0.2;
    const double c = 1.0 - (0.5 + 0.5 * std::tanh(fac * (1.0 - shift)));
    return (0.5 + 0.5 * std::tanh(fac * (x - shift))) + c;
}

// taper(i / (NB-1)), taper(1 - i / (NB-1)): local_pct over the block with its
// buffer (node.hpp:121-124)
struct Tapers
{
    double lo[18], hi[18];
};

// entries [ptr[b], ptr[b+1]) of block list[b]: neighbour directions (0..26).
// The taper takes 2 NB distinct values (node index i from the low or the high
// side), evaluated on the host. Up to 26 directions times reps dependent
// multiplications per node: a block is split over blockIdx.y (kSmoothNodes per
// thread) and the components over blockIdx.z; one CTA per block and component,
// with the 2 NB tanh in each, took 123 us for the 112 outer base blocks of the
// vortex ring.
constexpr int kSmoothNodes = 2;

template<int NB>
__global__ void __launch_bounds__(256) smooth_kernel(const __grid_constant__ Fields3 fs, const int* __restrict__ list,
                                                     const int* __restrict__ ptr, const int* __restrict__ dirs,
                                                     int reps, const __grid_constant__ Tapers tp)
{
    constexpr int N3 = NB * NB * NB;
    __shared__ double tlo[NB], thi[NB];
    __shared__ int s_dir[27];
    const int e0 = ptr[blockIdx.x], ne = ptr[blockIdx.x + 1] - e0;
    if (threadIdx.x < NB)
    {
        tlo[threadIdx.x] = tp.lo[threadIdx.x];
        thi[threadIdx.x] = tp.hi[threadIdx.x];
    }
    if (threadIdx.x < ne && threadIdx.x < 27) s_dir[threadIdx.x] = dirs[e0 + threadIdx.x];
    __syncthreads();
    double* b = fs.to[blockIdx.z] + (size_t)list[blockIdx.x] * N3;
    for (int k = 0; k < kSmoothNodes; ++k)
    {
        const int i = (blockIdx.y * kSmoothNodes + k) * 256 + threadIdx.x;
        if (i >= N3) return;
        const int ix = i % NB, iy = (i / NB) % NB, iz = i / (NB * NB);
        double v = b[i];
        for (int e = 0; e < ne; ++e)
        {
            const int d = s_dir[e], x = d % 3, y = (d / 3) % 3, z = d / 9;
            double sq = 0.0;
            int cnt = 0;
            if (z == 0) sq = fmax(sq, tlo[iz]), ++cnt;
            else if (z == 2) sq = fmax(sq, thi[iz]), ++cnt;
            if (y == 0) sq = fmax(sq, tlo[iy]), ++cnt;
            else if (y == 2) sq = fmax(sq, thi[iy]), ++cnt;
            if (x == 0) sq = fmax(sq, tlo[ix]), ++cnt;
            else if (x == 2) sq = fmax(sq, thi[ix]), ++cnt;
            if (cnt > 0)
                for (int r = 0; r < reps; ++r) v *= sq;
        }
        b[i] = v;
    }
}

template<class F>
void nb_switch(int Nb, F&& f)
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

void launch_clean_vf(Ctx& c, double* const* f, int n, const int* d_leaf, bool non_leaf_only, int width)
{
    if (!c.n_oct || n < 1 || n > 3) return;
    Fields3 p{};
    for (int k = 0; k < n; ++k) p.to[k] = f[k];
    nb_switch(c.Nb, [&](auto nbc) {
        constexpr int NB = decltype(nbc)::value;
        clean3_kernel<NB><<<dim3(c.n_oct, n), 256, 0, c.stream>>>(p, d_leaf, non_leaf_only ? 1 : 0, width);
    });
    c.launches += 1;
    IBLGF_CUDA(cudaGetLastError());
}

void launch_axpby_vf(Ctx& c, double* const* to, const double* const* from, int n, double a, int mode)
{
    const size_t pairs = c.field_elems() / 2;  // Nb is even
    if (!pairs || n < 1 || n > 3) return;
    Fields3 p{};
    for (int k = 0; k < n; ++k)
    {
        p.to[k] = to[k];
        p.from[k] = from[k];
    }
    const unsigned grid = (unsigned)std::min<size_t>((pairs + 255) / 256, 148 * 16 / n);
    axpby3_kernel<<<dim3(grid, n), 256, 0, c.stream>>>(p, a, pairs, mode);
    c.launches += 1;
    IBLGF_CUDA(cudaGetLastError());
}

void launch_lincomb_vf(Ctx& c, double* const* to, const double* const* x, const double* const* y, int n, double a,
                       int mode)
{
    const size_t pairs = c.field_elems() / 2;
    if (!pairs || n < 1 || n > 3) return;
    LinComb3 p{};
    for (int k = 0; k < n; ++k)
    {
        p.to[k] = to[k];
        p.x[k] = x[k];
        p.y[k] = y[k];
    }
    const unsigned grid = (unsigned)std::min<size_t>((pairs + 255) / 256, 148 * 16 / n);
    lincomb_kernel<<<dim3(grid, n), 256, 0, c.stream>>>(p, a, pairs, mode);
    c.launches += 1;
    IBLGF_CUDA(cudaGetLastError());
}

void launch_smooth_vf(Ctx& c, double* const* f, int m, const int* list, const int* ptr, const int* dirs, int n,
                      int reps)
{
    if (!n || m < 1 || m > 3) return;
    Fields3 p{};
    for (int k = 0; k < m; ++k) p.to[k] = f[k];
    Tapers tp{};
    for (int i = 0; i < c.Nb; ++i)
    {
        const double pc = (double)i / (c.Nb - 1);
        tp.lo[i] = taper(pc);
        tp.hi[i] = taper(1.0 - pc);
    }
    nb_switch(c.Nb, [&](auto nbc) {
        constexpr int NB = decltype(nbc)::value, per = 256 * kSmoothNodes;
        smooth_kernel<NB>
            <<<dim3(n, (NB * NB * NB + per - 1) / per, m), 256, 0, c.stream>>>(p, list, ptr, dirs, reps, tp);
    });
    c.launches += 1;
    IBLGF_CUDA(cudaGetLastError());
}

}  // namespace iblgf_b200
