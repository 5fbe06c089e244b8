// Cube-diagonal preconditioner: set-up on the host, application on the device (precond.hpp).
#include "precond.hpp"
#include "lane8.cuh"

#include <algorithm>
#include <cmath>
#include <complex>
#include <vector>

namespace a43g {

namespace {

// eigenvalues lam[k] and eigenvectors V[i][k] of a symmetric 4x4 matrix (cyclic Jacobi rotations)
void jacobi4(double const (&A0)[4][4], double (&lam)[4], double (&V)[4][4]) {
    double A[4][4];
    for (int i = 0; i < 4; ++i)
        for (int j = 0; j < 4; ++j) { A[i][j] = A0[i][j]; V[i][j] = (i == j) ? 1.0 : 0.0; }
    for (int sweep = 0; sweep < 50; ++sweep) {
        double off = 0;
        for (int i = 0; i < 4; ++i)
            for (int j = i + 1; j < 4; ++j) off += A[i][j]*A[i][j];
        if (off < 1e-30) break;
        for (int p = 0; p < 4; ++p)
            for (int q = p + 1; q < 4; ++q) {
                if (A[p][q] == 0.0) continue;
                double const theta = (A[q][q] - A[p][p])/(2*A[p][q]);
                double const t = (theta >= 0 ? 1.0 : -1.0)/(std::fabs(theta) + std::sqrt(theta*theta + 1));
                double const c = 1/std::sqrt(t*t + 1), s = t*c;
                for (int k = 0; k < 4; ++k) {            // A = J^T A J
                    double const akp = A[k][p], akq = A[k][q];
                    A[k][p] = c*akp - s*akq; A[k][q] = s*akp + c*akq;
                }
                for (int k = 0; k < 4; ++k) {
                    double const apk = A[p][k], aqk = A[q][k];
                    A[p][k] = c*apk - s*aqk; A[q][k] = s*apk + c*aqk;
                }
                for (int k = 0; k < 4; ++k) {
                    double const vkp = V[k][p], vkq = V[k][q];
                    V[k][p] = c*vkp - s*vkq; V[k][q] = s*vkp + c*vkq;
                }
            }
    }
    for (int k = 0; k < 4; ++k) lam[k] = A[k][k];
}

// the finite-difference weights of the distances 0..3 inside a cube (8th or 16th order) times
// the direction's prefactor -1/(2 h^2); zero where the direction has no kinetic term
void fd_weights(KineticLists const &kl, double (&w)[4]) {
    double const w8[4] = {-14350, 8064, -1008, 128}, w16[4] = {-924708642, 538137600, -94174080, 22830080};
    for (int k = 0; k < 4; ++k) w[k] = 0;
    if (kl.FD_range >= 8) for (int k = 0; k < 4; ++k) w[k] = kl.prefactor*w16[k]/302702400.;
    else if (kl.FD_range >= 1) for (int k = 0; k < 4; ++k) w[k] = kl.prefactor*w8[k]/5040.;
}

template <typename T> struct QOf;
template <> struct QOf<double> { using type = PrecondQ; };
template <> struct QOf<float> { using type = PrecondQf; };

// A warp takes 16 lanes of columns of a block (8 bytes each: one column in FP64, two in FP32), its
// halves the planes re and im; a lane holds all 64 points of its columns in registers, so that the
// 4-point transforms along x, y and z need no exchange, and only the complex scaling takes the other
// plane's values from the partner lane.  Everything is read before anything is written: y may be x.
//
// Measured on 4,096 blocks: FP32 58 us (4.6 TB/s), FP64 135 us (4.0 TB/s), against 73 and 136 us with a
// CTA per half block, the z-transform through shared memory and four barriers.  What bounds it: the
// 128 registers of the points leave 8 warps per SM, whose loads and transforms overlap little.
template <typename T>
__global__ void __launch_bounds__(128, 2)
k_precond(T *y, T const *x, uint32_t nnzb, int32_t const *__restrict__ veff, uint32_t ncells,
          T const *__restrict__ tab, uint16_t const *__restrict__ colindx, uint32_t nsrc_pair,
          uint8_t const *__restrict__ active, typename QOf<T>::type const Q)
{
    using V = typename LaneOf<T>::V;
    constexpr int W = 8/int(sizeof(T)), S = 64/W, NG = S/16;   // columns per lane, lanes per point, groups
    __shared__ V qs[3][2][4][4];                     // [direction][Q, transposed][row][column]
    uint64_t const item = uint64_t(blockIdx.x)*4 + (threadIdx.x >> 5);
    uint32_t const b = uint32_t(item/NG), group = uint32_t(item % NG);
    bool const mine = item < uint64_t(nnzb)*NG;
    uint32_t const s = mine ? colindx[b] : 0u;
    bool const work = mine && (!active || active[s]);   // uniform over the warp
    if (!__syncthreads_or(work)) return;
    if (threadIdx.x < 48) {
        int const d = threadIdx.x >> 4, i = (threadIdx.x >> 2) & 3, k = threadIdx.x & 3;
        V const q = vdup(T(Q.q[d][i][k]));
        qs[d][0][i][k] = q; qs[d][1][k][i] = q;
    }
    __syncthreads();
    if (!work) return;
    int const lane = threadIdx.x & 31, pl = lane >> 4;
    size_t const o = size_t(b)*8192 + pl*4096 + group*16*W + (lane & 15)*W;
    V const *xb = reinterpret_cast<V const*>(x + o);
    V v[64];
#pragma unroll
    for (int p = 0; p < 64; ++p) v[p] = xb[p*S];
    int32_t const cell = veff[b];
    T const *d = tab + ((size_t(s/nsrc_pair)*(ncells + 1) + (cell < 0 ? ncells : uint32_t(cell)))*64)*2;
    // out[k] = sum_i M[k][i] in[i] along one direction, M = Q^T (forward) or Q (back)
    auto transform = [&](V const (&M)[4][4], int stride) {
        V m[4][4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int i = 0; i < 4; ++i) m[k][i] = M[k][i];
#pragma unroll
        for (int p = 0; p < 64; ++p) {
            if ((p/stride) & 3) continue;            // first point of each line
            V t[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                t[k] = vmul(m[k][0], v[p]);
#pragma unroll
                for (int i = 1; i < 4; ++i) t[k] = vfma(m[k][i], v[p + i*stride], t[k]);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) v[p + k*stride] = t[k];
        }
    };
    transform(qs[0][1], 1);
    transform(qs[1][1], 4);
    transform(qs[2][1], 16);
#pragma unroll
    for (int p = 0; p < 64; ++p) {
        T const dr = __ldg(d + 2*p), di = __ldg(d + 2*p + 1);
        V const w = __shfl_xor_sync(0xffffffffu, v[p], 16);
        v[p] = vfma(v[p], vdup(dr), vmul(w, vdup(pl ? di : -di)));
    }
    transform(qs[2][0], 16);
    transform(qs[1][0], 4);
    transform(qs[0][0], 1);
    V *yb = reinterpret_cast<V*>(y + o);
#pragma unroll
    for (int p = 0; p < 64; ++p) yb[p*S] = v[p];
}

} // namespace

namespace {
bool upload_tables(BlockPreconditioner &pc, std::vector<double> const &t64, std::vector<float> const &t32,
                   cudaStream_t st) {
    size_t const n = t64.size();
    A43G_CUDA_TRY(cudaMemcpyAsync(pc.tab64.ptr, t64.data(), n*8, cudaMemcpyHostToDevice, st));
    A43G_CUDA_TRY(cudaMemcpyAsync(pc.tab32.ptr, t32.data(), n*4, cudaMemcpyHostToDevice, st));
    A43G_CUDA_TRY(cudaStreamSynchronize(st));      // the host tables go out of scope
    return true;
}
} // namespace

int precond_setup(GreenPlan const &hp, DevicePlan const &dp, BlockPreconditioner &pc, cudaStream_t st) {
    (void)dp;
    double lam[3][4];
    for (int d = 0; d < 3; ++d) {
        double w[4];
        fd_weights(hp.kinetic[d], w);
        double A[4][4], V[4][4];
        for (int i = 0; i < 4; ++i)
            for (int k = 0; k < 4; ++k) A[i][k] = w[i > k ? i - k : k - i];
        jacobi4(A, lam[d], V);
        for (int i = 0; i < 4; ++i)
            for (int k = 0; k < 4; ++k) { pc.Q.q[d][i][k] = V[i][k]; pc.Qf.q[d][i][k] = float(V[i][k]); }
    }
    uint32_t const ncells = uint32_t(hp.ncells());
    uint32_t const npairs = std::max(1u, hp.npairs);
    pc.ncells = ncells; pc.npairs = npairs;
    pc.nsrc_pair = (hp.npairs > 1) ? hp.nsrc_pair : std::max(1u, hp.nCols);
    std::vector<double> vbar(size_t(ncells) + 1, 0.0);
    for (uint32_t c = 0; c < ncells && hp.Vcell.size() >= size_t(ncells)*64; ++c) {
        double sum = 0;
        for (int p = 0; p < 64; ++p) sum += hp.Vcell[size_t(c)*64 + p];
        vbar[c] = sum/64;
    }
    size_t const n = size_t(npairs)*(ncells + 1)*64*2;
    std::vector<double> t64(n);
    std::vector<float> t32(n);
    for (uint32_t pr = 0; pr < npairs; ++pr) {
        double const Er = (hp.npairs > 1) ? hp.pair_E[2*pr] : hp.E_re;
        double const Ei = (hp.npairs > 1) ? hp.pair_E[2*pr + 1] : hp.E_im;
        for (uint32_t c = 0; c <= ncells; ++c)
            for (int z = 0; z < 4; ++z)
                for (int yy = 0; yy < 4; ++yy)
                    for (int xx = 0; xx < 4; ++xx) {
                        int const p = (z*4 + yy)*4 + xx;
                        std::complex<double> const den(lam[2][z] + lam[1][yy] + lam[0][xx] + vbar[c] - Er, -Ei);
                        std::complex<double> const v = (0.0 == std::abs(den)) ? std::complex<double>(INFINITY, 0) : 1.0/den;
                        if (!std::isfinite(v.real()) || !std::isfinite(v.imag()) ||
                            !std::isfinite(float(v.real())) || !std::isfinite(float(v.imag()))) {
                            set_error("preconditioner: the cube model is singular at this energy "
                                      "(a real energy on one of its eigenvalues)");
                            return A43G_ERR_ARGUMENT;
                        }
                        size_t const o = ((size_t(pr)*(ncells + 1) + c)*64 + p)*2;
                        t64[o] = v.real(); t64[o + 1] = v.imag();
                        t32[o] = float(v.real()); t32[o + 1] = float(v.imag());
                    }
    }
    if (!pc.tab64.alloc(n*8) || !pc.tab32.alloc(n*4)) return A43G_ERR_MEMORY;
    return upload_tables(pc, t64, t32, st) ? A43G_OK : A43G_ERR_CUDA;
}

template <typename T>
bool precond_apply(DevicePlan const &dp, BlockPreconditioner const &pc, T *y, T const *x, uint8_t const *active,
                   cudaStream_t st) {
    if (0 == dp.nnzb) return true;
    // four warps per CTA, each with 16 lanes of columns of a block
    unsigned const grid = unsigned((uint64_t(dp.nnzb)*(sizeof(T)/2) + 3)/4);
    T const *tab = (sizeof(T) == 8) ? reinterpret_cast<T const*>(pc.tab64.ptr) : reinterpret_cast<T const*>(pc.tab32.ptr);
    if constexpr (sizeof(T) == 8)
        k_precond<double><<<grid, 128, 0, st>>>(y, x, dp.nnzb, dptr<int32_t>(dp.veff_index), pc.ncells, tab,
                                                dptr<uint16_t>(dp.colindx), pc.nsrc_pair, active, pc.Q);
    else
        k_precond<float><<<grid, 128, 0, st>>>(y, x, dp.nnzb, dptr<int32_t>(dp.veff_index), pc.ncells, tab,
                                               dptr<uint16_t>(dp.colindx), pc.nsrc_pair, active, pc.Qf);
    count_launch();
    A43G_CUDA_TRY(cudaGetLastError());
    return true;
}

template bool precond_apply<double>(DevicePlan const &, BlockPreconditioner const &, double *, double const *,
                                    uint8_t const *, cudaStream_t);
template bool precond_apply<float>(DevicePlan const &, BlockPreconditioner const &, float *, float const *,
                                   uint8_t const *, cudaStream_t);

} // namespace a43g
