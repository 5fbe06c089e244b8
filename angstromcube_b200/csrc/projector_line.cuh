// Projection of the action on the CUDA cores (include/green_dyadic.hxx:112-288), FP32 and FP64,
// sum-factorized along the lines of cubes of an atom image.
//
// The projector functions are separable on the spherical mask,
//     P_(ix,iy,iz)(x, y, z) = H_ix(x) H_iy(y) H_iz(z)   for points inside the projection radius,
// and so is the whole sphere: all cubes of one x-line share H_iy(y) and H_iz(z), all lines of one
// z-slab of cubes share H_iz(z).  The x-contraction therefore accumulates over a whole line
// before the y-contraction is done once per line, and the z-contraction once per slab: with about
// 6 cubes per line and 36 per slab a block costs 64(L+1) + 16 N2/6 + 4 nSHO/36 multiply-adds per
// column (about 450 at L = 5, N2 = (L+1)(L+2)/2) instead of 64(L+1) + 16 N2 + 4 nSHO (944) when every
// block is contracted by itself, and 3584 for the dense product.
#pragma once

#include "device.cuh"

namespace a43g {
namespace line {

constexpr int kThreads = 128;         // 4 warps: warp z works on z-plane z of every cube

__host__ __device__ constexpr int nsho_of(int L) { return ((L + 1)*(L + 2)*(L + 3))/6; }
__host__ __device__ constexpr int n2_of(int L) { return ((L + 1)*(L + 2))/2; }

// 8 bytes per lane: one column in FP64, two neighbouring columns in FP32 (fma.rn.f32x2: one issue
// slot for both, each rounded as a scalar fma)
template <typename T> struct LaneOf;
template <> struct LaneOf<double> { using V = double; static constexpr int quarters = 4; };
template <> struct LaneOf<float> { using V = unsigned long long; static constexpr int quarters = 2; };

__device__ __forceinline__ double vfma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ unsigned long long vfma(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ double vadd(double a, double b) { return a + b; }
__device__ __forceinline__ unsigned long long vadd(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
template <typename V> struct alignas(16) Pair { V a, b; };

// element of a block ([2][64 points][64 columns]) at point 0, and of a coefficient row ([2][64]),
// that lane `lane` of quarter q works on
template <typename T> __device__ __forceinline__ int block_lane(int q, int lane) {
    return (sizeof(T) == 8) ? (q >> 1)*4096 + (q & 1)*32 + lane : q*4096 + 2*lane;
}
template <typename T> __device__ __forceinline__ int row_lane(int q, int lane) {
    return (sizeof(T) == 8) ? (q >> 1)*64 + (q & 1)*32 + lane : q*64 + 2*lane;
}

__device__ __forceinline__ uint32_t smem_u32(void const *p) { return uint32_t(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void copy16(void *dst, void const *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }

// N table values (consecutive, 16-byte aligned, stored to an even count)
template <typename V, int N> __device__ __forceinline__ void load_row(V (&h)[N], V const *p) {
#pragma unroll
    for (int i = 0; i < N; i += 2) {
        Pair<V> const t = *reinterpret_cast<Pair<V> const*>(p + i);
        h[i] = t.a;
        if (i + 1 < N) h[i + 1] = t.b;
    }
}

// ---------------------------------------------------------------- projection

// One work item: `count` consecutive positions of the block list of (image, source), each with a
// record {block, slot, mask}.  CTA = (item, quarter of the 128 columns): warp z takes z-plane z of
// every cube, a lane one 8-byte lane of columns, and the four warps meet only at the end of the
// item.  The points go from global memory straight to registers (each is used by one thread only,
// so staging them in shared memory would share nothing): as soon as the four points of one x are
// consumed, the same points of the next cube are requested into their registers.  Rows outside the
// sphere are not loaded; planes that the sphere cuts test each point (uniform over the warp).  The
// x- and y-tables of all cubes of the item are staged in shared memory once.
//
// What a thread carries (ax: 4(L+1), byx: N2, 16 points) fits 168 registers, so three CTAs share an
// SM.  Measured on the 64-atom cell with 8 sources (32,768 blocks, 155,000 (block, image) pairs),
// against one contraction per block staged through shared memory: FP32 1.14 -> 0.74 ms, FP64
// 2.83 -> 1.34 ms.  What bounds it: the FP64 pipe is busy 36 % of the time and issue slots 44 %;
// the atoms of that cell lie near its faces, where an image is a fragment with lines of 3 cubes.
template <typename T, int L, int LP>
__device__ __forceinline__ void project_item(T *__restrict__ apc, T const *__restrict__ x, uint32_t nrhs,
                                             PrjItem const &it, uint4 const *__restrict__ recs,
                                             typename LaneOf<T>::V const *__restrict__ tab, T *__restrict__ part,
                                             uint32_t *__restrict__ tickets, unsigned char *smem)
{
    using V = typename LaneOf<T>::V;
    constexpr int NS = nsho_of(L), N2 = n2_of(L), TS = 12*LP, TXY = 8*LP;
    constexpr int S = 64*int(sizeof(T))/8;                      // lanes of 8 bytes per point
    int const tid = threadIdx.x, zq = tid >> 5, lane = tid & 31, quarter = blockIdx.y;
    V *acc = reinterpret_cast<V*>(smem) + zq*NS*32 + lane;      // [4][NS][32] sums of the four planes
    V *tb = reinterpret_cast<V*>(smem) + 4*NS*32;               // [kMaxPrjItem][TXY] x- and y-tables
    uint4 *rec = reinterpret_cast<uint4*>(tb + kMaxPrjItem*TXY);
    int const count = int(it.count);
    for (int i = tid; i < count; i += kThreads) rec[i] = recs[it.first + i];
    __syncthreads();
    for (int q = tid; q < count*(TXY/2); q += kThreads) {       // 16-byte copies
        int const k = q/(TXY/2), o = (q - k*(TXY/2))*2;
        copy16(tb + k*TXY + o, tab + size_t(rec[k].y & kSlotMask)*TS + o);
    }
    copy_commit();
#pragma unroll
    for (int i = 0; i < NS; ++i) acc[i*32] = V(0);

    T const *xl = x + block_lane<T>(quarter, lane) + zq*1024;
    auto plane_mask = [&](int k) -> uint32_t {
        uint32_t const w = (zq & 2) ? rec[k].w : rec[k].z;
        return (zq & 1) ? (w >> 16) : (w & 0xffffu);
    };
    auto block = [&](int k) { return reinterpret_cast<V const*>(xl + size_t(rec[k].x)*8192); };
    V ax[4][L + 1], byx[N2], v[16];
#pragma unroll
    for (int i = 0; i < N2; ++i) byx[i] = V(0);
#pragma unroll
    for (int y = 0; y < 4; ++y)
#pragma unroll
        for (int i = 0; i <= L; ++i) ax[y][i] = V(0);
    uint32_t m = 0;
    if (count > 0) {
        m = plane_mask(0);
        V const *p = block(0);
#pragma unroll
        for (int y = 0; y < 4; ++y)
            if ((m >> (4*y)) & 0xfu) {
#pragma unroll
                for (int xx = 0; xx < 4; ++xx) v[4*y + xx] = __ldg(p + (4*y + xx)*S);
            }
    }
    copy_wait<0>();
    __syncthreads();                                            // the tables have landed
    for (int k = 0; k < count; ++k) {
        uint32_t const flags = rec[k].y;
        bool const last = (k + 1 == count);
        uint32_t const mn = last ? 0u : plane_mask(k + 1);
        V const *p = block(last ? k : k + 1);
        bool const r0 = mn & 0x000fu, r1 = mn & 0x00f0u, r2 = mn & 0x0f00u, r3 = mn & 0xf000u;
        V const *t = tb + k*TXY;
        if (0xffffu == m) {
#pragma unroll
            for (int xx = 0; xx < 4; ++xx) {
                V h[L + 1];
                load_row(h, t + xx*LP);
#pragma unroll
                for (int y = 0; y < 4; ++y)
#pragma unroll
                    for (int ix = 0; ix <= L; ++ix) ax[y][ix] = vfma(v[4*y + xx], h[ix], ax[y][ix]);
                if (r0) v[xx] = __ldg(p + xx*S);
                if (r1) v[4 + xx] = __ldg(p + (4 + xx)*S);
                if (r2) v[8 + xx] = __ldg(p + (8 + xx)*S);
                if (r3) v[12 + xx] = __ldg(p + (12 + xx)*S);
            }
        } else {
#pragma unroll
            for (int xx = 0; xx < 4; ++xx) {
                V h[L + 1];
                load_row(h, t + xx*LP);
#pragma unroll
                for (int y = 0; y < 4; ++y)
                    if (m & (1u << (4*y + xx))) {
#pragma unroll
                        for (int ix = 0; ix <= L; ++ix) ax[y][ix] = vfma(v[4*y + xx], h[ix], ax[y][ix]);
                    }
                if (r0) v[xx] = __ldg(p + xx*S);
                if (r1) v[4 + xx] = __ldg(p + (4 + xx)*S);
                if (r2) v[8 + xx] = __ldg(p + (8 + xx)*S);
                if (r3) v[12 + xx] = __ldg(p + (12 + xx)*S);
            }
        }
        m = mn;
        if ((flags & kLineEnd) || last) {
#pragma unroll
            for (int y = 0; y < 4; ++y) {
                V h[L + 1];
                load_row(h, t + (4 + y)*LP);
#pragma unroll
                for (int iy = 0, i = 0; iy <= L; ++iy)
#pragma unroll
                    for (int ix = 0; ix <= L - iy; ++ix, ++i) byx[i] = vfma(ax[y][ix], h[iy], byx[i]);
#pragma unroll
                for (int ix = 0; ix <= L; ++ix) ax[y][ix] = V(0);
            }
        }
        if ((flags & kSlabEnd) || last) {
            V h[L + 1];
            V const *tz = tab + size_t(flags & kSlotMask)*TS + (8 + zq)*LP;
#pragma unroll
            for (int iz = 0; iz <= L; ++iz) h[iz] = __ldg(tz + iz);
#pragma unroll
            for (int iz = 0, sho = 0; iz <= L; ++iz)
#pragma unroll
                for (int iy = 0; iy <= L - iz; ++iy)
#pragma unroll
                    for (int ix = 0; ix <= L - iz - iy; ++ix, ++sho)
                        acc[sho*32] = vfma(byx[iy*(2*L + 3 - iy)/2 + ix], h[iz], acc[sho*32]);
#pragma unroll
            for (int i = 0; i < N2; ++i) byx[i] = V(0);
        }
    }
    __syncthreads();
    // warp z adds the planes' sums of the coefficients sho = z (mod 4), in the order of the planes
    V const *sum = reinterpret_cast<V const*>(smem) + lane;
    auto total = [&](int sho) {
        return vadd(vadd(vadd(sum[sho*32], sum[(NS + sho)*32]), sum[(2*NS + sho)*32]), sum[(3*NS + sho)*32]);
    };
    V *out = reinterpret_cast<V*>(apc + (size_t(it.coeff)*nrhs + it.src)*128 + row_lane<T>(quarter, lane));
    size_t const row = size_t(nrhs)*128*sizeof(T)/8;            // lanes of 8 bytes between coefficients
    if (1 == it.g_count) {
        for (int sho = zq; sho < NS; sho += 4) out[sho*row] = total(sho);
        return;
    }
    // partial sums of a group of items; the last item to finish (ticket counter) adds them in item
    // order, so the result does not depend on the order in which the items ran
    constexpr int R = 128*int(sizeof(T))/8;
    V *pg = reinterpret_cast<V*>(part + size_t(it.g_row)*128 + row_lane<T>(quarter, lane));
    V *mine = pg + size_t(it.g_pos)*NS*R;
    for (int sho = zq; sho < NS; sho += 4) mine[sho*R] = total(sho);
    __threadfence();                                            // partials visible before the ticket
    __syncthreads();
    uint32_t *ticket_s = reinterpret_cast<uint32_t*>(tb);
    uint32_t *counter = tickets + size_t(it.g_id)*4 + quarter;
    if (0 == tid) ticket_s[0] = atomicAdd(counter, 1u);
    __syncthreads();
    if (ticket_s[0] + 1 != it.g_count) return;                  // uniform: not the last item of the group
    __threadfence();
    for (int sho = zq; sho < NS; sho += 4) {
        V s = V(0);
        for (uint32_t i = 0; i < it.g_count; ++i) s = vadd(s, __ldcg(pg + (size_t(i)*NS + sho)*R));
        out[sho*row] = s;
    }
    if (0 == tid) *counter = 0u;                                // ready for the next call
}

// LMAX odd: the smallest at or above the largest basis size of the plan; the tables hold LMAX + 1
// functions per point.  Items of every basis size run in one launch.
template <typename T, int LMAX>
__global__ void __launch_bounds__(kThreads, LMAX <= 5 ? 3 : 2)
sho_project_line_kernel(T *__restrict__ apc, T const *__restrict__ x, uint32_t nrhs, PrjItem const *__restrict__ items,
                        uint4 const *__restrict__ recs, typename LaneOf<T>::V const *__restrict__ tab,
                        uint8_t const *__restrict__ active, T *__restrict__ part, uint32_t *__restrict__ tickets)
{
    extern __shared__ __align__(16) unsigned char smem_line[];
    PrjItem const it = items[blockIdx.x];
    if (active && !active[it.src]) return;                      // uniform: a retired source
    constexpr int LP = LMAX + 1;
    switch (it.lmax) {
#define A43G_PROJECT_CASE(L) case L: if constexpr (L <= LMAX) project_item<T, L, LP>(apc, x, nrhs, it, recs, tab, part, tickets, smem_line); break;
        A43G_PROJECT_CASE(0) A43G_PROJECT_CASE(1) A43G_PROJECT_CASE(2) A43G_PROJECT_CASE(3)
        A43G_PROJECT_CASE(4) A43G_PROJECT_CASE(5) A43G_PROJECT_CASE(6) A43G_PROJECT_CASE(7)
#undef A43G_PROJECT_CASE
    }
}

template <int LMAX> constexpr int project_smem() {
    return (4*nsho_of(LMAX)*32 + int(kMaxPrjItem)*8*(LMAX + 1))*8 + int(kMaxPrjItem)*16;
}

template <typename T, int LMAX>
bool prepare_project() {
    A43G_CUDA_TRY(cudaFuncSetAttribute(sho_project_line_kernel<T, LMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       project_smem<LMAX>()));
    return true;
}

template <typename T, int LMAX>
void project(DevicePlan &dp, T *apc, T const *x, void const *tab, T *part, cudaStream_t st) {
    using V = typename LaneOf<T>::V;
    sho_project_line_kernel<T, LMAX><<<dim3(dp.prj_line.count, LaneOf<T>::quarters), kThreads, project_smem<LMAX>(), st>>>(
        apc, x, dp.nCols, dptr<PrjItem>(dp.prj_line.items), dptr<uint4>(dp.prj_rec), static_cast<V const*>(tab),
        dp.retire ? dptr<uint8_t>(dp.src_active) : nullptr, part, dptr<uint32_t>(dp.prj_line.tickets));
}

template <typename T>
bool prepare() { return prepare_project<T, 1>() && prepare_project<T, 3>() && prepare_project<T, 5>() && prepare_project<T, 7>(); }

template <typename T>
bool launch_project(DevicePlan &dp, T *apc, T const *x, void const *tab, cudaStream_t st) {
    if (0 == dp.prj_line.count) return true;
    T *part = dptr<T>(dp.prj_part);
    switch (dp.lmax_max | 1) {
        case 1: project<T, 1>(dp, apc, x, tab, part, st); break;
        case 3: project<T, 3>(dp, apc, x, tab, part, st); break;
        case 5: project<T, 5>(dp, apc, x, tab, part, st); break;
        default: project<T, 7>(dp, apc, x, tab, part, st); break;
    }
    count_launch();
    A43G_CUDA_TRY(cudaGetLastError());
    return true;
}

} // namespace line
} // namespace a43g
