// Projector contraction of the action on the CUDA cores (include/green_dyadic.hxx:112-288
// projection, :325-518 addition), FP32 and FP64, sum-factorized along the lines of cubes of an atom
// image.
//
// The projector functions are separable on the spherical mask,
//     P_(ix,iy,iz)(x, y, z) = H_ix(x) H_iy(y) H_iz(z)   for points inside the projection radius,
// and so is the whole sphere: all cubes of one x-line share H_iy(y) and H_iz(z), all lines of one
// z-slab of cubes share H_iz(z).  The x-contraction of the projection therefore accumulates over a whole line
// before the y-contraction is done once per line, and the z-contraction once per slab.  In the cells in
// use a line has 2.5 to 4.5 cubes (whole spheres about 6; images are cut by the faces of cells and
// truncation spheres) and is cut where a work item ends, so that 2.1 to 4.2 blocks share a y-contraction
// and 4 to 16 a z-contraction: 480 to 600 multiply-adds per block and column at L = 5 (480 on the
// 64-atom cell) instead of 64(L+1) + 16 N2 + 4 nSHO = 944, N2 = (L+1)(L+2)/2, when every block is
// contracted by itself, and 3584 for the dense product.
#pragma once

#include "device.cuh"
#include "lane8.cuh"

namespace a43g {
namespace line {

constexpr int kThreads = 128;         // 4 warps: warp z works on z-plane z of every cube

__host__ __device__ constexpr int nsho_of(int L) { return ((L + 1)*(L + 2)*(L + 3))/6; }
__host__ __device__ constexpr int n2_of(int L) { return ((L + 1)*(L + 2))/2; }

// columns per quarter (8-byte lanes of a warp): 32 in FP64, 64 in FP32
template <typename T> constexpr int quarters() { return int(sizeof(T))/2; }
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
void project(DevicePlan &dp, T *apc, T const *x, void const *tab, LineScratch const &sc, cudaStream_t st) {
    using V = typename LaneOf<T>::V;
    sho_project_line_kernel<T, LMAX><<<dim3(dp.prj_line.count, quarters<T>()), kThreads, project_smem<LMAX>(), st>>>(
        apc, x, dp.nCols, dptr<PrjItem>(dp.prj_line.items), dptr<uint4>(dp.prj_rec), static_cast<V const*>(tab),
        dp.retire ? dptr<uint8_t>(dp.src_active) : nullptr, static_cast<T*>(sc.part), sc.tickets);
}

// ---------------------------------------------------------------- addition

constexpr int kRecs = 32;             // records of a segment held in shared memory at a time
constexpr int kStages = 3;            // records whose coefficients and tables are in flight or in use

// one image on the cubes of a segment: c its coefficients [NS][32 lanes], t the tables (x of every
// cube, then y, then z), m the 16-point masks of this warp's plane of every cube
template <typename V, int L, int LP, int SEG>
__device__ __forceinline__ void add_image(V (&acc)[SEG][16], V const *c, V const *t, uint32_t const (&m)[SEG], int zq) {
    constexpr int N2 = n2_of(L);
    V byx[N2], ax[4][L + 1];
    {
        V h[L + 1];
        load_row(h, t + (4*SEG + 4 + zq)*LP);
#pragma unroll
        for (int iz = 0, sho = 0; iz <= L; ++iz)
#pragma unroll
            for (int iy = 0; iy <= L - iz; ++iy)
#pragma unroll
                for (int ix = 0; ix <= L - iz - iy; ++ix, ++sho) {
                    int const i = iy*(2*L + 3 - iy)/2 + ix;
                    byx[i] = (0 == iz) ? vmul(c[sho*32], h[iz]) : vfma(c[sho*32], h[iz], byx[i]);
                }
    }
#pragma unroll
    for (int y = 0; y < 4; ++y) {
        V h[L + 1];
        load_row(h, t + (4*SEG + y)*LP);
#pragma unroll
        for (int iy = 0, i = 0; iy <= L; ++iy)
#pragma unroll
            for (int ix = 0; ix <= L - iy; ++ix, ++i)
                ax[y][ix] = (0 == iy) ? vmul(byx[i], h[iy]) : vfma(byx[i], h[iy], ax[y][ix]);
    }
#pragma unroll
    for (int s = 0; s < SEG; ++s) {
        if (0xffffu == m[s]) {                                  // uniform over the warp
#pragma unroll
            for (int xx = 0; xx < 4; xx += 2) {                 // two points at a time: 8 independent chains
                V h[2][L + 1];
                load_row(h[0], t + (4*s + xx)*LP);
                load_row(h[1], t + (4*s + xx + 1)*LP);
#pragma unroll
                for (int ix = 0; ix <= L; ++ix)
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        V &a = acc[s][4*(q & 3) + xx + (q >> 2)];
                        a = vfma(ax[q & 3][ix], h[q >> 2][ix], a);
                    }
            }
        } else if (m[s]) {
#pragma unroll
            for (int xx = 0; xx < 4; ++xx) {
                V h[L + 1], f[4];
                load_row(h, t + (4*s + xx)*LP);
#pragma unroll
                for (int ix = 0; ix <= L; ++ix)
#pragma unroll
                    for (int y = 0; y < 4; ++y) f[y] = (0 == ix) ? vmul(ax[y][0], h[0]) : vfma(ax[y][ix], h[ix], f[y]);
#pragma unroll
                for (int y = 0; y < 4; ++y)
                    if (m[s] & (1u << (4*y + xx))) acc[s][4*y + xx] = vadd(acc[s][4*y + xx], f[y]);
            }
        }
    }
}

// a segment whose blocks the caller's colIndex gives to other columns than the plan's: every cube by
// itself, coefficients and tables read in place (a call that no solver makes).  Kept out of the loop over
// images: masks by column in there cost 2 to 3 % of the dyadic part of the 64-atom cell, this 0.5 % or less
template <typename T, int LP, int SEG>
__device__ __noinline__ void add_by_columns(T *yl, T const *cq, uint32_t nrhs, uint16_t const *colIndex, AddSegment const *seg,
                                            AddRecord const *recs, typename LaneOf<T>::V const *tab, int zq) {
    using V = typename LaneOf<T>::V;
    constexpr int S = 64*int(sizeof(T))/8;
    for (int s = 0; s < SEG; ++s) {
        if (!(uint32_t(seg->any[s] >> (16*zq)) & 0xffffu)) continue;
        T const *cs = cq + size_t(colIndex[seg->blk[s]])*128;
        V acc[16];
#pragma unroll
        for (int p = 0; p < 16; ++p) acc[p] = V(0);
        for (uint32_t i = 0; i < seg->count; ++i) {
            AddRecord const &r = recs[i];
            uint32_t const m = uint32_t(r.mask[s] >> (16*zq)) & 0xffffu;
            if (!m) continue;
            int const L = int(r.lmax);
            V const *hx = tab + size_t(r.slot[s])*12*LP, *hy = hx + 4*LP, *hz = hx + (8 + zq)*LP;
            T const *c = cs + size_t(r.coeff)*nrhs*128;
            V f[16];
#pragma unroll
            for (int p = 0; p < 16; ++p) f[p] = V(0);
            for (int iz = 0; iz <= L; ++iz)
                for (int iy = 0; iy <= L - iz; ++iy) {
                    V ax[4] = {V(0), V(0), V(0), V(0)};
                    for (int ix = 0; ix <= L - iz - iy; ++ix, c += size_t(nrhs)*128)
#pragma unroll
                        for (int xx = 0; xx < 4; ++xx) ax[xx] = vfma(*reinterpret_cast<V const*>(c), hx[xx*LP + ix], ax[xx]);
#pragma unroll
                    for (int p = 0; p < 16; ++p) f[p] = vfma(vmul(hy[(p >> 2)*LP + iy], hz[iz]), ax[p & 3], f[p]);
                }
#pragma unroll
            for (int p = 0; p < 16; ++p) if ((m >> p) & 1u) acc[p] = vadd(acc[p], f[p]);
        }
        V *yb = reinterpret_cast<V*>(yl + size_t(seg->blk[s])*8192);
#pragma unroll
        for (int p = 0; p < 16; ++p) yb[p*S] = vadd(yb[p*S], acc[p]);
    }
}

// y += the projector functions of all images times their coefficients (include/green_dyadic.hxx:
// 325-518).  CTA = (segment, quarter of the columns): a segment is up to SEG cubes of one x-line of
// a source that have images, with one record per image near any of them.  Warp z owns plane z of
// every cube, a lane 8 bytes of columns.  Per image the coefficients are contracted with the
// z-functions of the plane (56 multiply-adds at L = 5) and the y-functions of the rows (84) once for
// the whole segment, then with the x-functions of every cube (96); the sums over all images stay in
// registers and y is read and written once at the end.  Coefficients and
// tables of the next two records are in flight while one is applied.
//
// Measured on the 64-atom cell with 8 sources, against one contraction per (block, image) pair:
// FP32 1.91 -> 0.93 ms, FP64 3.86 -> 1.87 ms (1.02 and 2.07 ms with y staged in shared memory from
// the start of the CTA on).  The FMA pipe is about a third busy (issue slots too): the point sums
// take 128 of some 250 registers, which leaves two CTAs per SM.  Segments of 2 cubes and three CTAs
// per SM are 2 % slower there, and two records per barrier no faster.
template <typename T, int LMAX, int SEG>
__global__ void __launch_bounds__(kThreads, LMAX <= 5 ? 2 : 1)
sho_add_line_kernel(T *__restrict__ y, T const *__restrict__ cad, uint32_t nrhs, uint16_t const *__restrict__ colIndex,
                    AddSegment const *__restrict__ segs, AddRecord const *__restrict__ recs,
                    typename LaneOf<T>::V const *__restrict__ tab, uint8_t const *__restrict__ active)
{
    using V = typename LaneOf<T>::V;
    constexpr int LP = LMAX + 1, TS = 12*LP, NT = (4*SEG + 8)*LP, NC = nsho_of(LMAX)*32;
    constexpr int S = 64*int(sizeof(T))/8;                      // lanes of 8 bytes per point
    extern __shared__ __align__(16) unsigned char smem_line[];
    V *ring = reinterpret_cast<V*>(smem_line);                  // [kStages][NC + NT]
    AddRecord *rec = reinterpret_cast<AddRecord*>(ring + kStages*(NC + NT));   // [kRecs]
    int const tid = threadIdx.x, zq = tid >> 5, lane = tid & 31, quarter = blockIdx.y;
    AddSegment const *seg = segs + blockIdx.x;
    uint32_t const src = seg->src;
    if (active && !active[src]) return;                         // uniform: a retired source
    int const count = int(seg->count);
    AddRecord const *mine = recs + seg->first;
    T *yl = y + block_lane<T>(quarter, lane) + zq*1024;
    auto plane = [&](uint64_t mask) { return uint32_t(mask >> (16*zq)) & 0xffffu; };

    // the coefficients (rows of 32 lanes = 256 bytes) and tables of record i into ring slot i % kStages
    T const *cl = cad + size_t(src)*128 + row_lane<T>(quarter, 0);
    size_t const cstride = size_t(nrhs)*128;
    auto stage = [&](int i) {
        AddRecord const &r = rec[i];
        V *dst = ring + (i % kStages)*(NC + NT);
        int const L = int(r.lmax), nc = ((L + 1)*(L + 2)*(L + 3))/6;
        T const *c = cl + size_t(r.coeff)*cstride;
        for (int q = tid; q < nc*16; q += kThreads) {
            int const row = q >> 4, o = q & 15;
            copy16(dst + row*32 + 2*o, reinterpret_cast<V const*>(c + row*cstride) + 2*o);
        }
        V *td = dst + NC;
#pragma unroll
        for (int q = tid; q < NT/2; q += kThreads) {
            int const row = (2*q)/LP, o = 2*q - row*LP;         // table row: x of the cubes, y, z
            uint32_t const slot = (row < 4*SEG) ? r.slot[row >> 2] : r.yz_slot;
            int const tr = (row < 4*SEG) ? (row & 3) : row - 4*SEG + 4;
            if (slot != kNoSlot) copy16(td + row*LP + o, tab + size_t(slot)*TS + tr*LP + o);
        }
    };

    V acc[SEG][16];
#pragma unroll
    for (int s = 0; s < SEG; ++s)
#pragma unroll
        for (int p = 0; p < 16; ++p) acc[s][p] = V(0);
    for (int r0 = 0; r0 < count; r0 += kRecs) {
        int const n = min(kRecs, count - r0);
        __syncthreads();                                        // the ring and the records are free
        constexpr int RQ = int(sizeof(AddRecord))/16;
        for (int q = tid; q < n*RQ; q += kThreads)
            reinterpret_cast<uint4*>(rec)[q] = __ldg(reinterpret_cast<uint4 const*>(mine + r0) + q);
        __syncthreads();
        stage(0);
        copy_commit();
        if (n > 1) stage(1);
        copy_commit();
        for (int i = 0; i < n; ++i) {
            copy_wait<1>();
            __syncthreads();                                    // record i has landed; record i - 1 is done with
            if (i + 2 < n) stage(i + 2);
            copy_commit();
            V const *c = ring + (i % kStages)*(NC + NT) + lane;
            V const *t = ring + (i % kStages)*(NC + NT) + NC;
            uint32_t m[SEG];
#pragma unroll
            for (int s = 0; s < SEG; ++s) m[s] = plane(rec[i].mask[s]);
            switch (rec[i].lmax) {
#define A43G_ADD_CASE(L) case L: if constexpr (L <= LMAX) add_image<V, L, LP, SEG>(acc, c, t, m, zq); break;
                A43G_ADD_CASE(0) A43G_ADD_CASE(1) A43G_ADD_CASE(2) A43G_ADD_CASE(3)
                A43G_ADD_CASE(4) A43G_ADD_CASE(5) A43G_ADD_CASE(6) A43G_ADD_CASE(7)
#undef A43G_ADD_CASE
            }
        }
    }
    // y: two cubes' reads in flight at a time, and beside the first ones the caller's columns
    static_assert(0 == SEG % 2, "cubes are updated in pairs");
#pragma unroll
    for (int s = 0; s < SEG; s += 2) {
        V v[2][16];
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (plane(seg->any[s + h])) {
                V const *p = reinterpret_cast<V const*>(yl + size_t(seg->blk[s + h])*8192);
#pragma unroll
                for (int k = 0; k < 16; ++k) v[h][k] = p[k*S];
            }
        if (0 == s) {
            bool other = false;
#pragma unroll
            for (int i = 0; i < SEG; ++i) other |= seg->any[i] && colIndex[seg->blk[i]] != src;
            if (other) {                                        // uniform: the sums are of other columns
                add_by_columns<T, LP, SEG>(yl, cad + row_lane<T>(quarter, lane), nrhs, colIndex, seg, mine, tab, zq);
                return;
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (plane(seg->any[s + h])) {
                V *p = reinterpret_cast<V*>(yl + size_t(seg->blk[s + h])*8192);
#pragma unroll
                for (int k = 0; k < 16; ++k) p[k*S] = vadd(v[h][k], acc[s + h][k]);
            }
    }
}

template <int LMAX> constexpr int segment_cubes() { return LMAX <= 5 ? int(kSegment) : int(kSegment)/2; }
template <int LMAX> constexpr int add_smem() {
    constexpr int SEG = segment_cubes<LMAX>();
    return kStages*(nsho_of(LMAX)*32 + (4*SEG + 8)*(LMAX + 1))*8 + kRecs*int(sizeof(AddRecord));
}

template <typename T, int LMAX>
bool prepare_add() {
    A43G_CUDA_TRY(cudaFuncSetAttribute(sho_add_line_kernel<T, LMAX, segment_cubes<LMAX>()>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, add_smem<LMAX>()));
    return true;
}

template <typename T, int LMAX>
void add(DevicePlan &dp, T *y, T const *cad, uint16_t const *colIndex, void const *tab, cudaStream_t st) {
    using V = typename LaneOf<T>::V;
    sho_add_line_kernel<T, LMAX, segment_cubes<LMAX>()><<<dim3(dp.add_segments, quarters<T>()), kThreads, add_smem<LMAX>(), st>>>(
        y, cad, dp.nCols, colIndex, dptr<AddSegment>(dp.add_seg), dptr<AddRecord>(dp.add_rec),
        static_cast<V const*>(tab), dp.retire ? dptr<uint8_t>(dp.src_active) : nullptr);
}

template <typename T>
bool launch_add(DevicePlan &dp, T *y, T const *cad, uint16_t const *colIndex, void const *tab, cudaStream_t st) {
    if (0 == dp.add_segments) return true;
    switch (dp.lmax_max | 1) {
        case 1: add<T, 1>(dp, y, cad, colIndex, tab, st); break;
        case 3: add<T, 3>(dp, y, cad, colIndex, tab, st); break;
        case 5: add<T, 5>(dp, y, cad, colIndex, tab, st); break;
        default: add<T, 7>(dp, y, cad, colIndex, tab, st); break;
    }
    count_launch();
    A43G_CUDA_TRY(cudaGetLastError());
    return true;
}

template <typename T>
bool prepare() {
    return prepare_project<T, 1>() && prepare_project<T, 3>() && prepare_project<T, 5>() && prepare_project<T, 7>() &&
           prepare_add<T, 1>() && prepare_add<T, 3>() && prepare_add<T, 5>() && prepare_add<T, 7>();
}

template <typename T>
bool launch_project(DevicePlan &dp, T *apc, T const *x, void const *tab, LineScratch const &sc, cudaStream_t st) {
    if (0 == dp.prj_line.count) return true;
    switch (dp.lmax_max | 1) {
        case 1: project<T, 1>(dp, apc, x, tab, sc, st); break;
        case 3: project<T, 3>(dp, apc, x, tab, sc, st); break;
        case 5: project<T, 5>(dp, apc, x, tab, sc, st); break;
        default: project<T, 7>(dp, apc, x, tab, sc, st); break;
    }
    count_launch();
    A43G_CUDA_TRY(cudaGetLastError());
    return true;
}

} // namespace line
} // namespace a43g
