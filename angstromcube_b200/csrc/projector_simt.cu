// Addition of the action on the CUDA cores (FP32 and FP64), sum-factorized
// (include/green_dyadic.hxx:325-518), and the launches of the projection along lines.
//
// The projector functions are separable on the spherical mask,
//     P_(ix,iy,iz)(x, y, z) = H_ix(x) H_iy(y) H_iz(z)   for points inside the projection radius,
// so one (block, image) pair costs 64*(L+1) + 16*(L+1)(L+2)/2 + 4*nSHO fused multiply-adds per
// column instead of 64*nSHO for the dense product (944 instead of 3584 at numax 5).
//
// One CTA per run of blocks, one thread per (real/imaginary plane, column) with the 1D tables of
// the current (image, row) slot and the point sums in registers (loops fully unrolled for the
// basis size L): the contributions of all images near a block are summed and y is updated once;
// the coefficients of the next image are staged in shared memory with cp.async while the current
// one is applied (16-byte copies of rows that start on 512-byte boundaries of the plan's
// coefficient array).
#include "device.cuh"

#include <algorithm>

namespace a43g {

namespace {

constexpr int kBlk = 8192;            // floats per block: 2 planes x 64 points x 64 columns
constexpr int kThreads = 128;

__host__ __device__ constexpr int nsho_of(int L) { return ((L + 1)*(L + 2)*(L + 3))/6; }

__device__ __forceinline__ uint32_t smem_addr(void const *p) { return uint32_t(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void cp_async16(void *dst, void const *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait0() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// the 1D tables of one slot, H[nu][dir][i] at tab[(nu*3 + dir)*4 + i], dir 0/1/2 = x/y/z, staged in
// shared memory: FP32 copies them into registers, FP64 (twice the registers) reads them in place
template <typename T, int L> struct Tables;
template <int L> struct Tables<float, L> {
    float h[L + 1][3][4];
    __device__ __forceinline__ void load(float const *tab) {
#pragma unroll
        for (int nu = 0; nu <= L; ++nu)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                float4 const v = *reinterpret_cast<float4 const*>(tab + (nu*3 + d)*4);
                h[nu][d][0] = v.x; h[nu][d][1] = v.y; h[nu][d][2] = v.z; h[nu][d][3] = v.w;
            }
    }
    __device__ __forceinline__ float operator()(int nu, int d, int i) const { return h[nu][d][i]; }
};
template <int L> struct Tables<double, L> {
    double const *p;
    __device__ __forceinline__ void load(double const *tab) { p = tab; }
    __device__ __forceinline__ double operator()(int nu, int d, int i) const { return p[(nu*3 + d)*4 + i]; }
};

__device__ __forceinline__ float fmat(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fmat(double a, double b, double c) { return fma(a, b, c); }

// CTAs per SM the kernels are compiled for (FP64 needs twice the registers and shared memory)
template <typename T> struct Occ { static constexpr int add = 2; };
template <> struct Occ<double> { static constexpr int add = 1; };

__device__ __forceinline__ void cp_async8(void *dst, void const *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" :: "r"(smem_addr(dst)), "l"(src) : "memory");
}

// ---------------------------------------------------------------- addition

// contribution of one image with basis size L to the 64 point sums of this thread
// ZS threads share a column and split its x-points (FP64: the 64 sums of one thread would not
// fit the registers): thread zh owns x = zh*(4/ZS) ... of every (z, y) row, so each stage of
// the contraction (x, then y, then z) is split between them without repeating any work.  The
// sums are ordered acc[(z*4 + y)*(4/ZS) + x - zh*(4/ZS)].
// UZ: the z-orders unrolled (tables and coefficient offsets known at compile time) or one at a
// time (fewer registers)
template <typename T, int L, bool FULL, int ZS, bool UZ>
__device__ __forceinline__ void add_image(T (&acc)[64/ZS], Tables<T, L> const &t, uint64_t mask,
                                          T const *__restrict__ c, size_t cstride, int zh) {
    constexpr int kUnrollZ = UZ ? L + 1 : 1;
    constexpr int NX = 4/ZS;                                   // x-points of this thread
    int const x0 = (1 == ZS) ? 0 : zh*NX;
    int sho = 0;
#pragma unroll kUnrollZ
    for (int iz = 0; iz <= L; ++iz) {
        T byx[4*NX];
#pragma unroll
        for (int i = 0; i < 4*NX; ++i) byx[i] = T(0);
#pragma unroll
        for (int iy = 0; iy <= L - iz; ++iy) {
            T ax[NX];
#pragma unroll
            for (int xl = 0; xl < NX; ++xl) ax[xl] = T(0);
#pragma unroll
            for (int ix = 0; ix <= L - iz - iy; ++ix, ++sho) {
                T const cv = c[size_t(sho)*cstride];
#pragma unroll
                for (int xl = 0; xl < NX; ++xl) ax[xl] = fmat(t(ix, 0, x0 + xl), cv, ax[xl]);
            }
#pragma unroll
            for (int yy = 0; yy < 4; ++yy) {
                T const hy = t(iy, 1, yy);
#pragma unroll
                for (int xl = 0; xl < NX; ++xl) byx[yy*NX + xl] = fmat(hy, ax[xl], byx[yy*NX + xl]);
            }
        }
#pragma unroll
        for (int z = 0; z < 4; ++z) {
            T const hz = t(iz, 2, z);
#pragma unroll
            for (int q = 0; q < 4*NX; ++q) {
                int const pl = z*4*NX + q, p = z*16 + (q/NX)*4 + x0 + (q % NX);
                if (FULL) acc[pl] = fmat(hz, byx[q], acc[pl]);
                else acc[pl] = ((mask >> p) & 1u) ? fmat(hz, byx[q], acc[pl]) : acc[pl];
            }
        }
    }
}

template <typename T, int L, int ZS, bool UZ>
__device__ __forceinline__ void add_image_L(T (&acc)[64/ZS], T const *__restrict__ tab, uint64_t mask,
                                            T const *__restrict__ c, size_t cstride, int zh) {
    Tables<T, L> t;
    t.load(tab);
    if (~0ull == mask) add_image<T, L, true, ZS, UZ>(acc, t, mask, c, cstride, zh);
    else add_image<T, L, false, ZS, UZ>(acc, t, mask, c, cstride, zh);
}

// LMAX: largest basis size of the plan (the instantiation has no larger one).  One CTA walks the
// blocks [b0, b1) (consecutive, same order as y) and treats their (block, image) pairs as one
// stream: the coefficients, table and mask of the next pair are staged while the current pair is
// applied, and the y values of the next block with atoms are staged during the whole of the
// current block, so neither the start of a block nor its final y update waits for memory.
template <typename T, int LMAX, int ZS = int(sizeof(T))/4, bool UZ = true>
__global__ void __launch_bounds__(kThreads*ZS, Occ<T>::add)
sho_add_simt_kernel(T *__restrict__ y, T const *__restrict__ cad, uint32_t nrhs, uint32_t nnzb,
                    uint32_t blocks_per_cta, uint16_t const *__restrict__ colIndex,
                    uint32_t const *__restrict__ add_start, uint4 const *__restrict__ info,
                    T const *__restrict__ slot_H, uint64_t const *__restrict__ slot_mask, int stride,
                    uint8_t const *__restrict__ active)
{
    constexpr int NCMAX = nsho_of(LMAX);
    constexpr int TE = 16/int(sizeof(T));                  // elements per 16-byte copy
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *cbuf = reinterpret_cast<T*>(smem_raw);              // [2][NCMAX][128] coefficients of two pairs
    T *ybuf = cbuf + 2*NCMAX*128;                          // [8192] y of the current block
    __shared__ __align__(16) T tbuf[2][(LMAX + 1)*12];
    __shared__ uint64_t mbuf[2];
    uint32_t const b0 = blockIdx.x*blocks_per_cta, b1 = min(b0 + blocks_per_cta, nnzb);
    if (b0 >= b1) return;
    uint32_t const T0 = add_start[b0], T1 = add_start[b1];
    if (T0 >= T1) return;                                  // no atoms near any of these blocks
    constexpr int NT = kThreads*ZS, NP = 64/ZS;             // threads, point sums per thread
    int const tid = threadIdx.x, zh = tid/kThreads, reim = (tid >> 6) & 1, j = tid & 63;
    size_t const cstride = size_t(nrhs)*128;

    // the block owning pair t: blocks are visited in order, skipping blocks without pairs
    uint32_t bb = b0;
    while (add_start[bb + 1] <= T0) ++bb;
    uint32_t s = colIndex[bb];
    uint32_t bend = add_start[bb + 1];                     // first pair of the next block

    // pairs of a retired source stage nothing and carry an empty mask: no work, no y update
    auto stage_pair = [&](uint4 const inf, uint32_t src_col, int buf) {
        if (active && !active[src_col]) {
            if (tid == NT - 1) mbuf[buf] = 0;
            return;
        }
        int const L = int(inf.z), nc = nsho_of(L);
        T const *src = cad + (size_t(inf.y)*nrhs + src_col)*128;
        T *dst = cbuf + buf*NCMAX*128;
        constexpr int CPR = 128/TE;                        // 16-byte copies per coefficient row
        for (int q = tid; q < nc*CPR; q += NT) {
            int const row = q/CPR, part = (q % CPR)*TE;
            cp_async16(dst + row*128 + part, src + size_t(row)*cstride + part);
        }
        if (tid < (L + 1)*12/TE) cp_async16(&tbuf[buf][tid*TE], slot_H + size_t(inf.x)*stride + tid*TE);
        if (tid == NT - 1) cp_async8(&mbuf[buf], slot_mask + inf.x);
    };
    auto stage_y = [&](uint32_t blk) {
        if (active && !active[colIndex[blk]]) return;
        T const *src = y + size_t(blk)*kBlk;
#pragma unroll
        for (int r = 0; r < kBlk/(TE*NT); ++r) {
            int const o = (r*NT + tid)*TE;
            cp_async16(ybuf + o, src + o);
        }
    };
    // the source column of the pair after t (it may belong to a later block)
    auto column_of = [&](uint32_t t) -> uint32_t {
        uint32_t c = bb;
        while (add_start[c + 1] <= t) ++c;
        return colIndex[c];
    };

    T acc[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) acc[i] = T(0);
    uint64_t mask_all = 0;
    uint4 const zero4 = make_uint4(0u, 0u, 0u, 0u);
    uint4 cur = info[T0];
    stage_y(bb);
    stage_pair(cur, s, 0);
    cp_async_commit();
    uint4 nxt = (T0 + 1 < T1) ? info[T0 + 1] : zero4;
    int buf = 0;
    for (uint32_t t = T0; t < T1; ++t, buf ^= 1) {
        if (t + 1 < T1) stage_pair(nxt, (t + 1 < bend) ? s : column_of(t + 1), buf ^ 1);
        cp_async_commit();
        uint4 const after = (t + 2 < T1) ? info[t + 2] : zero4;
        cp_async_wait1();
        __syncthreads();
        uint64_t const mask = mbuf[buf];
        if (mask) {
            mask_all |= mask;
            T const *tab = tbuf[buf];
            T const *c = cbuf + buf*NCMAX*128 + reim*64 + j;
            int const L = int(cur.z);                      // uniform over the CTA
            if (L == LMAX) add_image_L<T, LMAX, ZS, UZ>(acc, tab, mask, c, 128, zh);
            else if (LMAX > 0 && L == 0) add_image_L<T, 0, ZS, UZ>(acc, tab, mask, c, 128, zh);
            else if (LMAX > 1 && L == 1) add_image_L<T, (LMAX > 1 ? 1 : 0), ZS, UZ>(acc, tab, mask, c, 128, zh);
            else if (LMAX > 2 && L == 2) add_image_L<T, (LMAX > 2 ? 2 : 0), ZS, UZ>(acc, tab, mask, c, 128, zh);
            else if (LMAX > 3 && L == 3) add_image_L<T, (LMAX > 3 ? 3 : 0), ZS, UZ>(acc, tab, mask, c, 128, zh);
            else if (LMAX > 4 && L == 4) add_image_L<T, (LMAX > 4 ? 4 : 0), ZS, UZ>(acc, tab, mask, c, 128, zh);
            else if (LMAX > 5 && L == 5) add_image_L<T, (LMAX > 5 ? 5 : 0), ZS, UZ>(acc, tab, mask, c, 128, zh);
            else if (LMAX > 6 && L == 6) add_image_L<T, (LMAX > 6 ? 6 : 0), ZS, UZ>(acc, tab, mask, c, 128, zh);
        }
        cur = nxt; nxt = after;
        if (t + 1 == bend) {
            // last pair of block bb: y[bb] = staged y + sums on the points inside the spheres
            cp_async_wait0();
            __syncthreads();
            T const *yb_s = ybuf + reim*4096 + j;
            T *yb = y + size_t(bb)*kBlk + reim*4096 + j;
#pragma unroll
            for (int pl = 0; pl < NP; ++pl) {
                int const p = (pl/(4/ZS))*4 + zh*(4/ZS) + pl % (4/ZS);   // this thread's points
                if ((mask_all >> p) & 1u) yb[p*64] = yb_s[p*64] + acc[pl];
                acc[pl] = T(0);
            }
            mask_all = 0;
            __syncthreads();                               // ybuf free
            if (t + 1 < T1) {
                ++bb;
                while (add_start[bb + 1] <= t + 1) ++bb;
                s = colIndex[bb];
                bend = add_start[bb + 1];
                stage_y(bb);                               // lands during the pairs of block bb
            }
        }
        __syncthreads();                                   // buffers buf are free for pair t + 2
    }
}

template <typename T> T const *simt_table(DevicePlan const &dp);
template <> float const *simt_table<float>(DevicePlan const &dp) { return dptr<float>(dp.slot_H32); }
template <> double const *simt_table<double>(DevicePlan const &dp) { return dptr<double>(dp.slot_H); }

template <typename T, int LMAX>
void launch_add_L(DevicePlan &dp, T *y, uint16_t const *colIndex, cudaStream_t st) {
    constexpr int smem = (2*nsho_of(LMAX)*128 + kBlk)*int(sizeof(T));
    constexpr int ZS = int(sizeof(T))/4;
    uint32_t const per_cta = std::max<uint32_t>(1, dp.add_blocks);
    unsigned const grid = (dp.nnzb + per_cta - 1)/per_cta;
    auto *k = sho_add_simt_kernel<T, LMAX, ZS, true>;
    if (sizeof(T) == 8 && !dp.add64_unrolled) k = sho_add_simt_kernel<T, LMAX, ZS, false>;
    k<<<grid, kThreads*ZS, smem, st>>>(y, dptr<T>(dp.cad), dp.nCols, dp.nnzb, per_cta,
        colIndex, dptr<uint32_t>(dp.add_start), dptr<uint4>(dp.add_info), simt_table<T>(dp),
        dptr<uint64_t>(dp.slot_mask), dp.table_stride, dp.retire ? dptr<uint8_t>(dp.src_active) : nullptr);
}

template <typename T, int L>
void set_smem_attributes() {
    cudaFuncSetAttribute(sho_add_simt_kernel<T, L, int(sizeof(T))/4, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (2*nsho_of(L)*128 + kBlk)*int(sizeof(T)));
    if (sizeof(T) == 8)
        cudaFuncSetAttribute(sho_add_simt_kernel<T, L, int(sizeof(T))/4, false>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (2*nsho_of(L)*128 + kBlk)*int(sizeof(T)));
}

} // namespace

bool prepare_simt_kernels() {
    // the dynamic shared memory the kernels need beyond 48 KB (per device: called with the
    // device current, before any launch and outside stream capture)
    set_smem_attributes<float, 0>(); set_smem_attributes<float, 1>(); set_smem_attributes<float, 2>();
    set_smem_attributes<float, 3>(); set_smem_attributes<float, 4>(); set_smem_attributes<float, 5>();
    set_smem_attributes<float, 6>(); set_smem_attributes<float, 7>();
    set_smem_attributes<double, 0>(); set_smem_attributes<double, 1>(); set_smem_attributes<double, 2>();
    set_smem_attributes<double, 3>(); set_smem_attributes<double, 4>(); set_smem_attributes<double, 5>();
    A43G_CUDA_TRY(cudaGetLastError());
    return true;
}

bool simt_projector_supported(DevicePlan const &dp, void const *x, void const *y, size_t real_bytes) {
    // 16-byte staging copies; the FP64 addition stages up to numax 5 (shared memory)
    int const lmax_limit = (8 == real_bytes) ? 5 : 7;
    return dp.slot_H32.ptr && dp.lmax_max <= lmax_limit && 0 == (reinterpret_cast<uintptr_t>(x) & 15u) &&
           0 == (reinterpret_cast<uintptr_t>(y) & 15u);
}

template <typename T>
bool launch_project_simt(DevicePlan &dp, T const *x, cudaStream_t st) {
    if (!ensure_prj_part(dp, sizeof(T))) return false;
    return launch_project_line(dp, dptr<T>(dp.apc), x, sizeof(T) == 8 ? dp.line_tab64.ptr : dp.line_tab32.ptr, st);
}

// (FP64 up to numax 5: its two coefficient stages and y fit 227 KB of shared memory)
template <typename T>
bool launch_add_simt(DevicePlan &dp, T *y, uint16_t const *colIndex, cudaStream_t st) {
    switch (dp.lmax_max) {
        case 0: launch_add_L<T, 0>(dp, y, colIndex, st); break;
        case 1: launch_add_L<T, 1>(dp, y, colIndex, st); break;
        case 2: launch_add_L<T, 2>(dp, y, colIndex, st); break;
        case 3: launch_add_L<T, 3>(dp, y, colIndex, st); break;
        case 4: launch_add_L<T, 4>(dp, y, colIndex, st); break;
        case 5: launch_add_L<T, 5>(dp, y, colIndex, st); break;
        default:
            if constexpr (sizeof(T) == 4) {
                if (6 == dp.lmax_max) launch_add_L<T, 6>(dp, y, colIndex, st);
                else launch_add_L<T, 7>(dp, y, colIndex, st);
            }
            break;
    }
    count_launch();
    A43G_CUDA_TRY(cudaGetLastError());
    return true;
}

template bool launch_project_simt<float>(DevicePlan &, float const *, cudaStream_t);
template bool launch_project_simt<double>(DevicePlan &, double const *, cudaStream_t);
template bool launch_add_simt<float>(DevicePlan &, float *, uint16_t const *, cudaStream_t);
template bool launch_add_simt<double>(DevicePlan &, double *, uint16_t const *, cudaStream_t);

} // namespace a43g
