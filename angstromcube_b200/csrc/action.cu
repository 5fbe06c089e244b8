// The Green-function action y = (H - E S) x on sm_100a.
//
//  * local part (potential V - E and the finite-difference kinetic energy) in ONE pass:
//    local_pencil_kernel walks the z-lines of cubes of one source column block, with the x- and
//    y-stencils in registers and the z-stencil from three cubes in shared memory, so y is written
//    exactly once per block (the reference makes four passes that re-read and re-write y,
//    include/green_action.hxx:159-167).
//    Plans with a 17-point stencil in some direction use the generic per-direction kernels.
//  * dyadic part (PAW projectors): projection, atom-matrix multiply, addition
//    (include/green_dyadic.hxx:856-922), with the image/atom coefficient scratch owned by
//    the plan instead of being allocated on every call.
#include "device.cuh"
#include "lane8.cuh"

#include <algorithm>

namespace a43g {

namespace {

constexpr int kBlockReals = 8192;   // 2 x 64 x 64

template <typename T>
struct Stencil9 { T c[3][5]; };      // per direction, c[0] centre ... c[4] distance 4

template <typename T>
Stencil9<T> make_stencil9(DevicePlan const &dp) {
    // 8th-order second derivative {-14350, 8064, -1008, 128, -9}/5040 times -1/(2h^2),
    // formed in double and rounded to real_t as include/green_kinetic.hxx:37-42 does
    Stencil9<T> s;
    double const w[5] = {-14350, 8064, -1008, 128, -9};
    for (int d = 0; d < 3; ++d) {
        double const norm = dp.prefactor[d]/5040.;
        for (int k = 0; k < 5; ++k) s.c[d][k] = T(w[k]*norm);
        if (dp.FD_range[d] < 1) for (int k = 0; k < 5; ++k) s.c[d][k] = T(0);
    }
    return s;
}

// energy and Bloch phases of one (energy, k-point) pair of a batch plan
template <typename T>
struct PairArgs { T E_re, E_im; T ph[3][2][2]; };

template <typename T>
struct LocalArgs {
    Stencil9<T> st;
    T E_re, E_im;
    T ph[3][2][2];                   // Bloch phases [dd][left,right][re,im]
    PairArgs<T> const *pairs;        // batch plan: per-pair values (nullptr: the values above)
    uint16_t const *colindx;         // block -> source column (batch plans and retirement)
    uint8_t const *active;           // per-source flag: 0 = retired, skip (nullptr: all active)
    uint32_t nsrc_pair;              // sources per pair
};

// the values of the pair that owns block b (uniform over a CTA that works on one z-line: the
// lines of a batch plan never mix sources); false if b's source is retired
template <typename T>
__device__ __forceinline__ bool line_args(LocalArgs<T> &a, int32_t b) {
    if (!a.colindx) return true;
    uint32_t const s = a.colindx[b];
    if (a.active && !a.active[s]) return false;
    if (a.pairs) {
        PairArgs<T> const &q = a.pairs[s/a.nsrc_pair];
        a.E_re = q.E_re; a.E_im = q.E_im;
#pragma unroll
        for (int d = 0; d < 3; ++d)
#pragma unroll
            for (int u = 0; u < 2; ++u) { a.ph[d][u][0] = q.ph[d][u][0]; a.ph[d][u][1] = q.ph[d][u][1]; }
    }
    return true;
}

// 4 consecutive points (x = 0..3 of one (z, y) row) of one column from shared memory
template <typename T> struct Row4 { T v[4]; };
template <typename T>
__device__ __forceinline__ Row4<T> lds_row(T const *p) {
    Row4<T> r;
    if (sizeof(T) == 4) {
        float4 const a = *reinterpret_cast<float4 const*>(p);
        r.v[0] = T(a.x); r.v[1] = T(a.y); r.v[2] = T(a.z); r.v[3] = T(a.w);
    } else {
        double2 const a = *reinterpret_cast<double2 const*>(p), b = *reinterpret_cast<double2 const*>(p + 2);
        r.v[0] = T(a.x); r.v[1] = T(a.y); r.v[2] = T(b.x); r.v[3] = T(b.y);
    }
    return r;
}
template <typename T>
__device__ __forceinline__ void sts_row(T *p, T const (&v)[4]) {
    if (sizeof(T) == 4) {
        *reinterpret_cast<float4*>(p) = make_float4(float(v[0]), float(v[1]), float(v[2]), float(v[3]));
    } else {
        *reinterpret_cast<double2*>(p) = make_double2(double(v[0]), double(v[1]));
        *reinterpret_cast<double2*>(p + 2) = make_double2(double(v[2]), double(v[3]));
    }
}

// 4 contiguous values from global memory (one potential row)
template <typename T>
__device__ __forceinline__ Row4<T> lds_row_global(T const *__restrict__ p) {
    Row4<T> r;
    if (sizeof(T) == 4) {
        float4 const a = __ldg(reinterpret_cast<float4 const*>(p));
        r.v[0] = T(a.x); r.v[1] = T(a.y); r.v[2] = T(a.z); r.v[3] = T(a.w);
    } else {
        double2 const a = __ldg(reinterpret_cast<double2 const*>(p)), b = __ldg(reinterpret_cast<double2 const*>(p) + 1);
        r.v[0] = T(a.x); r.v[1] = T(a.y); r.v[2] = T(b.x); r.v[3] = T(b.y);
    }
    return r;
}

// the row (z, y) = r of one cube (encoded e) for column col: 4 points x = 0..3, real and
// imaginary part, optionally rotated by a Bloch phase (pr, pi)
template <typename T>
__device__ __forceinline__ void load_row(T const *__restrict__ x, int32_t e, T pr, T pi, int r, int col,
                                         T (&re)[4], T (&im)[4]) {
    if (-1 == e) {
#pragma unroll
        for (int i = 0; i < 4; ++i) { re[i] = T(0); im[i] = T(0); }
        return;
    }
    T const *b = x + size_t(nbr_block(e))*kBlockReals + (r*4)*64 + col;
#pragma unroll
    for (int i = 0; i < 4; ++i) { re[i] = __ldg(b + i*64); im[i] = __ldg(b + 4096 + i*64); }
    if (e < -1) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            T const a = pr*re[i] - pi*im[i], c = pr*im[i] + pi*re[i];
            re[i] = a; im[i] = c;
        }
    }
}

// list entry (inzb+1, 0, -(inzb+1)) to neighbour code (>= 0 plain, -1 zero, <= -2 phase)
__device__ __forceinline__ int32_t list_code(int32_t entry) {
    return (entry > 0) ? entry - 1 : ((entry < 0) ? -(-entry - 1) - 2 : -1);
}

// One CTA per (z-line of cubes, slice of S columns).  Thread (j, r) owns row r = (z, y) of
// every cube of the line for column j: the x-stencil runs in registers (with the x-neighbour
// rows loaded directly), the y- and z-stencils read whole rows from shared memory, where the
// previous, current and next cube of the line and the two y-neighbour cubes are staged.
// Shared rows are padded to 68 points, so the 128-bit row accesses of a quarter warp hit
// distinct banks.
template <typename T, int S>
__global__ void __launch_bounds__(S*16)
local_fused_kernel(T *__restrict__ y, T const *__restrict__ x,
                   uint32_t const *__restrict__ zstart, int32_t const *__restrict__ zlist,
                   int32_t const *__restrict__ nbr, int32_t const *__restrict__ veff,
                   T const *__restrict__ Vcell, LocalArgs<T> a)
{
    constexpr int NSL = 64/S, PAD = 68;
    __shared__ __align__(16) T sm[5][2][S][PAD];   // slots: 3 rotating z-slots, y-, y+
    int const line = blockIdx.x/NSL, slice = blockIdx.x % NSL;
    int const j = threadIdx.x % S, r = threadIdx.x/S;       // r = z*4 + y
    int const zq = r >> 2, yq = r & 3, col = slice*S + j;
    int32_t const *L = zlist + zstart[line];
    int n = 0;
    while (L[4 + n] > 0) ++n;        // lists end with 4 non-positive entries
    if (0 == n || !line_args(a, L[4] - 1)) return;           // uniform over the CTA
    T const (&cx)[5] = a.st.c[0];
    T const (&cy)[5] = a.st.c[1];
    T const (&cz)[5] = a.st.c[2];
    T const c0 = cx[0] + cy[0] + cz[0];

    T cre[4], cim[4], nre[4], nim[4];
    {   // left z-halo into slot 0, first cube into slot 1
        T pre[4], pim[4];
        load_row(x, list_code(L[3]), a.ph[2][0][0], a.ph[2][0][1], r, col, pre, pim);
        sts_row(&sm[0][0][j][r*4], pre); sts_row(&sm[0][1][j][r*4], pim);
    }
    load_row(x, L[4] - 1, T(0), T(0), r, col, cre, cim);
    sts_row(&sm[1][0][j][r*4], cre); sts_row(&sm[1][1][j][r*4], cim);
    int sp = 0, sc = 1, sn = 2;                      // rotating slots: previous, current, next cube

    for (int k = 0; k < n; ++k) {
        int32_t const b = L[4 + k] - 1;
        int32_t const *nb = nbr + 6*size_t(b);
        int32_t const exm = nb[0], exp_ = nb[1], eym = nb[2], eyp = nb[3];
        load_row(x, list_code(L[5 + k]), a.ph[2][1][0], a.ph[2][1][1], r, col, nre, nim);
        T ymr[4], ymi[4], ypr[4], ypi[4];
        load_row(x, eym, a.ph[1][0][0], a.ph[1][0][1], r, col, ymr, ymi);
        load_row(x, eyp, a.ph[1][1][0], a.ph[1][1][1], r, col, ypr, ypi);
        T lr[12], li[12];                            // x-line: left row | own row | right row
        load_row(x, exm, a.ph[0][0][0], a.ph[0][0][1], r, col, *reinterpret_cast<T(*)[4]>(&lr[0]), *reinterpret_cast<T(*)[4]>(&li[0]));
        load_row(x, exp_, a.ph[0][1][0], a.ph[0][1][1], r, col, *reinterpret_cast<T(*)[4]>(&lr[8]), *reinterpret_cast<T(*)[4]>(&li[8]));
#pragma unroll
        for (int i = 0; i < 4; ++i) { lr[4 + i] = cre[i]; li[4 + i] = cim[i]; }
        __syncthreads();                             // previous step finished reading the slots
        sts_row(&sm[sn][0][j][r*4], nre); sts_row(&sm[sn][1][j][r*4], nim);
        sts_row(&sm[3][0][j][r*4], ymr); sts_row(&sm[3][1][j][r*4], ymi);
        sts_row(&sm[4][0][j][r*4], ypr); sts_row(&sm[4][1][j][r*4], ypi);
        __syncthreads();
        T accr[4], acci[4];
        {
            int32_t const iloc = veff[b];
            T V[4];
            if (iloc < 0) { V[0] = V[1] = V[2] = V[3] = T(0); }
            else { Row4<T> const v = lds_row_global(Vcell + size_t(iloc)*64 + r*4); V[0] = v.v[0]; V[1] = v.v[1]; V[2] = v.v[2]; V[3] = v.v[3]; }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                T const Vt = V[i] - a.E_re;
                accr[i] = Vt*cre[i] + a.E_im*cim[i] + c0*cre[i];
                acci[i] = Vt*cim[i] - a.E_im*cre[i] + c0*cim[i];
            }
        }
        // x direction in registers
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int d = 1; d <= 4; ++d) {
                accr[i] += cx[d]*(lr[4 + i - d] + lr[4 + i + d]);
                acci[i] += cx[d]*(li[4 + i - d] + li[4 + i + d]);
            }
        // y and z directions: whole rows from shared memory
#pragma unroll
        for (int d = 1; d <= 4; ++d) {
            int const ym = yq - d, yp = yq + d, zm = zq - d, zp = zq + d;
            int const s_ym = (ym < 0) ? 3 : sc, s_yp = (yp > 3) ? 4 : sc;
            int const s_zm = (zm < 0) ? sp : sc, s_zp = (zp > 3) ? sn : sc;
            int const o_ym = (zq*4 + (ym & 3))*4, o_yp = (zq*4 + (yp & 3))*4;
            int const o_zm = ((zm & 3)*4 + yq)*4, o_zp = ((zp & 3)*4 + yq)*4;
            Row4<T> const r1 = lds_row(&sm[s_ym][0][j][o_ym]), r2 = lds_row(&sm[s_yp][0][j][o_yp]);
            Row4<T> const r3 = lds_row(&sm[s_zm][0][j][o_zm]), r4 = lds_row(&sm[s_zp][0][j][o_zp]);
            Row4<T> const i1 = lds_row(&sm[s_ym][1][j][o_ym]), i2 = lds_row(&sm[s_yp][1][j][o_yp]);
            Row4<T> const i3 = lds_row(&sm[s_zm][1][j][o_zm]), i4 = lds_row(&sm[s_zp][1][j][o_zp]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                accr[i] += cy[d]*(r1.v[i] + r2.v[i]) + cz[d]*(r3.v[i] + r4.v[i]);
                acci[i] += cy[d]*(i1.v[i] + i2.v[i]) + cz[d]*(i3.v[i] + i4.v[i]);
            }
        }
        T *yb = y + size_t(b)*kBlockReals + (r*4)*64 + col;
#pragma unroll
        for (int i = 0; i < 4; ++i) { yb[i*64] = accr[i]; yb[4096 + i*64] = acci[i]; }
        int const t = sp; sp = sc; sc = sn; sn = t;  // rotate the z-slots
#pragma unroll
        for (int i = 0; i < 4; ++i) { cre[i] = nre[i]; cim[i] = nim[i]; }
    }
}

// Pencil kernel (FP32 and FP64): one CTA per (z-line, group of 16 lanes of columns).  A lane holds 8
// bytes of columns, one in FP64, two in FP32 (.f32x2 arithmetic); a warp is one z-plane zq, its two
// halves the planes re and im.  A thread owns the 16 points of its plane: the x- and y-stencils run
// in registers, the rows of the x- and y-neighbours come straight from global memory (the L2), those
// in x a z-stencil ahead of their use.  Only the z-stencil reads shared memory, where the previous, current
// and next cube of the line are staged by 16-byte asynchronous copies, [slot][re, im][point][lane]
// (a half warp reads 128 contiguous bytes); the copy of the cube after the next one starts as soon
// as the z-stencil is done with the previous cube.  The only couplings of re and im, -i Im(E) x and
// the Bloch phases of halo cubes, take the other plane's values from the partner lane (lane ^ 16).
//
// Measured on the 64-atom cell with 8 sources (32,768 blocks): FP64 1.36 ms (4.3 GB read and written
// once: 0.66 ms), FP32 0.68 ms; with the x-neighbours' rows loaded after the barrier 1.60 and 0.83
// ms; with the z-successor also in registers instead of copied, one FP32 column per lane, and the
// length of the line found by walking it, 1.80 and 0.89 ms.  Three CTAs per SM (168 registers): four
// leave too few of the rows in flight (FP64 1.92 ms), two too few warps (1.55 ms), and carrying the
// rows of the y-neighbours and of the next step ahead as well spills (1.67 ms).  What bounds it: the
// latency of those loads, and the 8 shared-memory reads per point of the z-stencil.
constexpr int kMaxLine = 128;        // cubes of a line (the host checks)
constexpr int kPencilThreads = 128;
constexpr int kPencilSmem = 3*2*64*16*8;          // bytes of the three z-slots

// a lane's 8 bytes of global memory on an A-byte boundary
template <int A> __device__ __forceinline__ double lane_load(double const *p) { return __ldg(p); }
template <int A> __device__ __forceinline__ unsigned long long lane_load(unsigned long long const *p) {
    if (A >= 8) return __ldg(p);
    float const *f = reinterpret_cast<float const*>(p);
    float const a = __ldg(f), b = __ldg(f + 1);
    unsigned long long d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
}
template <int A> __device__ __forceinline__ void lane_store(double *p, double v) { *p = v; }
template <int A> __device__ __forceinline__ void lane_store(unsigned long long *p, unsigned long long v) {
    if (A >= 8) { *p = v; return; }
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    float *f = reinterpret_cast<float*>(p);
    f[0] = a; f[1] = b;
}
// asynchronous copy of A = 4, 8 or 16 bytes to shared memory (only 16 can pass the L1 by)
template <int A> __device__ __forceinline__ void copy_async(void *dst, void const *src) {
    uint32_t const d = uint32_t(__cvta_generic_to_shared(dst));
    if (16 == A) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(d), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" :: "r"(d), "l"(src), "n"(A) : "memory");
}

// A: the boundary in bytes that x and y lie on (16, 8 or 4); off 16 bytes the copies are as small as A, and
// two loads and stores make a lane on 4.  On the cell above FP64 takes 1.67 ms on 8 bytes, FP32 0.88 ms on
// 8 and 0.95 ms on 4; the rows kernel takes 3.56 and 1.49 ms.
template <typename T, int A>
__global__ void __launch_bounds__(kPencilThreads, 3)
local_pencil_kernel(T *__restrict__ y, T const *__restrict__ x,
                    uint32_t const *__restrict__ zstart, int32_t const *__restrict__ zlist,
                    int32_t const *__restrict__ nbr, int32_t const *__restrict__ veff,
                    T const *__restrict__ Vcell, T const *__restrict__ zero, LocalArgs<T> a)
{
    using V = typename LaneOf<T>::V;
    constexpr int W = 8/int(sizeof(T)), S = 64/W, NG = S/16;   // columns per lane, lanes per point, groups
    extern __shared__ __align__(16) unsigned char slot_raw[];
    V *slots = reinterpret_cast<V*>(slot_raw);         // [3][2][64][16]
    __shared__ int32_t code[kMaxLine][8];              // per step: block, x-, x+, y-, y+, veff, z-next
    int const line = blockIdx.x/NG, group = blockIdx.x % NG;
    int const tid = threadIdx.x, lane = tid & 31, zq = tid >> 5, pl = lane >> 4, j = lane & 15;
    int32_t const *L = zlist + zstart[line];
    int const n = int(zstart[line + 1] - zstart[line]) - 8;    // lists have 4 halo entries at both ends
    if (n < 1 || !line_args(a, L[4] - 1)) return;      // uniform: nothing on this line, or retired
    int32_t const zleft = list_code(L[3]);
    for (int k = tid; k < n; k += kPencilThreads) {
        int32_t const b = L[4 + k] - 1;
        int32_t const *nb = nbr + 6*size_t(b);
        code[k][0] = b; code[k][1] = nb[0]; code[k][2] = nb[1]; code[k][3] = nb[2]; code[k][4] = nb[3];
        code[k][5] = veff[b]; code[k][6] = list_code(L[5 + k]);
    }
    size_t const lo = size_t(pl)*4096 + group*16*W + j*W;      // element of this lane at point 0
    V *mine = slots + (pl*64 + zq*16)*16 + j;                  // this thread's points of slot 0
    constexpr int SLOT = 2*64*16;
    auto fetch = [&](int slot, int32_t e) {                    // cube e into a slot (-1: zeros)
        V *dst = slots + slot*SLOT;
        if (-1 == e) {
#pragma unroll
            for (int i = 0; i < 16; ++i) mine[slot*SLOT + i*16] = V(0);
        } else {
            T const *src = x + size_t(nbr_block(e))*kBlockReals + group*16*W;
            constexpr int P = 128/A, E = A/int(sizeof(T));     // pieces of a row of 128 bytes, elements of a piece
#pragma unroll
            for (int q = 0; q < 2*64*P/kPencilThreads; ++q) {
                int const c = q*kPencilThreads + tid, row = c/P, part = c % P;
                copy_async<A>(reinterpret_cast<T*>(dst + row*16) + part*E, src + row*64 + part*E);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto land = [&]() {                                        // all copies, everybody's
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
    };
    auto phase = [&](V v, T pr, T pi) {
        return vfma(vdup(pr), v, vmul(vdup(pl ? pi : -pi), __shfl_xor_sync(0xffffffffu, v, 16)));
    };
    auto turn = [&](int slot, T const (&ph)[2]) {              // Bloch phase of a staged halo cube
#pragma unroll
        for (int i = 0; i < 16; ++i) mine[slot*SLOT + i*16] = phase(mine[slot*SLOT + i*16], ph[0], ph[1]);
    };
    auto base = [&](int32_t e) {                               // this thread's plane of neighbour e
        T const *p = (-1 == e) ? zero : x + size_t(nbr_block(e))*kBlockReals;
        return reinterpret_cast<V const*>(p + lo) + zq*16*S;
    };
    V const cx1 = vdup(a.st.c[0][1]), cx2 = vdup(a.st.c[0][2]), cx3 = vdup(a.st.c[0][3]), cx4 = vdup(a.st.c[0][4]);
    V const cy1 = vdup(a.st.c[1][1]), cy2 = vdup(a.st.c[1][2]), cy3 = vdup(a.st.c[1][3]), cy4 = vdup(a.st.c[1][4]);
    V const cz1 = vdup(a.st.c[2][1]), cz2 = vdup(a.st.c[2][2]), cz3 = vdup(a.st.c[2][3]), cz4 = vdup(a.st.c[2][4]);
    V const cx[5] = {V(0), cx1, cx2, cx3, cx4}, cy[5] = {V(0), cy1, cy2, cy3, cy4}, cz[5] = {V(0), cz1, cz2, cz3, cz4};
    V const c0 = vdup(a.st.c[0][0] + a.st.c[1][0] + a.st.c[2][0]);
    V const eim = vdup(pl ? -a.E_im : a.E_im);                 // re: + Im(E) im, im: - Im(E) re
    __syncthreads();                                           // code[] complete
    fetch(0, zleft); fetch(1, code[0][0]); fetch(2, code[0][6]);
    land();
    if (zleft < -1) turn(0, a.ph[2][0]);
    if (code[0][6] < -1) turn(2, a.ph[2][1]);
    if (zleft < -1 || code[0][6] < -1) __syncthreads();
    int sp = 0, sc = 1, sn = 2;
    for (int k = 0; k < n; ++k) {
        int32_t const exm = code[k][1], exp_ = code[k][2], eym = code[k][3], eyp = code[k][4], iloc = code[k][5];
        V const *pxm = base(exm), *pxp = base(exp_), *pym = base(eym), *pyp = base(eyp);
        T const *pot = ((iloc < 0) ? zero : Vcell + size_t(iloc)*64) + zq*16;
        // the rows of the x-neighbours, requested before the z-stencil and its barrier
        V xm[16], xp[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) { xm[i] = lane_load<A>(pxm + i*S); xp[i] = lane_load<A>(pxp + i*S); }
        V cur[16], acc[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) cur[i] = mine[sc*SLOT + i*16];
        // potential and centre; the other plane of the own points from the partner lane
#pragma unroll
        for (int i = 0; i < 16; ++i)
            acc[i] = vfma(c0, cur[i], vfma(vdup(__ldg(pot + i) - a.E_re), cur[i],
                                           vmul(eim, __shfl_xor_sync(0xffffffffu, cur[i], 16))));
        // z-stencil from the three staged cubes
#pragma unroll
        for (int d = 1; d <= 4; ++d) {
            int const zm = zq - d, zp = zq + d;
            V const *m = slots + ((zm < 0) ? sp : sc)*SLOT + (pl*64 + (zm & 3)*16)*16 + j;
            V const *p = slots + ((zp > 3) ? sn : sc)*SLOT + (pl*64 + (zp & 3)*16)*16 + j;
#pragma unroll
            for (int i = 0; i < 16; ++i) acc[i] = vfma(cz[d], vadd(m[i*16], p[i*16]), acc[i]);
        }
        __syncthreads();                                       // the previous cube is done with
        if (k + 1 < n) fetch(sp, code[k + 1][6]);              // arrives during the rest of this step
        // y-stencil inside the cube
#pragma unroll
        for (int yy = 0; yy < 4; ++yy)
#pragma unroll
            for (int yo = 0; yo < 4; ++yo) {
                if (yo == yy) continue;
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[yy*4 + i] = vfma(cy[(yo > yy) ? yo - yy : yy - yo], cur[yo*4 + i], acc[yy*4 + i]);
            }
        // x-stencil: the rows of the x-neighbours at (zq, yy)
#pragma unroll
        for (int yy = 0; yy < 4; ++yy) {
            V l[12];
#pragma unroll
            for (int i = 0; i < 4; ++i) { l[i] = xm[yy*4 + i]; l[4 + i] = cur[yy*4 + i]; l[8 + i] = xp[yy*4 + i]; }
            if (exm < -1) {
#pragma unroll
                for (int i = 0; i < 4; ++i) l[i] = phase(l[i], a.ph[0][0][0], a.ph[0][0][1]);
            }
            if (exp_ < -1) {
#pragma unroll
                for (int i = 8; i < 12; ++i) l[i] = phase(l[i], a.ph[0][1][0], a.ph[0][1][1]);
            }
#pragma unroll
            for (int d = 1; d <= 4; ++d)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[yy*4 + i] = vfma(cx[d], vadd(l[4 + i - d], l[4 + i + d]), acc[yy*4 + i]);
        }
        // y-neighbour cubes: row yo of y- sits at y = yo - 4, row yo of y+ at y = yo + 4
#pragma unroll
        for (int yo = 0; yo < 4; ++yo) {
            V ym[4], yp[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) { ym[i] = lane_load<A>(pym + (yo*4 + i)*S); yp[i] = lane_load<A>(pyp + (yo*4 + i)*S); }
            if (eym < -1) {
#pragma unroll
                for (int i = 0; i < 4; ++i) ym[i] = phase(ym[i], a.ph[1][0][0], a.ph[1][0][1]);
            }
            if (eyp < -1) {
#pragma unroll
                for (int i = 0; i < 4; ++i) yp[i] = phase(yp[i], a.ph[1][1][0], a.ph[1][1][1]);
            }
#pragma unroll
            for (int yy = 0; yy < 4; ++yy) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (yy <= yo) acc[yy*4 + i] = vfma(cy[(yy - yo + 4) & 7], ym[i], acc[yy*4 + i]);
                    if (yy >= yo) acc[yy*4 + i] = vfma(cy[(yo + 4 - yy) & 7], yp[i], acc[yy*4 + i]);
                }
            }
        }
        V *yb = reinterpret_cast<V*>(y + size_t(code[k][0])*kBlockReals + lo) + zq*16*S;
#pragma unroll
        for (int i = 0; i < 16; ++i) lane_store<A>(yb + i*S, acc[i]);
        if (k + 1 < n) {
            land();                                            // the cube after the next one
            if (code[k + 1][6] < -1) { turn(sp, a.ph[2][1]); __syncthreads(); }
        }
        int const t = sp; sp = sc; sc = sn; sn = t;            // rotate the z-slots
    }
}

// ---------------------------------------------------------------- generic local path

// y = (V - E) x for every block (include/green_potential.hxx:15-139, collinear)
template <typename T>
__global__ void __launch_bounds__(256)
potential_kernel(T *__restrict__ y, T const *__restrict__ x, int32_t const *__restrict__ veff,
                 T const *__restrict__ Vcell, uint32_t nnzb, LocalArgs<T> const a0)
{
    for (uint32_t b = blockIdx.x; b < nnzb; b += gridDim.x) {
        LocalArgs<T> a = a0;
        if (!line_args(a, int32_t(b))) continue;          // uniform: the CTA works on block b
        T const Er = a.E_re, Ei = a.E_im;
        int32_t const iloc = veff[b];
        T const *xb = x + size_t(b)*kBlockReals;
        T *yb = y + size_t(b)*kBlockReals;
        for (int t = threadIdx.x; t < 4096; t += blockDim.x) {
            int const i = t >> 6;
            T const Vt = ((iloc < 0) ? T(0) : Vcell[size_t(iloc)*64 + i]) - Er;
            T const xr = xb[t], xi = xb[4096 + t];
            yb[t] = Vt*xr + Ei*xi;
            yb[4096 + t] = Vt*xi - Ei*xr;
        }
    }
}

// y += T_dd x along the lists of one direction, or y = (V - E) x + T_dd x (FIRST: the first direction,
// which then needs no pass for the potential and does not read y); NH halo cubes (1: 9-point, 2:
// 17-point stencil).  One CTA per (list, cross-section row i16), 64 threads = columns, each for re
// and im.  The cube that enters the window next, and y, are requested before the current cube is
// computed.  Measured on the isolated 12^3 cell (16th order, 4,336 blocks, FP64; 284 MB a vector):
// 114 us for the first direction and 155 us for each other one, against 99 us for a pass of the
// potential and 208 us per direction.
template <typename T>
struct Coef17 { T c[9]; };

template <typename T, int NH, bool FIRST>
__global__ void __launch_bounds__(64)
kinetic_list_kernel(T *__restrict__ y, T const *__restrict__ x, uint32_t const *__restrict__ lstart,
                    int32_t const *__restrict__ lists, int stride, Coef17<T> const coef, int dd,
                    int32_t const *__restrict__ veff, T const *__restrict__ Vcell, LocalArgs<T> a)
{
    constexpr int W = 4*(2*NH + 1);   // window points: NH cubes left, current, NH right
    constexpr int R = 4*NH;           // stencil reach in points
    int const i16 = blockIdx.y, col = threadIdx.x;
    int const base = (16 == stride) ? i16 : ((4 == stride) ? (16*(i16 >> 2) + (i16 & 3)) : 4*i16);
    int32_t const *L = lists + lstart[blockIdx.x];
    int const n = int(lstart[blockIdx.x + 1] - lstart[blockIdx.x]) - 8;   // 4 halo entries at both ends
    if (n < 1 || !line_args(a, L[4] - 1)) return;       // uniform: empty list, or a retired source
    T const plr = a.ph[dd][0][0], pli = a.ph[dd][0][1], prr = a.ph[dd][1][0], pri = a.ph[dd][1][1];
    T c[R + 1];
#pragma unroll
    for (int k = 0; k <= R; ++k) c[k] = coef.c[k];
    T wr[W], wi[W];
    // cube at list position p (0-based among the cubes), with halo handling at both ends
    auto fetch = [&](int p, T (&fr)[4], T (&fi)[4]) {
        int32_t entry = 0; T pr = T(1), pi = T(0);
        if (p >= 0 && p < n) entry = L[4 + p];
        else if (1 == NH && -1 == p) { entry = L[3]; pr = plr; pi = pli; }
        else if (1 == NH && n == p) { entry = L[4 + n]; pr = prr; pi = pri; }
        if (0 == entry) {
#pragma unroll
            for (int i4 = 0; i4 < 4; ++i4) { fr[i4] = T(0); fi[i4] = T(0); }
            return;
        }
        int32_t const b = (entry > 0) ? entry - 1 : -entry - 1;
        T const *xb = x + size_t(b)*kBlockReals + base*64 + col;
#pragma unroll
        for (int i4 = 0; i4 < 4; ++i4) {
            T const r = xb[i4*stride*64], i = xb[4096 + i4*stride*64];
            if (entry < 0) { fr[i4] = pr*r - pi*i; fi[i4] = pr*i + pi*r; }
            else { fr[i4] = r; fi[i4] = i; }
        }
    };
#pragma unroll
    for (int s = 0; s < 2*NH + 1; ++s)
        fetch(s - NH, *reinterpret_cast<T(*)[4]>(&wr[4*s]), *reinterpret_cast<T(*)[4]>(&wi[4*s]));
    for (int k = 0; k < n; ++k) {
        int32_t const b = L[4 + k] - 1;
        T *yb = y + size_t(b)*kBlockReals + base*64 + col;
        T nr[4], ni[4], yr[4], yi[4];
        fetch(k + 1 + NH, nr, ni);                      // arrives while this cube is computed
        if (FIRST) {
            int32_t const iloc = veff[b];
#pragma unroll
            for (int i4 = 0; i4 < 4; ++i4) {
                T const Vt = ((iloc < 0) ? T(0) : Vcell[size_t(iloc)*64 + base + i4*stride]) - a.E_re;
                T const xr = wr[4*NH + i4], xi = wi[4*NH + i4];
                yr[i4] = Vt*xr + a.E_im*xi;
                yi[i4] = Vt*xi - a.E_im*xr;
            }
        } else {
#pragma unroll
            for (int i4 = 0; i4 < 4; ++i4) { yr[i4] = yb[i4*stride*64]; yi[i4] = yb[4096 + i4*stride*64]; }
        }
#pragma unroll
        for (int i4 = 0; i4 < 4; ++i4) {
            int const p = 4*NH + i4;
            T sr = c[0]*wr[p], si = c[0]*wi[p];
#pragma unroll
            for (int d = 1; d <= R; ++d) { sr += c[d]*(wr[p - d] + wr[p + d]); si += c[d]*(wi[p - d] + wi[p + d]); }
            yb[i4*stride*64] = yr[i4] + sr;
            yb[4096 + i4*stride*64] = yi[i4] + si;
        }
#pragma unroll
        for (int q = 0; q < W - 4; ++q) { wr[q] = wr[q + 4]; wi[q] = wi[q + 4]; }
#pragma unroll
        for (int i4 = 0; i4 < 4; ++i4) { wr[W - 4 + i4] = nr[i4]; wi[W - 4 + i4] = ni[i4]; }
    }
}

// ---------------------------------------------------------------- dyadic part

__host__ __device__ constexpr int nsho_c(int L) { return ((L + 1)*(L + 2)*(L + 3))/6; }
__host__ __device__ constexpr int n2ho_c(int L) { return ((L + 1)*(L + 2))/2; }

// Projector tables of one (atom image, target row) slot staged in shared memory: the 1D
// Hermite-Gauss functions H[nu][dir][i4] (unnormalized, H_0 = exp(-xi^2/2) inside the
// projection radius, H_{n+1} = xi H_n - n/2 H_{n-1}, include/green_dyadic.hxx:33-107) and
// the 64-point spherical mask, both precomputed by the plan builder.
template <typename T, int LM>
__device__ __forceinline__ void stage_table(T (*H)[3][4], double const *__restrict__ slot_H, int stride,
                                            uint32_t slot, int lmax, int tid) {
    if (tid < (lmax + 1)*12) (&H[0][0][0])[tid] = T(slot_H[size_t(slot)*stride + tid]);
}

// apc[(i0 + sho)*nrhs + s][reim][j] = sum over the blocks of source s near image a of the
// masked projector functions times x (include/green_dyadic.hxx:112-288), for images whose
// basis size is exactly L (the host launches one grid per distinct L).  Sum-factorized:
// contract x, then y, then z.  One CTA per work item (image, source, chunk of at most 16
// blocks of its list), 128 threads = (reim, column); the chunks of one (image, source) are
// summed with atomics into the zeroed coefficients.
template <typename T, int L>
__global__ void __launch_bounds__(128)
sho_project_kernel(T *__restrict__ apc, T const *__restrict__ x, uint32_t nrhs,
                   uint32_t const *__restrict__ items,
                   uint32_t const *__restrict__ prj_col, uint64_t const *__restrict__ prj_coloff,
                   uint32_t const *__restrict__ prj_slot,
                   double const *__restrict__ slot_H, uint64_t const *__restrict__ slot_mask, int stride,
                   uint32_t const *__restrict__ img_starts)
{
    constexpr int NS = nsho_c(L), N2 = n2ho_c(L);
    __shared__ T Hs[2][L + 1][3][4];
    uint32_t const *item = items + 4*size_t(blockIdx.x);
    uint32_t const a = item[0], s = item[1], k0 = item[2], k1 = item[3];
    int const tid = threadIdx.x;
    int const reim = tid >> 6, j = tid & 63;
    uint64_t const off = prj_coloff[s];
    T acc[NS];
#pragma unroll
    for (int i = 0; i < NS; ++i) acc[i] = T(0);
    int buf = 0;
    for (uint32_t k = k0; k < k1; ++k, buf ^= 1) {
        uint32_t const b = prj_col[off + k];
        uint32_t const slot = prj_slot[off + k];
        stage_table<T, L>(Hs[buf], slot_H, stride, slot, L, tid);
        uint64_t const mask = slot_mask[slot];
        __syncthreads();             // double-buffered tables: one barrier per block
        T (*H)[3][4] = Hs[buf];
        T const *xb = x + size_t(b)*kBlockReals + reim*4096 + j;
        for (int z = 0; z < 4; ++z) {
            if (0 == ((mask >> (16*z)) & 0xffffu)) continue;
            T byx[N2];
#pragma unroll
            for (int i = 0; i < N2; ++i) byx[i] = T(0);
            for (int yy = 0; yy < 4; ++yy) {
                unsigned const row = unsigned(mask >> (16*z + 4*yy)) & 0xfu;
                if (0 == row) continue;
                T ax[L + 1];
#pragma unroll
                for (int i = 0; i <= L; ++i) ax[i] = T(0);
#pragma unroll
                for (int xx = 0; xx < 4; ++xx) {
                    if ((row >> xx) & 1u) {
                        T const ps = xb[((z*4 + yy)*4 + xx)*64];
#pragma unroll
                        for (int ix = 0; ix <= L; ++ix) ax[ix] += ps*H[ix][0][xx];
                    }
                }
#pragma unroll
                for (int iy = 0, iyx = 0; iy <= L; ++iy) {
                    T const hy = H[iy][1][yy];
#pragma unroll
                    for (int ix = 0; ix <= L - iy; ++ix, ++iyx) byx[iyx] += ax[ix]*hy;
                }
            }
#pragma unroll
            for (int iz = 0, sho = 0; iz <= L; ++iz) {
                T const hz = H[iz][2][z];
#pragma unroll
                for (int iy = 0; iy <= L - iz; ++iy) {
                    int const iyx = iy*(2*L + 3 - iy)/2;
#pragma unroll
                    for (int ix = 0; ix <= L - iz - iy; ++ix, ++sho) acc[sho] += byx[iyx + ix]*hz;
                }
            }
        }
    }
    T *out = apc + (size_t(img_starts[a])*nrhs + s)*128 + reim*64 + j;
#pragma unroll
    for (int sho = 0; sho < NS; ++sho) atomicAdd(out + size_t(sho)*nrhs*128, acc[sho]);
}

// aac[(a0 + c)*nrhs + s] = sum over the images i of atom A of phase_i * apc[(i0 + c)*nrhs + s]
// (collect) in double (include/green_dyadic.hxx:600-702).  Grid (nAtoms, nrhs, rows), 64 threads.
// per-source selection of the pair values of a batch plan (image phases and atom matrices
// stored [pair][...]) and the retirement flags (nullptr: every source active)
struct DyadicPairs {
    uint32_t nsrc_pair;              // sources per pair (= nrhs for a one-pair plan)
    size_t img_stride, mat_stride;   // doubles per pair of img_phase and of the atom matrices
    uint8_t const *active;
};

template <typename T>
__global__ void __launch_bounds__(64)
sho_collect_kernel(double *__restrict__ aac, T const *__restrict__ apc, uint32_t nrhs,
                   uint32_t const *__restrict__ atom_starts, int8_t const *__restrict__ atom_lmax,
                   uint32_t const *__restrict__ sum_start, uint32_t const *__restrict__ sum_col,
                   uint32_t const *__restrict__ img_starts, double const *__restrict__ img_phase,
                   DyadicPairs const bp)
{
    int const A = blockIdx.x, s = blockIdx.y, j = threadIdx.x;
    if (bp.active && !bp.active[s]) return;
    img_phase += (s/bp.nsrc_pair)*bp.img_stride;
    int const nc = nsho_c(atom_lmax[A]);
    size_t const a0 = atom_starts[A];
    for (int c = blockIdx.z; c < nc; c += gridDim.z) {
        double re = 0, im = 0;
        for (uint32_t k = sum_start[A]; k < sum_start[A + 1]; ++k) {
            uint32_t const i = sum_col[k];
            double const pr = img_phase[4*i], pi = img_phase[4*i + 1];
            T const *src = apc + ((size_t(img_starts[i]) + c)*nrhs + s)*128;
            double const xr = double(src[j]), xi = double(src[64 + j]);
            re += pr*xr - pi*xi;
            im += pr*xi + pi*xr;
        }
        double *dst = aac + ((a0 + c)*nrhs + s)*128;
        dst[j] = re; dst[64 + j] = im;
    }
}

constexpr int kMulRows = 8;

// out[(a0 + i)*nrhs + s] = sum_k M_A[i][k] in[(a0 + k)*nrhs + s], complex, accumulated in
// double (include/green_dyadic.hxx:740-826).  Grid (nAtoms, nrhs, groups of 8 rows), 64 threads.
template <typename Tin, typename Tout>
__global__ void __launch_bounds__(64)
sho_mul_kernel(Tout *__restrict__ out, Tin const *__restrict__ in, uint32_t nrhs,
               uint32_t const *__restrict__ atom_starts, int8_t const *__restrict__ atom_lmax,
               double const *__restrict__ mats, uint32_t const *__restrict__ mat_off, DyadicPairs const bp)
{
    int const A = blockIdx.x, s = blockIdx.y, j = threadIdx.x;
    if (bp.active && !bp.active[s]) return;
    mats += (s/bp.nsrc_pair)*bp.mat_stride;
    int const nc = nsho_c(atom_lmax[A]);
    size_t const a0 = atom_starts[A];
    double const *Mr = mats + mat_off[A], *Mi = Mr + nc*nc;
    constexpr int R = kMulRows;                // output rows per pass: each input value is loaded once per R rows
    for (int i0 = blockIdx.z*R; i0 < nc; i0 += gridDim.z*R) {
        double re[R], im[R];
#pragma unroll
        for (int r = 0; r < R; ++r) { re[r] = 0; im[r] = 0; }
        for (int k = 0; k < nc; ++k) {
            Tin const *src = in + ((a0 + k)*nrhs + s)*128;
            double const xr = double(src[j]), xi = double(src[64 + j]);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                int const i = (i0 + r < nc) ? i0 + r : nc - 1;   // clamped rows are not stored
                double const mr = __ldg(Mr + i*nc + k), mi = __ldg(Mi + i*nc + k);
                re[r] += mr*xr - mi*xi;
                im[r] += mr*xi + mi*xr;
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (i0 + r >= nc) break;
            Tout *dst = out + ((a0 + i0 + r)*nrhs + s)*128;
            dst[j] = Tout(re[r]); dst[64 + j] = Tout(im[r]);
        }
    }
}

// cad[(i0 + c)*nrhs + s] = conj(phase_i) * cadd[(a0 + c)*nrhs + s] for every image i of atom A
// (broadcast, include/green_dyadic.hxx:683-694).  Grid (nAtoms, nrhs, rows), 64 threads.
template <typename T>
__global__ void __launch_bounds__(64)
sho_broadcast_kernel(T *__restrict__ cad, double const *__restrict__ cadd, uint32_t nrhs,
                     uint32_t const *__restrict__ atom_starts, int8_t const *__restrict__ atom_lmax,
                     uint32_t const *__restrict__ sum_start, uint32_t const *__restrict__ sum_col,
                     uint32_t const *__restrict__ img_starts, double const *__restrict__ img_phase,
                     DyadicPairs const bp)
{
    int const A = blockIdx.x, s = blockIdx.y, j = threadIdx.x;
    if (bp.active && !bp.active[s]) return;
    img_phase += (s/bp.nsrc_pair)*bp.img_stride;
    int const nc = nsho_c(atom_lmax[A]);
    size_t const a0 = atom_starts[A];
    for (uint32_t k = sum_start[A]; k < sum_start[A + 1]; ++k) {
        uint32_t const i = sum_col[k];
        double const pr = img_phase[4*i], pi = -img_phase[4*i + 1];
        for (int c = blockIdx.z; c < nc; c += gridDim.z) {
            double const *src = cadd + ((a0 + c)*nrhs + s)*128;
            double const xr = src[j], xi = src[64 + j];
            T *dst = cad + ((size_t(img_starts[i]) + c)*nrhs + s)*128;
            dst[j] = T(pr*xr - pi*xi);
            dst[64 + j] = T(pr*xi + pi*xr);
        }
    }
}

// The atom-matrix chain in one kernel (collect, multiply, broadcast of the three kernels above),
// per (atom, source, half of the 64 columns): the coefficients of the atom's images summed with
// their Bloch phases into shared memory, multiplied by M_A (complex, FP64) and written to every
// image with the conjugate phase.  M_A is copied to shared memory while the images are summed (read
// from global memory element by element, every fourth one waited for the L2).  Warp g of the eight
// works on the rows g, g + 8, ... all at once, lane j on column half*32 + j.  Plans without periodic
// images take no phases (the reference's direct path).  nSHO <= 56.
//
// Measured against rows one after the other on 4 warps with M_A from global memory: 8 atoms, 4
// sources 98 -> 22 us; 64 atoms, 8 sources 147 -> 84 us; 193 atoms, 32 sources 1188 -> 646 us.
// What bounds it: the latency of the image loads (two CTAs per SM: 77 KB of shared memory).
constexpr int kAtomRows = 56, kAtomWarps = 8;
int atom_smem(int lmax) { int const n = nsho_c(lmax); return 2*n*n*8 + 2*n*32*8; }

template <typename T>
__global__ void __launch_bounds__(32*kAtomWarps)
sho_atom_kernel(T *__restrict__ cad, T const *__restrict__ apc, uint32_t nrhs,
                int8_t const *__restrict__ atom_lmax, uint32_t const *__restrict__ sum_start,
                uint32_t const *__restrict__ sum_col, uint32_t const *__restrict__ img_starts,
                double const *__restrict__ img_phase, double const *__restrict__ mats,
                uint32_t const *__restrict__ mat_off, int use_phase, DyadicPairs const bp)
{
    constexpr int RW = kAtomRows/kAtomWarps;          // rows per warp
    constexpr int kImg = 32;                          // images of the atom staged in shared memory
    extern __shared__ __align__(16) double atom_raw[];
    __shared__ uint32_t simg[kImg];
    __shared__ double sph[kImg][2];
    int const A = blockIdx.x, s = blockIdx.y, half = blockIdx.z;
    int const tid = threadIdx.x, j = tid & 31, g = tid >> 5, col = half*32 + j;
    if (bp.active && !bp.active[s]) return;
    img_phase += (s/bp.nsrc_pair)*bp.img_stride;
    mats += (s/bp.nsrc_pair)*bp.mat_stride;
    int const nc = nsho_c(atom_lmax[A]);
    double *M = atom_raw;                             // [2][nc][nc]
    double *x = atom_raw + 2*nc*nc;                   // [nc][2][32]
    for (int q = tid; q < nc*nc; q += 32*kAtomWarps)  // 2 nc^2 doubles, 16 bytes at a time
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::
                     "r"(uint32_t(__cvta_generic_to_shared(M + 2*q))), "l"(mats + mat_off[A] + 2*size_t(q)) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
    uint32_t const k0 = sum_start[A], k1 = sum_start[A + 1];
    // the atom's images (their coefficient start and phase) once, instead of a chain of three
    // dependent loads per row and image
    for (uint32_t k = k0 + tid; k < k1 && k < k0 + kImg; k += 32*kAtomWarps) {
        uint32_t const i = sum_col[k];
        simg[k - k0] = img_starts[i];
        sph[k - k0][0] = img_phase[4*i]; sph[k - k0][1] = img_phase[4*i + 1];
    }
    __syncthreads();
    auto image = [&](uint32_t k, uint32_t &start, double &pr, double &pi) {
        if (k - k0 < uint32_t(kImg)) { start = simg[k - k0]; pr = sph[k - k0][0]; pi = sph[k - k0][1]; }
        else { uint32_t const i = sum_col[k]; start = img_starts[i]; pr = img_phase[4*i]; pi = img_phase[4*i + 1]; }
    };
    size_t const stride = size_t(nrhs)*128;
    double re[RW], im[RW];
#pragma unroll
    for (int r = 0; r < RW; ++r) re[r] = im[r] = 0;
#pragma unroll 2
    for (uint32_t k = k0; k < k1; ++k) {
        uint32_t start; double pr, pi;
        image(k, start, pr, pi);
        T const *src = apc + (size_t(start)*nrhs + s)*128 + col;
        T xr[RW], xi[RW];
#pragma unroll
        for (int r = 0; r < RW; ++r) {
            int const c = min(g + r*kAtomWarps, nc - 1);   // clamped rows are not stored
            xr[r] = src[c*stride]; xi[r] = src[c*stride + 64];
        }
#pragma unroll
        for (int r = 0; r < RW; ++r) {
            double const a = double(xr[r]), b = double(xi[r]);
            if (use_phase) {
                re[r] += pr*a - pi*b;
                im[r] += pr*b + pi*a;
            } else {
                re[r] += a; im[r] += b;
            }
        }
    }
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        int const c = g + r*kAtomWarps;
        if (c < nc) { x[c*64 + j] = re[r]; x[c*64 + 32 + j] = im[r]; }
        re[r] = im[r] = 0;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    double const *Mr[RW];
#pragma unroll
    for (int r = 0; r < RW; ++r) Mr[r] = M + min(g + r*kAtomWarps, nc - 1)*nc;
    int const plane = nc*nc;
#pragma unroll 2
    for (int k = 0; k < nc; ++k) {
        double const a = x[k*64 + j], b = x[k*64 + 32 + j];
#pragma unroll
        for (int r = 0; r < RW; ++r) {
            double const mr = Mr[r][k], mi = Mr[r][plane + k];
            re[r] += mr*a - mi*b;
            im[r] += mr*b + mi*a;
        }
    }
    for (uint32_t k = k0; k < k1; ++k) {
        uint32_t start; double pr, pi;
        image(k, start, pr, pi);
        pi = -pi;
        T *dst = cad + (size_t(start)*nrhs + s)*128 + col;
#pragma unroll
        for (int r = 0; r < RW; ++r) {
            int const c = g + r*kAtomWarps;
            if (c >= nc) break;                       // uniform over the warp
            if (use_phase) {
                dst[c*stride] = T(pr*re[r] - pi*im[r]);
                dst[c*stride + 64] = T(pr*im[r] + pi*re[r]);
            } else {
                dst[c*stride] = T(re[r]); dst[c*stride + 64] = T(im[r]);
            }
        }
    }
}

// y[b] += sum over the images a near block b of the masked projector functions times
// cad[a, rhs(b)] (include/green_dyadic.hxx:325-518); sum-factorized over z, y, x.
// One CTA per block, 128 threads = (reim, column); only masked points are written.
template <typename T>
__global__ void __launch_bounds__(128)
sho_add_kernel(T *__restrict__ y, T const *__restrict__ cad, uint32_t nrhs, uint32_t nnzb,
               uint16_t const *__restrict__ colIndex, uint32_t const *__restrict__ add_start,
               uint32_t const *__restrict__ add_col, uint32_t const *__restrict__ add_slot,
               double const *__restrict__ slot_H, uint64_t const *__restrict__ slot_mask, int stride,
               int8_t const *__restrict__ img_lmax, uint32_t const *__restrict__ img_starts)
{
    constexpr int LM = 7;
    __shared__ T Hs[2][LM + 1][3][4];
    uint32_t const b = blockIdx.x;
    if (add_start[b] >= add_start[b + 1]) return;
    int const tid = threadIdx.x, reim = tid >> 6, j = tid & 63;
    uint32_t const s = colIndex[b];
    T acc[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) acc[i] = T(0);
    uint64_t mask_all = 0;
    int buf = 0;
    for (uint32_t k = add_start[b]; k < add_start[b + 1]; ++k, buf ^= 1) {
        uint32_t const a = add_col[k], slot = add_slot[k];
        int const lmax = img_lmax[a];
        stage_table<T, LM>(Hs[buf], slot_H, stride, slot, lmax, tid);
        uint64_t const mask = slot_mask[slot];
        __syncthreads();
        if (!mask) continue;
        mask_all |= mask;
        T (*H)[3][4] = Hs[buf];
        T const *c = cad + (size_t(img_starts[a])*nrhs + s)*128 + reim*64 + j;
        int sho = 0;
        for (int iz = 0; iz <= lmax; ++iz) {
            T byx[4][4];
#pragma unroll
            for (int yy = 0; yy < 4; ++yy)
#pragma unroll
                for (int xx = 0; xx < 4; ++xx) byx[yy][xx] = T(0);
            for (int iy = 0; iy <= lmax - iz; ++iy) {
                T ax[4] = {T(0), T(0), T(0), T(0)};
                for (int ix = 0; ix <= lmax - iz - iy; ++ix, ++sho) {
                    T const ca = c[size_t(sho)*nrhs*128];
#pragma unroll
                    for (int xx = 0; xx < 4; ++xx) ax[xx] += H[ix][0][xx]*ca;
                }
#pragma unroll
                for (int yy = 0; yy < 4; ++yy) {
                    T const hy = H[iy][1][yy];
#pragma unroll
                    for (int xx = 0; xx < 4; ++xx) byx[yy][xx] += hy*ax[xx];
                }
            }
#pragma unroll
            for (int z = 0; z < 4; ++z) {
                T const hz = H[iz][2][z];
#pragma unroll
                for (int yy = 0; yy < 4; ++yy)
#pragma unroll
                    for (int xx = 0; xx < 4; ++xx) {
                        int const p = (z*4 + yy)*4 + xx;
                        if ((mask >> p) & 1) acc[p] += hz*byx[yy][xx];
                    }
            }
        }
    }
    T *yb = y + size_t(b)*kBlockReals + reim*4096 + j;
#pragma unroll
    for (int p = 0; p < 64; ++p) if ((mask_all >> p) & 1) yb[p*64] += acc[p];
}

// grids of the three-kernel chain: the rows of an atom over the z-index, 4 rows per CTA (a plan of 64
// atoms and one source would keep 64 CTAs busy with 56 rows each: 239 us against 23 for the collect
// kernel)
dim3 row_grid(DevicePlan const &dp) { return dim3(dp.nAtoms, dp.nCols, unsigned((nsho_c(std::max(dp.lmax_max, 0)) + 3)/4)); }
dim3 mul_grid(DevicePlan const &dp) { return dim3(dp.nAtoms, dp.nCols, unsigned((nsho_c(std::max(dp.lmax_max, 0)) + kMulRows - 1)/kMulRows)); }

DyadicPairs dyadic_pairs(DevicePlan const &dp) {
    DyadicPairs bp;
    bp.nsrc_pair = dp.nsrc_pair ? dp.nsrc_pair : std::max(1u, dp.nCols);
    bp.img_stride = (dp.npairs > 1) ? size_t(dp.nAI)*4 : 0;
    bp.mat_stride = (dp.npairs > 1) ? dp.mat_stride : 0;
    bp.active = dp.retire ? dptr<uint8_t>(dp.src_active) : nullptr;
    return bp;
}

template <typename T> T const *vcell(DevicePlan &dp);
template <> double const *vcell<double>(DevicePlan &dp) { return dptr<double>(dp.Vcell64); }
template <> float const *vcell<float>(DevicePlan &dp) { return dptr<float>(dp.Vcell32); }

template <typename T, int L>
void launch_project_L(DevicePlan &dp, T const *x, cudaStream_t st) {
    auto const &g = dp.prj_items[L];
    if (0 == g.count) return;
    sho_project_kernel<T, L><<<g.count, 128, 0, st>>>(
        dptr<T>(dp.apc), x, dp.nCols, dptr<uint32_t>(g.items),
        dptr<uint32_t>(dp.prj_col), dptr<uint64_t>(dp.prj_coloff),
        dptr<uint32_t>(dp.prj_slot), dptr<double>(dp.slot_H), dptr<uint64_t>(dp.slot_mask), dp.table_stride,
        dptr<uint32_t>(dp.img_starts));
        count_launch();
}

} // namespace

bool prepare_local_kernels() {
    // the pencil kernel's three z-slots are 48 KB of dynamic shared memory beside its static part
    A43G_CUDA_TRY(cudaFuncSetAttribute(local_pencil_kernel<float, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPencilSmem));
    A43G_CUDA_TRY(cudaFuncSetAttribute(local_pencil_kernel<float, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPencilSmem));
    A43G_CUDA_TRY(cudaFuncSetAttribute(local_pencil_kernel<float, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPencilSmem));
    A43G_CUDA_TRY(cudaFuncSetAttribute(local_pencil_kernel<double, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPencilSmem));
    A43G_CUDA_TRY(cudaFuncSetAttribute(local_pencil_kernel<double, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPencilSmem));
    A43G_CUDA_TRY(cudaFuncSetAttribute(sho_atom_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, atom_smem(5)));
    A43G_CUDA_TRY(cudaFuncSetAttribute(sho_atom_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, atom_smem(5)));
    return true;
}

// kernel arguments of the local part: stencil, energy and phases of a one-pair plan, or the
// per-pair table of a batch plan; the source flags when some sources are retired
template <typename T>
LocalArgs<T> local_args(DevicePlan const &dp) {
    LocalArgs<T> a;
    a.st = make_stencil9<T>(dp);
    a.E_re = T(dp.E_re); a.E_im = T(dp.E_im);
    for (int d = 0; d < 3; ++d) for (int s = 0; s < 2; ++s) for (int c = 0; c < 2; ++c) a.ph[d][s][c] = T(dp.phase[d][s][c]);
    bool const batch = dp.npairs > 1;
    a.pairs = batch ? dptr<PairArgs<T>>(sizeof(T) == 8 ? dp.pair_args64 : dp.pair_args32) : nullptr;
    a.active = dp.retire ? dptr<uint8_t>(dp.src_active) : nullptr;
    a.colindx = (batch || a.active) ? dptr<uint16_t>(dp.colindx) : nullptr;
    a.nsrc_pair = dp.nsrc_pair ? dp.nsrc_pair : dp.nCols;
    return a;
}

template <typename T>
bool launch_local(DevicePlan &dp, T *y, T const *x, cudaStream_t st) {
    if (0 == dp.nnzb) return true;
    LocalArgs<T> a = local_args<T>(dp);
    if (dp.fused_local) {
        constexpr int S = (sizeof(T) == 8) ? 8 : 16;
        unsigned const nblk = dp.nlists[2]*(64/S);
        // the pencils hold the codes of a line; the rows kernel takes longer lines
        bool const pencils = !dp.local_rows && dp.max_zline <= kMaxLine;
        if (nblk && pencils) {
            auto *kernel = vectors_aligned(x, y, 16) ? local_pencil_kernel<T, 16> :
                           vectors_aligned(x, y, 8) ? local_pencil_kernel<T, 8> : local_pencil_kernel<T, int(sizeof(T))>;
            kernel<<<dp.nlists[2]*(unsigned(sizeof(T))/2), kPencilThreads, kPencilSmem, st>>>(y, x,
                dptr<uint32_t>(dp.lists_start[2]), dptr<int32_t>(dp.lists[2]), dptr<int32_t>(dp.nbr),
                dptr<int32_t>(dp.veff_index), vcell<T>(dp), dptr<T>(dp.zero_block), a);
            count_launch();
        } else if (nblk) {
            local_fused_kernel<T, S><<<nblk, S*16, 0, st>>>(y, x, dptr<uint32_t>(dp.lists_start[2]),
                dptr<int32_t>(dp.lists[2]), dptr<int32_t>(dp.nbr), dptr<int32_t>(dp.veff_index), vcell<T>(dp), a);
            count_launch();
        }
    } else {
        // every block lies on one line of each direction, so the first direction with a kinetic term
        // writes all of y
        bool first = true;
        for (int d = 0; d < 3; ++d) {
            int const nFD = dp.FD_range[d];
            if (nFD < 1 || 0 == dp.nlists[d]) continue;
            dim3 const grid(dp.nlists[d], 16);
            // 8th order {-14350, 8064, -1008, 128, -9}/5040 or 16th order
            // {-924708642, 538137600, -94174080, 22830080, -5350800, 1053696, -156800, 15360, -735}/302702400,
            // times -1/(2h^2) (include/green_kinetic.hxx:37-42, 215-225)
            Coef17<T> coef;
            if (8 == nFD) {
                double const w[9] = {-924708642, 538137600, -94174080, 22830080, -5350800, 1053696, -156800, 15360, -735};
                double const norm = dp.prefactor[d]/302702400.;
                for (int k = 0; k < 9; ++k) coef.c[k] = T(w[k]*norm);
            } else {
                double const w[5] = {-14350, 8064, -1008, 128, -9};
                double const norm = dp.prefactor[d]/5040.;
                for (int k = 0; k < 9; ++k) coef.c[k] = T(k < 5 ? w[k]*norm : 0.0);
            }
            auto *kernel = (8 == nFD) ? (first ? kinetic_list_kernel<T, 2, true> : kinetic_list_kernel<T, 2, false>)
                                      : (first ? kinetic_list_kernel<T, 1, true> : kinetic_list_kernel<T, 1, false>);
            kernel<<<grid, 64, 0, st>>>(y, x, dptr<uint32_t>(dp.lists_start[d]), dptr<int32_t>(dp.lists[d]), 1 << (2*d),
                                        coef, d, dptr<int32_t>(dp.veff_index), vcell<T>(dp), a);
            first = false;
            count_launch();
        }
        if (first) {                                    // no kinetic term at all
            unsigned const nb = std::min<uint32_t>(dp.nnzb, 148u*16);
            potential_kernel<T><<<nb, 256, 0, st>>>(y, x, dptr<int32_t>(dp.veff_index), vcell<T>(dp), dp.nnzb, a);
            count_launch();
        }
    }
    A43G_CUDA_TRY(cudaGetLastError());
    return true;
}

template <typename T>
bool launch_dyadic(DevicePlan &dp, T *y, T const *x, uint16_t const *colIndex, cudaStream_t st) {
    if (dp.nAI < 1 || dp.nCols < 1) return true;
    if (!ensure_dyadic_scratch(dp, sizeof(T))) return false;
    // the tensor-core projection stages x with 16-byte copies; the line kernels take 8-byte lanes of x and
    // y, and vectors on 16 bytes; other vectors take the generic kernels
    bool const aligned16 = vectors_aligned(x, x, 16);
    bool const tc = (sizeof(T) == 4) && dp.use_tc && dp.slot_H32.ptr && aligned16 && tc_projector_supported(dp);
    bool const lines = !tc && vectors_aligned(x, y, 16);
    if (tc) {
        if (!launch_project_tc(dp, (float const*)x, st)) return false;
    } else if (lines) {
        if (!ensure_prj_part(dp, sizeof(T))) return false;
        if (!launch_project_line(dp, dptr<T>(dp.apc), x, sizeof(T) == 8 ? dp.line_tab64.ptr : dp.line_tab32.ptr,
                                 LineScratch{dp.prj_part.ptr, dptr<uint32_t>(dp.prj_line.tickets)}, st)) return false;
    } else {
        // coefficients of images without any block stay zero
        A43G_CUDA_TRY(cudaMemsetAsync(dp.apc.ptr, 0, size_t(dp.ncoeffI)*dp.nCols*128*sizeof(T), st));
        launch_project_L<T, 0>(dp, x, st); launch_project_L<T, 1>(dp, x, st);
        launch_project_L<T, 2>(dp, x, st); launch_project_L<T, 3>(dp, x, st);
        launch_project_L<T, 4>(dp, x, st); launch_project_L<T, 5>(dp, x, st);
        launch_project_L<T, 6>(dp, x, st); launch_project_L<T, 7>(dp, x, st);
    }
    dim3 const ga = row_grid(dp), gm = mul_grid(dp);
    if (one_atom_kernel(dp)) {
        sho_atom_kernel<T><<<dim3(dp.nAtoms, dp.nCols, 2), 32*kAtomWarps, atom_smem(dp.lmax_max), st>>>(dptr<T>(dp.cad), dptr<T>(dp.apc), dp.nCols,
            dptr<int8_t>(dp.atom_lmax), dptr<uint32_t>(dp.sum_start), dptr<uint32_t>(dp.sum_col),
            dptr<uint32_t>(dp.img_starts), dptr<double>(dp.img_phase), dptr<double>(dp.atom_mat),
            dptr<uint32_t>(dp.atom_mat_off), dp.nAI > dp.nAtoms ? 1 : 0, dyadic_pairs(dp));
        count_launch();
    } else if (dp.nAI > dp.nAtoms) {
        sho_collect_kernel<T><<<ga, 64, 0, st>>>(dptr<double>(dp.aac), dptr<T>(dp.apc), dp.nCols,
            dptr<uint32_t>(dp.atom_starts), dptr<int8_t>(dp.atom_lmax), dptr<uint32_t>(dp.sum_start),
            dptr<uint32_t>(dp.sum_col), dptr<uint32_t>(dp.img_starts), dptr<double>(dp.img_phase), dyadic_pairs(dp));
        count_launch();
        sho_mul_kernel<double, double><<<gm, 64, 0, st>>>(dptr<double>(dp.cadd), dptr<double>(dp.aac), dp.nCols,
            dptr<uint32_t>(dp.atom_starts), dptr<int8_t>(dp.atom_lmax), dptr<double>(dp.atom_mat), dptr<uint32_t>(dp.atom_mat_off), dyadic_pairs(dp));
        count_launch();
        sho_broadcast_kernel<T><<<ga, 64, 0, st>>>(dptr<T>(dp.cad), dptr<double>(dp.cadd), dp.nCols,
            dptr<uint32_t>(dp.atom_starts), dptr<int8_t>(dp.atom_lmax), dptr<uint32_t>(dp.sum_start),
            dptr<uint32_t>(dp.sum_col), dptr<uint32_t>(dp.img_starts), dptr<double>(dp.img_phase), dyadic_pairs(dp));
        count_launch();
    } else {
        sho_mul_kernel<T, T><<<gm, 64, 0, st>>>(dptr<T>(dp.cad), dptr<T>(dp.apc), dp.nCols,
            dptr<uint32_t>(dp.atom_starts), dptr<int8_t>(dp.atom_lmax), dptr<double>(dp.atom_mat), dptr<uint32_t>(dp.atom_mat_off), dyadic_pairs(dp));
        count_launch();
    }
    if (tc) {
        if (!launch_add_tc(dp, (float*)y, colIndex, st)) return false;
    } else if (lines) {
        if (!launch_add_line(dp, y, dptr<T>(dp.cad), colIndex, st)) return false;
    } else {
        sho_add_kernel<T><<<dp.nnzb, 128, 0, st>>>(y, dptr<T>(dp.cad), dp.nCols, dp.nnzb, colIndex,
            dptr<uint32_t>(dp.add_start), dptr<uint32_t>(dp.add_col), dptr<uint32_t>(dp.add_slot),
            dptr<double>(dp.slot_H), dptr<uint64_t>(dp.slot_mask), dp.table_stride,
            dptr<int8_t>(dp.img_lmax), dptr<uint32_t>(dp.img_starts));
        count_launch();
    }
    A43G_CUDA_TRY(cudaGetLastError());
    return true;
}

template <typename T>
bool launch_action(DevicePlan &dp, T *y, T const *x, uint16_t const *colIndex, cudaStream_t st) {
    if (!launch_local<T>(dp, y, x, st)) return false;
    return launch_dyadic<T>(dp, y, x, colIndex, st);
}

// ---------------------------------------------------------------- pieces of the dyadic part with
// caller-given buffers and tables (FP64), for the vector-Jacobian products

namespace {
template <typename T, int L>
void project_into_L(DevicePlan &dp, T *apc, T const *x, double const *table, cudaStream_t st) {
    auto const &g = dp.prj_items[L];
    if (0 == g.count) return;
    sho_project_kernel<T, L><<<g.count, 128, 0, st>>>(
        apc, x, dp.nCols, dptr<uint32_t>(g.items), dptr<uint32_t>(dp.prj_col), dptr<uint64_t>(dp.prj_coloff),
        dptr<uint32_t>(dp.prj_slot), table, dptr<uint64_t>(dp.slot_mask), dp.table_stride, dptr<uint32_t>(dp.img_starts));
    count_launch();
}

// generic projection (zeroes apc, then atomics per work item) into a caller-given buffer
template <typename T>
bool project_into(DevicePlan &dp, T *apc, T const *x, double const *table, cudaStream_t st) {
    A43G_CUDA_TRY(cudaMemsetAsync(apc, 0, size_t(dp.ncoeffI)*dp.nCols*128*sizeof(T), st));
    project_into_L<T, 0>(dp, apc, x, table, st); project_into_L<T, 1>(dp, apc, x, table, st);
    project_into_L<T, 2>(dp, apc, x, table, st); project_into_L<T, 3>(dp, apc, x, table, st);
    project_into_L<T, 4>(dp, apc, x, table, st); project_into_L<T, 5>(dp, apc, x, table, st);
    project_into_L<T, 6>(dp, apc, x, table, st); project_into_L<T, 7>(dp, apc, x, table, st);
    A43G_CUDA_TRY(cudaGetLastError());
    return true;
}
} // namespace

bool launch_collect_with(DevicePlan &dp, double *aac, double const *apc, double const *img_phase, cudaStream_t st) {
    dim3 const ga = row_grid(dp);
    sho_collect_kernel<double><<<ga, 64, 0, st>>>(aac, apc, dp.nCols, dptr<uint32_t>(dp.atom_starts),
        dptr<int8_t>(dp.atom_lmax), dptr<uint32_t>(dp.sum_start), dptr<uint32_t>(dp.sum_col),
        dptr<uint32_t>(dp.img_starts), img_phase, dyadic_pairs(dp));
    count_launch();
    A43G_CUDA_TRY(cudaGetLastError());
    return true;
}

bool launch_mul_with(DevicePlan &dp, double *out, double const *in, cudaStream_t st) {
    dim3 const gm = mul_grid(dp);
    sho_mul_kernel<double, double><<<gm, 64, 0, st>>>(out, in, dp.nCols, dptr<uint32_t>(dp.atom_starts),
        dptr<int8_t>(dp.atom_lmax), dptr<double>(dp.atom_mat), dptr<uint32_t>(dp.atom_mat_off), dyadic_pairs(dp));
    count_launch();
    A43G_CUDA_TRY(cudaGetLastError());
    return true;
}

// the whole action with the dyadic coefficients in caller-given scratch (generic kernels only)
template <typename T>
bool launch_action_scratch(DevicePlan &dp, T *y, T const *x, uint16_t const *colIndex, cudaStream_t st,
                           DyadicScratch const &sc) {
    if (!launch_local<T>(dp, y, x, st)) return false;
    if (dp.nAI < 1 || dp.nCols < 1) return true;
    T *apc = static_cast<T*>(sc.apc), *cad = static_cast<T*>(sc.cad);
    if (!project_into<T>(dp, apc, x, dptr<double>(dp.slot_H), st)) return false;
    dim3 const ga = row_grid(dp), gm = mul_grid(dp);
    if (dp.nAI > dp.nAtoms) {
        sho_collect_kernel<T><<<ga, 64, 0, st>>>(sc.aac, apc, dp.nCols,
            dptr<uint32_t>(dp.atom_starts), dptr<int8_t>(dp.atom_lmax), dptr<uint32_t>(dp.sum_start),
            dptr<uint32_t>(dp.sum_col), dptr<uint32_t>(dp.img_starts), dptr<double>(dp.img_phase), dyadic_pairs(dp));
        count_launch();
        sho_mul_kernel<double, double><<<gm, 64, 0, st>>>(sc.cadd, sc.aac, dp.nCols,
            dptr<uint32_t>(dp.atom_starts), dptr<int8_t>(dp.atom_lmax), dptr<double>(dp.atom_mat), dptr<uint32_t>(dp.atom_mat_off), dyadic_pairs(dp));
        count_launch();
        sho_broadcast_kernel<T><<<ga, 64, 0, st>>>(cad, sc.cadd, dp.nCols,
            dptr<uint32_t>(dp.atom_starts), dptr<int8_t>(dp.atom_lmax), dptr<uint32_t>(dp.sum_start),
            dptr<uint32_t>(dp.sum_col), dptr<uint32_t>(dp.img_starts), dptr<double>(dp.img_phase), dyadic_pairs(dp));
        count_launch();
    } else {
        sho_mul_kernel<T, T><<<gm, 64, 0, st>>>(cad, apc, dp.nCols,
            dptr<uint32_t>(dp.atom_starts), dptr<int8_t>(dp.atom_lmax), dptr<double>(dp.atom_mat), dptr<uint32_t>(dp.atom_mat_off), dyadic_pairs(dp));
        count_launch();
    }
    sho_add_kernel<T><<<dp.nnzb, 128, 0, st>>>(y, cad, dp.nCols, dp.nnzb, colIndex,
        dptr<uint32_t>(dp.add_start), dptr<uint32_t>(dp.add_col), dptr<uint32_t>(dp.add_slot),
        dptr<double>(dp.slot_H), dptr<uint64_t>(dp.slot_mask), dp.table_stride,
        dptr<int8_t>(dp.img_lmax), dptr<uint32_t>(dp.img_starts));
    count_launch();
    A43G_CUDA_TRY(cudaGetLastError());
    return true;
}

template bool launch_action_scratch<double>(DevicePlan &, double *, double const *, uint16_t const *, cudaStream_t, DyadicScratch const &);
template bool launch_action_scratch<float>(DevicePlan &, float *, float const *, uint16_t const *, cudaStream_t, DyadicScratch const &);

template bool launch_local<double>(DevicePlan &, double *, double const *, cudaStream_t);
template bool launch_local<float>(DevicePlan &, float *, float const *, cudaStream_t);
template bool launch_dyadic<double>(DevicePlan &, double *, double const *, uint16_t const *, cudaStream_t);
template bool launch_dyadic<float>(DevicePlan &, float *, float const *, uint16_t const *, cudaStream_t);
template bool launch_action<double>(DevicePlan &, double *, double const *, uint16_t const *, cudaStream_t);
template bool launch_action<float>(DevicePlan &, float *, float const *, uint16_t const *, cudaStream_t);

} // namespace a43g
