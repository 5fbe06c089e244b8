// Device-side plan, scratch buffers and launch interfaces shared by the CUDA sources.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>
#include <string>
#include <vector>

#include "plan.hpp"

namespace a43g {

// error state of the calling host thread (capi.cu)
void set_error(std::string const &msg);
// kernel launch counter (instrumentation, capi.cu)
void count_launch();
#define A43G_CUDA_TRY(call) do { cudaError_t e_ = (call); if (cudaSuccess != e_) { \
    ::a43g::set_error(std::string(#call) + ": " + cudaGetErrorString(e_)); return false; } } while (0)

// neighbour encoding in DevicePlan::nbr: -1 no cube (zero), >= 0 plain block index,
// <= -2 block (-e - 2) seen across a periodic boundary (multiply by the Bloch phase)
__host__ __device__ inline int32_t nbr_block(int32_t e) { return (e >= 0) ? e : (-e - 2); }

struct DeviceBuffer {
    void *ptr = nullptr;
    size_t bytes = 0;
    bool alloc(size_t n);
    void release();
    ~DeviceBuffer() { release(); }
};

template <typename T> T *dptr(DeviceBuffer const &b) { return (T*)b.ptr; }

// work item of the projection: positions [first, first + count) of the block list of one (image,
// source) pair; the items of a pair form a group (position g_pos of g_count, ticket counters
// 4 g_id ..., partial sums from row g_row on)
struct PrjItem {
    uint64_t first;
    uint32_t count, coeff, src, lmax;          // coeff: first coefficient of the image
    uint32_t g_pos, g_count, g_id, g_row;
};
constexpr uint32_t kMaxPrjItem = 40;           // positions per item at most
// slot of a list position with its flags: last cube of its x-line, last line of its z-slab
constexpr uint32_t kLineEnd = 1u << 30, kSlabEnd = 1u << 31, kSlotMask = kLineEnd - 1;

// segment of the addition: up to kSegment cubes of one x-line of a source that have atom images
// near, the points any image reaches, and the records [first, first + count) of the images
constexpr uint32_t kSegment = 4, kNoSlot = 0xffffffffu;
struct AddSegment { uint32_t blk[kSegment]; uint64_t any[kSegment]; uint32_t first, count, src, pad; };
// one image near a segment: its first coefficient and basis size, and per cube of the segment the
// slot (kNoSlot: not near) and the mask; the cubes share the y- and z-tables of yz_slot
struct AddRecord { uint32_t coeff, lmax, slot[kSegment], yz_slot, pad; uint64_t mask[kSegment]; };
static_assert(0 == sizeof(AddRecord) % 16, "the kernel copies records 16 bytes at a time");

// scratch of a projection outside the action (its own stream)
struct OwnLineScratch { DeviceBuffer part, tickets; size_t groups = 0; };

struct DevicePlan {
    bool uploaded = false;       // plan geometry on the device
    bool values_dirty = true;    // potential / matrices / phases need re-upload
    uint32_t nnzb = 0, nRows = 0, nCols = 0, nAtoms = 0, nAI = 0;
    uint32_t ncoeffI = 0, ncoeffA = 0;
    int lmax_max = -1;
    int FD_range[3] = {0, 0, 0};
    double prefactor[3] = {0, 0, 0};
    double phase[3][2][2] = {};
    double grid[4] = {0, 0, 0, 0};
    double E_re = 0, E_im = 0;
    bool fused_local = false;    // all directions use the 9-point stencil: fused kernel
    uint32_t max_zline = 0;      // cubes in the longest z-line
    // schedule parameters, set by the autotuner (autotune.cu) or left at these defaults
    uint32_t prj_chunk = 0;          // blocks per projection work item (0: by the plan's size)
    bool local_rows = false;         // the local part by the rows kernel
    bool atom_chain3 = false;        // atom matrices by the collect/multiply/broadcast kernels instead of one
    uint32_t nlists[3] = {0, 0, 0};

    DeviceBuffer veff_index;     // int32 [nnzb]
    DeviceBuffer Vcell64, Vcell32;  // [ncells][64]
    DeviceBuffer nbr;            // int32 [nnzb][6]  x-, x+, y-, y+, z-, z+
    DeviceBuffer lists_start[3], lists[3];
    DeviceBuffer zero_block;     // a block of zeros: neighbours that do not exist
    DeviceBuffer colindx;        // uint16 [nnzb]
    DeviceBuffer prj_start, prj_col;   // [nCols][nAI+1], concatenated cols
    DeviceBuffer prj_coloff;           // uint64 [nCols]
    DeviceBuffer add_start, add_col;   // [nnzb+1], [nnz]
    DeviceBuffer sum_start, sum_col;   // [nAtoms+1], [nnz]
    DeviceBuffer img_lmax, img_starts, img_phase;
    DeviceBuffer atom_starts, atom_lmax, atom_mat, atom_mat_off;
    DeviceBuffer subset_dev;     // uint32 [nCols] diagonal block of each source column
    DeviceBuffer slot_H, slot_mask, prj_slot, add_slot;   // projector tables per (image, row)
    DeviceBuffer slot_H32;       // float copy of slot_H for the tensor-core projector (ensure_tc_tables)
    int table_stride = 0;        // doubles per slot in slot_H
    DeviceBuffer dev_error;      // int: first error code recorded by a kernel (0: none)
    bool use_tc = true;          // FP32 projector on the tensor cores (else the CUDA cores)
    struct ImageGroup { uint32_t count = 0; DeviceBuffer images; } img_group[8];  // images by basis size
    // work items of the generic projection kernel by basis size: (image, source, first, last) list
    // positions, each at most 16 blocks
    struct PrjItems { uint32_t count = 0; DeviceBuffer items; } prj_items[8];
    // the projection along lines (projector_line.cuh): items of every (image, source) pair, one
    // record {block, slot and flags, mask} per list position, and the slots' tables as
    // [dir][point][order] with 8 bytes per value (FP32: the value twice), the orders padded to even
    struct PrjLine { uint32_t count = 0; size_t part_rows = 0, groups = 0; DeviceBuffer items, tickets; } prj_line;
    DeviceBuffer prj_rec, line_tab64, line_tab32;
    uint32_t nslots = 0;
    uint32_t add_segments = 0;   // the addition along lines: AddSegment, AddRecord
    DeviceBuffer add_seg, add_rec;
    DeviceBuffer prj_part;       // partial projection sums of multi-item groups
    // batch plans (GreenPlan::replicate): npairs (energy, k-point) pairs of nsrc_pair sources each
    uint32_t npairs = 1, nsrc_pair = 0;
    size_t mat_stride = 0;       // doubles of atom matrices per pair
    DeviceBuffer pair_args32, pair_args64;   // per pair: E_re, E_im, phases [3][2][2] (float, double)
    // retirement: sources whose columns have all finished are skipped by every kernel of the
    // action and of the solver while retire is set (uint8 per source, 1 = active)
    bool retire = false;
    DeviceBuffer src_active;
    // the blocks of every source in order (the solver's fixed-order column reductions)
    DeviceBuffer src_start, src_blocks;      // uint32 [nCols + 1], uint32 [nnzb]
    uint32_t max_src_blocks = 0;
    // scratch of the dyadic part (allocated once per plan, never per call)
    DeviceBuffer apc;            // real_t [ncoeffI*nCols][2][64] image projection coefficients
    DeviceBuffer aac, cadd;      // double [ncoeffA*nCols][2][64] of the three-kernel atom chain
    DeviceBuffer cad;            // real_t [ncoeffI*nCols][2][64] image addition coefficients
};

bool upload_plan(GreenPlan const &hp, DevicePlan &dp);
// kernel attributes (dynamic shared memory above 48 KB) of the current device
bool prepare_local_kernels();
bool prepare_tc_kernels();
// kernel launch counter: n launches at once (replays of a captured graph)
void count_launches(uint64_t n);
uint64_t launches_so_far();
// potential, matrices, phases and energies; earlier calls on st are waited for before they are replaced
bool upload_values(GreenPlan const &hp, DevicePlan &dp, cudaStream_t st);
// copies of host arrays made on the legacy stream have reached the device: kernels of any stream may
// read them.  Kernels launched on st have finished: arrays that they read may be replaced.
bool uploads_landed();
bool readers_done(cudaStream_t st);
// projection work items (image, source, up to dp.prj_chunk consecutive blocks of its list); no kernel
// that reads the present ones may be running (readers_done)
bool build_prj_items(GreenPlan const &hp, DevicePlan &dp);
uint32_t prj_chunk_by_size(GreenPlan const &hp);
// a table [slot][order][dir][point] of the plan's slots in the layout of the line kernels
bool make_line_table(DevicePlan const &dp, double const *slot_H, DeviceBuffer &t64, DeviceBuffer *t32, cudaStream_t st);
// chooses the schedule parameters of the action for this plan by timing them (autotune.cu)
template <typename T>
bool autotune(GreenPlan const &hp, DevicePlan &dp, cudaStream_t st, std::string &report);
bool ensure_dyadic_scratch(DevicePlan &dp, size_t elem_bytes);
// tables of the tensor-core projector: made before use_tc is set, since most plans never use them
bool ensure_tc_tables(GreenPlan const &hp, DevicePlan &dp);
// the atom matrices by one kernel (its shared memory holds basis sizes up to 5)
inline bool one_atom_kernel(DevicePlan const &dp) { return dp.lmax_max <= 5 && !dp.atom_chain3; }
// partial-sum buffer of the deterministic projection for reals of elem_bytes
bool ensure_prj_part(DevicePlan &dp, size_t elem_bytes);

// the action y = (H - E S) x on real_t = double or float
template <typename T>
bool launch_action(DevicePlan &dp, T *y, T const *x, uint16_t const *colIndex, cudaStream_t s);

// parts of the action (tests, VJP and benchmarks use them separately)
template <typename T>
bool launch_local(DevicePlan &dp, T *y, T const *x, cudaStream_t s);          // potential + kinetic
template <typename T>
bool launch_dyadic(DevicePlan &dp, T *y, T const *x, uint16_t const *colIndex, cudaStream_t s);

double action_flops(GreenPlan const &hp, int real_bytes);

// the action with the dyadic coefficients in caller-given scratch instead of the plan's
// buffers: apc, cad hold ncoeffI*nCols*128 reals of the action's precision, aac, cadd
// ncoeffA*nCols*128 doubles (apc is zeroed by the call; the others are overwritten)
struct DyadicScratch { void *apc, *cad; double *aac, *cadd; };
template <typename T>
bool launch_action_scratch(DevicePlan &dp, T *y, T const *x, uint16_t const *colIndex, cudaStream_t st,
                           DyadicScratch const &sc);

// FP64 pieces of the dyadic part on caller-given buffers (vector-Jacobian products):
// aac = sum over images of img_phase * apc; out = M in (atom matrices of the plan)
bool launch_collect_with(DevicePlan &dp, double *aac, double const *apc, double const *img_phase, cudaStream_t st);
bool launch_mul_with(DevicePlan &dp, double *out, double const *in, cudaStream_t st);

// tensor-core (tcgen05, 3xTF32) projection and addition of the FP32 action (projector_tc.cu)
bool tc_projector_supported(DevicePlan const &dp);
bool launch_project_tc(DevicePlan &dp, float const *x, cudaStream_t st);
bool launch_add_tc(DevicePlan &dp, float *y, uint16_t const *colIndex, cudaStream_t st);

// both vectors lie on a boundary of `bytes` (a power of two)
inline bool vectors_aligned(void const *x, void const *y, unsigned bytes) {
    return 0 == ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & uintptr_t(bytes - 1));
}
// the projection along lines with the given tables (every coefficient of an active source is written);
// the scratch of callers that may run on different streams must not be shared: partial sums
// (prj_part_bytes), and tickets that are zero before the first call and after every call
struct LineScratch { void *part; uint32_t *tickets; };
bool launch_project_line(DevicePlan &dp, float *apc, float const *x, void const *tab, LineScratch const &sc, cudaStream_t st);
bool launch_project_line(DevicePlan &dp, double *apc, double const *x, void const *tab, LineScratch const &sc, cudaStream_t st);
bool ensure_line_scratch(DevicePlan const &dp, OwnLineScratch &own, size_t elem_bytes, cudaStream_t st, LineScratch &sc);
inline size_t prj_part_bytes(DevicePlan const &dp, size_t elem_bytes) {
    size_t const n = dp.prj_line.part_rows*128*elem_bytes;
    return n < 16 ? 16 : n;
}
bool launch_add_line(DevicePlan &dp, float *y, float const *cad, uint16_t const *colIndex, cudaStream_t st);
bool launch_add_line(DevicePlan &dp, double *y, double const *cad, uint16_t const *colIndex, cudaStream_t st);
bool prepare_line_kernels32();
bool prepare_line_kernels64();

} // namespace a43g
