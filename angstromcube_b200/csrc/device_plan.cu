// Upload of a host plan to the device and the derived neighbour table.
#include "device.cuh"

#include <algorithm>
#include <cstdlib>
#include <cstring>

namespace a43g {

bool DeviceBuffer::alloc(size_t n) {
    if (n <= bytes && ptr) return true;
    release();
    if (0 == n) return true;
    cudaError_t const e = cudaMalloc(&ptr, n);
    if (cudaSuccess != e) {
        ptr = nullptr; bytes = 0;
        set_error(std::string("cudaMalloc of ") + std::to_string(n) + " bytes: " + cudaGetErrorString(e));
        return false;
    }
    bytes = n;
    return true;
}

void DeviceBuffer::release() {
    if (ptr) cudaFree(ptr);
    ptr = nullptr; bytes = 0;
}

namespace {

template <typename T>
bool put(DeviceBuffer &b, std::vector<T> const &v) {
    size_t const n = v.size()*sizeof(T);
    if (!b.alloc(std::max<size_t>(n, 16))) return false;
    if (n) A43G_CUDA_TRY(cudaMemcpy(b.ptr, v.data(), n, cudaMemcpyHostToDevice));
    return true;
}

// Neighbour of every block along each direction, read off the finite-difference lists:
// consecutive list entries are neighbours; the entries before the first and after the last
// cube are the halo (0: zero cube, negative: periodic image, src/kinetic_plan.cxx:153-179).
std::vector<int32_t> neighbour_table(GreenPlan const &hp) {
    size_t const nnzb = hp.nnzb();
    std::vector<int32_t> nbr(6*nnzb, -1);
    for (int dd = 0; dd < 3; ++dd) {
        auto const &K = hp.kinetic[dd];
        for (uint32_t il = 0; il < K.nlists(); ++il) {
            int32_t const *L = &K.entry[K.start[il]];
            int const len = int(K.start[il + 1] - K.start[il]);
            int n = 0;
            while (kNhalo + n < len && L[kNhalo + n] > 0) ++n;
            for (int i = 0; i < n; ++i) {
                int32_t const b = L[kNhalo + i] - 1;
                auto code = [](int32_t entry) -> int32_t {
                    if (entry > 0) return entry - 1;          // plain neighbour
                    if (entry < 0) return -(-entry - 1) - 2;  // periodic image
                    return -1;                                 // zero cube
                };
                nbr[6*size_t(b) + 2*dd + 0] = code(L[kNhalo + i - 1]);
                nbr[6*size_t(b) + 2*dd + 1] = code(L[kNhalo + i + 1]);
            }
        }
    }
    return nbr;
}

// slot_H [slot][order][dir][point] as [slot][dir][point][order], the orders padded to lp; the FP32
// table holds every value twice (a pair of columns)
__global__ void k_line_table(double *t64, float2 *t32, double const *slot_H, size_t n, int nu, int lp) {
    size_t const k = size_t(blockIdx.x)*blockDim.x + threadIdx.x;
    if (k >= n) return;
    int const m = int(k % lp), di = int(k/lp % 12);
    double const h = (m < nu) ? slot_H[(k/lp/12*nu + m)*12 + di] : 0.0;
    t64[k] = h;
    if (t32) t32[k] = make_float2(float(h), float(h));
}

bool build_add_segments(GreenPlan const &hp, DevicePlan &dp);

} // namespace

// A copy from pageable memory may return while its last piece is still on the way, and the kernels of
// a non-blocking stream are not ordered behind the legacy stream that it runs on.
bool uploads_landed() {
    A43G_CUDA_TRY(cudaStreamSynchronize(nullptr));
    return true;
}

// The legacy stream does not wait for a non-blocking stream either: arrays that kernels launched on st
// may still read are replaced only when they are done.  A stream under capture has nothing running.
bool readers_done(cudaStream_t st) {
    if (!st) return true;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    A43G_CUDA_TRY(cudaStreamIsCapturing(st, &cs));
    if (cudaStreamCaptureStatusNone == cs) A43G_CUDA_TRY(cudaStreamSynchronize(st));
    return true;
}

bool upload_plan(GreenPlan const &hp, DevicePlan &dp) {
    if (!prepare_line_kernels32() || !prepare_line_kernels64() || !prepare_tc_kernels() || !prepare_local_kernels()) return false;
    dp.nnzb = uint32_t(hp.nnzb()); dp.nRows = hp.nRows; dp.nCols = hp.nCols;
    dp.nAtoms = hp.nAtoms; dp.nAI = hp.nAtomImages;
    dp.ncoeffI = uint32_t(hp.ncoeff_images()); dp.ncoeffA = uint32_t(hp.ncoeff_atoms());
    dp.lmax_max = -1;
    for (auto l : hp.AtomImageLmax) dp.lmax_max = std::max(dp.lmax_max, int(l));
    bool all4 = true;
    for (int d = 0; d < 3; ++d) {
        dp.FD_range[d] = hp.kinetic[d].FD_range;
        dp.prefactor[d] = hp.kinetic[d].prefactor;
        dp.nlists[d] = hp.kinetic[d].nlists();
        all4 = all4 && (dp.FD_range[d] >= 1 && dp.FD_range[d] != 8);
        dp.grid[d] = hp.grid_spacing_dyadic[d];
    }
    dp.grid[3] = hp.grid_spacing_dyadic[3];
    dp.fused_local = all4;
    dp.max_zline = 0;
    {
        auto const &K = hp.kinetic[2];
        for (uint32_t il = 0; il < K.nlists(); ++il) {
            uint32_t const len = K.start[il + 1] - K.start[il];
            dp.max_zline = std::max(dp.max_zline, len > 2*kNhalo ? len - 2*kNhalo : 0u);
        }
    }

    if (!put(dp.veff_index, hp.veff_index)) return false;
    if (!put(dp.nbr, neighbour_table(hp))) return false;
    if (!dp.zero_block.alloc(8192*sizeof(double))) return false;
    A43G_CUDA_TRY(cudaMemset(dp.zero_block.ptr, 0, 8192*sizeof(double)));
    for (int d = 0; d < 3; ++d) {
        if (!put(dp.lists_start[d], hp.kinetic[d].start)) return false;
        if (!put(dp.lists[d], hp.kinetic[d].entry)) return false;
    }
    if (!put(dp.colindx, hp.colindx)) return false;
    // dyadic sparsity
    std::vector<uint32_t> ps, pc; std::vector<uint64_t> po;
    for (uint32_t s = 0; s < hp.nCols; ++s) {
        po.push_back(pc.size());
        auto const &c = hp.SHOprj[s];
        if (c.start.empty()) ps.insert(ps.end(), hp.nAtomImages + 1, 0u);
        else ps.insert(ps.end(), c.start.begin(), c.start.end());
        pc.insert(pc.end(), c.col.begin(), c.col.end());
    }
    if (!put(dp.prj_start, ps) || !put(dp.prj_col, pc) || !put(dp.prj_coloff, po)) return false;
    if (!put(dp.add_start, hp.SHOadd.start) || !put(dp.add_col, hp.SHOadd.col)) return false;
    if (!put(dp.sum_start, hp.SHOsum.start) || !put(dp.sum_col, hp.SHOsum.col)) return false;
    if (!put(dp.img_lmax, hp.AtomImageLmax)) return false;
    if (!put(dp.img_starts, hp.AtomImageStarts)) return false;
    if (!put(dp.atom_starts, hp.AtomStarts) || !put(dp.atom_lmax, hp.AtomLmax)) return false;
    if (!put(dp.atom_mat_off, hp.AtomMatOffset)) return false;
    for (int L = 0; L < 8; ++L) {
        std::vector<uint32_t> imgs;
        for (uint32_t a = 0; a < hp.nAtomImages; ++a) if (hp.AtomImageLmax[a] == L) imgs.push_back(a);
        dp.img_group[L].count = uint32_t(imgs.size());
        if (!put(dp.img_group[L].images, imgs)) return false;
    }
    // positions per projection work item: by the plan's size (default) or a given number
    if (char const *c = std::getenv("A43G_PRJ_CHUNK")) dp.prj_chunk = uint32_t(std::max(0, std::atoi(c)));
    if (dp.lmax_max > 7) { set_error("projector basis sizes above numax 7 are not supported"); return false; }
    if (!build_prj_items(hp, dp)) return false;
    dp.table_stride = (hp.table_lmax + 1)*12;
    if (!put(dp.slot_H, hp.slot_H) || !put(dp.slot_mask, hp.slot_mask)) return false;
    if (!put(dp.prj_slot, hp.prj_slot) || !put(dp.add_slot, hp.add_slot)) return false;
    {   // tables of the line kernels (FP32: every value twice, a pair of columns) and their records
        dp.nslots = uint32_t(hp.slot_mask.size());
        if (!make_line_table(dp, dptr<double>(dp.slot_H), dp.line_tab64, &dp.line_tab32, nullptr)) return false;
        if (hp.slot_mask.size() > kSlotMask) { set_error("too many projector slots"); return false; }
        std::vector<uint32_t> rec(4*pc.size());
        size_t k = 0;
        for (auto const &c : hp.SHOprj)
            for (uint32_t a = 0; a + 1 < c.start.size(); ++a)
                for (uint32_t p = c.start[a]; p < c.start[a + 1]; ++p, ++k) {
                    float const *here = &hp.rowCubePos[4*size_t(hp.rowindx[c.col[p]])];
                    float const *next = (p + 1 < c.start[a + 1]) ? &hp.rowCubePos[4*size_t(hp.rowindx[c.col[p + 1]])] : nullptr;
                    bool const slab = !next || next[2] != here[2], line = slab || next[1] != here[1];
                    uint64_t const m = hp.slot_mask[hp.prj_slot[k]];
                    rec[4*k + 0] = c.col[p];
                    rec[4*k + 1] = hp.prj_slot[k] | (line ? kLineEnd : 0u) | (slab ? kSlabEnd : 0u);
                    rec[4*k + 2] = uint32_t(m); rec[4*k + 3] = uint32_t(m >> 32);
                }
        if (!put(dp.prj_rec, rec)) return false;
    }
    if (!build_add_segments(hp, dp)) return false;
    if (!put(dp.subset_dev, hp.subset)) return false;
    {   // blocks of every source, in block order
        std::vector<uint32_t> start(hp.nCols + 1, 0), blocks(hp.nnzb());
        for (size_t b = 0; b < hp.nnzb(); ++b) ++start[hp.colindx[b] + 1];
        for (uint32_t c = 0; c < hp.nCols; ++c) start[c + 1] += start[c];
        std::vector<uint32_t> fill(start.begin(), start.end() - 1);
        for (size_t b = 0; b < hp.nnzb(); ++b) blocks[fill[hp.colindx[b]]++] = uint32_t(b);
        dp.max_src_blocks = 0;
        for (uint32_t c = 0; c < hp.nCols; ++c) dp.max_src_blocks = std::max(dp.max_src_blocks, start[c + 1] - start[c]);
        if (!put(dp.src_start, start) || !put(dp.src_blocks, blocks)) return false;
        if (!put(dp.src_active, std::vector<uint8_t>(std::max<size_t>(hp.nCols, 1), uint8_t(1)))) return false;
        dp.retire = false;
    }
    dp.npairs = hp.npairs;
    dp.nsrc_pair = (hp.npairs > 1) ? hp.nsrc_pair : hp.nCols;
    dp.mat_stride = hp.AtomMatrices.size();
    if (!put(dp.dev_error, std::vector<int32_t>(4, 0))) return false;
    {
        // FP32 projector: CUDA cores (default) or the tensor cores ("tc"); FP64 always on the CUDA cores
        char const *e = std::getenv("A43G_PROJECTOR");
        dp.use_tc = (e && 0 == std::strcmp(e, "tc"));
        // local kernel: pencils (default) or "rows" (also "plain"), the kernel of lines beyond the pencils' limit
        char const *l = std::getenv("A43G_LOCAL"), *l64 = std::getenv("A43G_LOCAL64");
        dp.local_rows = (l && (0 == std::strcmp(l, "rows") || 0 == std::strcmp(l, "plain"))) ||
                        (l64 && 0 == std::strcmp(l64, "rows"));
        // atom-matrix chain: one kernel (default) or "three" (collect, multiply, broadcast)
        char const *ac = std::getenv("A43G_ATOM_CHAIN");
        dp.atom_chain3 = (ac && 0 == std::strcmp(ac, "three"));
    }
    if (dp.use_tc && !ensure_tc_tables(hp, dp)) return false;
    if (!one_atom_kernel(dp) &&
        (!dp.aac.alloc(std::max<size_t>(16, size_t(dp.ncoeffA)*dp.nCols*128*sizeof(double))) ||
         !dp.cadd.alloc(std::max<size_t>(16, size_t(dp.ncoeffA)*dp.nCols*128*sizeof(double))))) return false;
    // A cudaMalloc that the driver's pool cannot serve takes 0.35 ms whatever its size, several times an
    // application of the small plans whose coefficient scratch is 4 MB or less (64 blocks: 0.06 ms), so
    // they get theirs here, for FP64.  Larger ones get it in their first application, where its precision
    // is known: half of it for FP32.
    if (dp.nAI > 0 && 2*size_t(dp.ncoeffI)*dp.nCols*1024 + prj_part_bytes(dp, 8) <= (size_t(4) << 20) &&
        (!ensure_dyadic_scratch(dp, 8) || !ensure_prj_part(dp, 8))) return false;
    dp.uploaded = true;
    dp.values_dirty = true;
    return upload_values(hp, dp, nullptr);          // waits for the legacy stream: the tables above too
}

// positions per item: enough items for about 12 CTAs per SM (two CTAs per item at least), since small
// plans would leave SMs idle, and as many as an item's tables in shared memory allow
uint32_t prj_chunk_by_size(GreenPlan const &hp) {
    size_t npos = 0;
    for (auto const &c : hp.SHOprj) npos += c.nnz();
    return uint32_t(std::min<size_t>(kMaxPrjItem, std::max<size_t>(8, 2*npos/(148*12))));
}

bool build_prj_items(GreenPlan const &hp, DevicePlan &dp) {
    constexpr uint32_t kGenericChunk = 16;
    uint32_t const chunk = std::min(dp.prj_chunk ? dp.prj_chunk : prj_chunk_by_size(hp), kMaxPrjItem);
    std::vector<uint32_t> items[8];
    std::vector<PrjItem> line;
    uint32_t groups = 0;
    size_t rows = 0;
    uint64_t off = 0;
    for (uint32_t s = 0; s < hp.nCols; ++s) {
        auto const &c = hp.SHOprj[s];
        for (uint32_t a = 0; a < hp.nAtomImages; ++a) {
            int const L = hp.AtomImageLmax[a];
            uint32_t const k0 = c.start.empty() ? 0 : c.start[a], k1 = c.start.empty() ? 0 : c.start[a + 1];
            for (uint32_t k = k0; k < k1; k += kGenericChunk) {
                uint32_t const it[4] = {a, s, k, std::min(k + kGenericChunk, k1)};
                items[L].insert(items[L].end(), it, it + 4);
            }
            // a pair without blocks has one empty item, which writes its zero coefficients
            uint32_t const len = k1 - k0, n = std::max(1u, (len + chunk - 1)/chunk);
            for (uint32_t i = 0; i < n; ++i) {
                uint64_t const b = k0 + uint64_t(len)*i/n, e = k0 + uint64_t(len)*(i + 1)/n;
                line.push_back(PrjItem{off + b, uint32_t(e - b), hp.AtomImageStarts[a], s, uint32_t(L), i, n,
                                       groups, uint32_t(rows)});
            }
            ++groups;
            if (n > 1) rows += size_t(n)*nsho(L);
        }
        off += c.col.size();
    }
    for (int L = 0; L < 8; ++L) {
        dp.prj_items[L].count = uint32_t(items[L].size()/4);
        if (!put(dp.prj_items[L].items, items[L])) return false;
    }
    dp.prj_line.count = uint32_t(line.size());
    dp.prj_line.part_rows = rows;
    dp.prj_line.groups = groups;
    return put(dp.prj_line.items, line) && put(dp.prj_line.tickets, std::vector<uint32_t>(4*size_t(groups), 0u)) &&
           uploads_landed();
}

namespace {
bool build_add_segments(GreenPlan const &hp, DevicePlan &dp) {
    // numax 6 and 7 take segments of half the length (registers)
    uint32_t const len = (dp.lmax_max <= 5) ? kSegment : kSegment/2;
    std::vector<AddSegment> segs;
    std::vector<AddRecord> recs;
    recs.reserve(hp.SHOadd.nnz()/2 + 16);
    auto close = [&](uint32_t const *blk, uint32_t n) {
        AddSegment sg{};
        sg.first = uint32_t(recs.size()); sg.src = hp.colindx[blk[0]];
        uint32_t at[kSegment], end[kSegment];
        for (uint32_t i = 0; i < n; ++i) { sg.blk[i] = blk[i]; at[i] = hp.SHOadd.start[blk[i]]; end[i] = hp.SHOadd.start[blk[i] + 1]; }
        while (true) {                               // the images of the cubes, merged in ascending order
            uint32_t a = kNoSlot;
            for (uint32_t i = 0; i < n; ++i) if (at[i] < end[i]) a = std::min(a, hp.SHOadd.col[at[i]]);
            if (kNoSlot == a) break;
            AddRecord r{};
            r.coeff = hp.AtomImageStarts[a]; r.lmax = uint32_t(hp.AtomImageLmax[a]);
            for (uint32_t i = 0; i < kSegment; ++i) r.slot[i] = kNoSlot;
            for (uint32_t i = 0; i < n; ++i) {
                if (at[i] >= end[i] || hp.SHOadd.col[at[i]] != a) continue;
                r.slot[i] = r.yz_slot = hp.add_slot[at[i]++];
                r.mask[i] = hp.slot_mask[r.slot[i]];
                sg.any[i] |= r.mask[i];
            }
            recs.push_back(r);
        }
        sg.count = uint32_t(recs.size()) - sg.first;
        segs.push_back(sg);
    };
    auto const &K = hp.kinetic[0];
    for (uint32_t il = 0; il < K.nlists(); ++il) {
        uint32_t blk[kSegment], n = 0;
        for (uint32_t k = K.start[il] + kNhalo; k < K.start[il + 1] && K.entry[k] > 0; ++k) {
            uint32_t const b = uint32_t(K.entry[k] - 1);
            if (hp.SHOadd.start[b] == hp.SHOadd.start[b + 1]) continue;
            blk[n++] = b;
            if (n == len) { close(blk, n); n = 0; }
        }
        if (n) close(blk, n);
    }
    dp.add_segments = uint32_t(segs.size());
    return put(dp.add_seg, segs) && put(dp.add_rec, recs);
}
} // namespace

bool make_line_table(DevicePlan const &dp, double const *slot_H, DeviceBuffer &t64, DeviceBuffer *t32, cudaStream_t st) {
    int const nu = dp.table_stride/12, lp = (dp.lmax_max | 1) + 1;
    size_t const n = size_t(dp.nslots)*12*std::max(lp, 0);
    if (nu < 1 || 0 == n) return true;
    if (!t64.alloc(n*8) || (t32 && !t32->alloc(n*8))) return false;
    k_line_table<<<unsigned((n + 255)/256), 256, 0, st>>>(dptr<double>(t64), t32 ? dptr<float2>(*t32) : nullptr, slot_H, n, nu, lp);
    count_launch();
    A43G_CUDA_TRY(cudaGetLastError());
    return true;
}

bool ensure_tc_tables(GreenPlan const &hp, DevicePlan &dp) {
    return dp.slot_H32.ptr || (put(dp.slot_H32, std::vector<float>(hp.slot_H.begin(), hp.slot_H.end())) && uploads_landed());
}

bool ensure_prj_part(DevicePlan &dp, size_t elem_bytes) {
    return dp.prj_part.alloc(prj_part_bytes(dp, elem_bytes));
}

bool ensure_line_scratch(DevicePlan const &dp, OwnLineScratch &own, size_t elem_bytes, cudaStream_t st, LineScratch &sc) {
    if (!own.part.alloc(prj_part_bytes(dp, elem_bytes))) return false;
    if (own.groups < dp.prj_line.groups || !own.tickets.ptr) {
        size_t const n = std::max<size_t>(16, 4*dp.prj_line.groups*sizeof(uint32_t));
        if (!own.tickets.alloc(n)) return false;
        A43G_CUDA_TRY(cudaMemsetAsync(own.tickets.ptr, 0, n, st));
        own.groups = dp.prj_line.groups;
    }
    sc = LineScratch{own.part.ptr, dptr<uint32_t>(own.tickets)};
    return true;
}

bool upload_values(GreenPlan const &hp, DevicePlan &dp, cudaStream_t st) {
    if (!readers_done(st)) return false;
    if (!put(dp.Vcell64, hp.Vcell)) return false;
    std::vector<float> v32(hp.Vcell.begin(), hp.Vcell.end());
    if (!put(dp.Vcell32, v32)) return false;
    if (hp.npairs > 1) {
        // batch plan: image phases and atom matrices [pair][...], energies and phases per pair
        if (!put(dp.atom_mat, hp.pair_mats)) return false;
        if (!put(dp.img_phase, hp.pair_img_phase)) return false;
        std::vector<double> a64(14*size_t(hp.npairs));
        std::vector<float> a32(14*size_t(hp.npairs));
        for (uint32_t p = 0; p < hp.npairs; ++p) {
            a64[14*p] = hp.pair_E[2*p]; a64[14*p + 1] = hp.pair_E[2*p + 1];
            for (int k = 0; k < 12; ++k) a64[14*p + 2 + k] = hp.pair_phase[12*size_t(p) + k];
        }
        for (size_t k = 0; k < a64.size(); ++k) a32[k] = float(a64[k]);
        if (!put(dp.pair_args64, a64) || !put(dp.pair_args32, a32)) return false;
    } else {
        if (!put(dp.atom_mat, hp.AtomMatrices)) return false;
        if (!put(dp.img_phase, hp.AtomImagePhase)) return false;
    }
    std::memcpy(dp.phase, hp.phase, sizeof(dp.phase));
    dp.E_re = hp.E_re; dp.E_im = hp.E_im;
    if (!uploads_landed()) return false;            // the values may be used on any stream from here on
    dp.values_dirty = false;
    return true;
}

bool ensure_dyadic_scratch(DevicePlan &dp, size_t elem_bytes) {
    size_t const n = std::max<size_t>(16, size_t(dp.ncoeffI)*dp.nCols*128*elem_bytes);
    if (dp.apc.bytes >= n && dp.cad.bytes >= n) return true;
    return dp.apc.alloc(n) && dp.cad.alloc(n);
}

// flop count of one application as the reference counts it (include/green_potential.hxx:171-177,
// include/green_kinetic.hxx:381, include/dyadic_plan.hxx:93-103), R1C2 = 2, Noco = 1
double action_flops(GreenPlan const &hp, int /*real_bytes*/) {
    double const nnzb = double(hp.nnzb());
    double f = (1 + 2*(0 != hp.E_im))*nnzb*4096*2;
    for (int d = 0; d < 3; ++d) {
        int const nFD = (hp.kinetic[d].FD_range >= 1 && hp.kinetic[d].nlists() > 0) ? hp.kinetic[d].FD_range : 0;
        f += nnzb*(2*nFD + 1)*2*4096*2;
    }
    if (hp.nAtomImages > 0 && hp.nCols > 0) {
        auto flop_prj_add = [](int L) {
            return 2*(64*(L + 1) + 16*(((L + 1)*(L + 2))/2) + 4*(((L + 1)*(L + 2)*(L + 3))/6));
        };
        double gen = 0, addc = 0, mul = 0, sum = 0;
        for (uint32_t k = 0; k < hp.SHOadd.nnz(); ++k) {
            int const L = hp.AtomImageLmax[hp.SHOadd.col[k]];
            addc += 64.0*flop_prj_add(L);
            gen += 12.0*(7 + 4*L);
        }
        for (uint32_t ia = 0; ia < hp.nAtoms; ++ia) { double const n = nsho(hp.AtomImageLmax[ia]); mul += n*n; }
        mul *= 2.0*hp.nCols*64;
        if (hp.nAtomImages > hp.nAtoms) {
            for (uint32_t a = 0; a < hp.nAtomImages; ++a) sum += nsho(hp.AtomImageLmax[a]);
            sum *= 2.0*hp.nCols*64;
        }
        f += mul*4 + 2*sum*4 + 2*gen + 2*addc*2;
    }
    return f;
}

} // namespace a43g
