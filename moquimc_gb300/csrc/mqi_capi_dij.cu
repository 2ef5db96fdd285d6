// C ABI of the Dij scorer: the (voxel, spot) table, its CSR build, and the two sparse products.
#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "mqi_ctx.h"

using namespace mqi_gpu;

namespace
{

int
bit_length(uint64_t v) {
    int b = 0;
    while (v) {
        ++b;
        v >>= 1;
    }
    return b;
}

void
free_csr(DijCsr& m) {
    cudaFree(m.slab);
    m = DijCsr{};
}

/// Arrays cut from one allocation, each on a 256-byte boundary.  Laid out first with no memory, for
/// its size.
struct Carve {
    char*  base = nullptr;
    size_t used = 0;
    template<typename T>
    void
    take(T*& p, uint64_t n) {
        p = base ? reinterpret_cast<T*>(base + used) : nullptr;
        used += (std::max<uint64_t>(n, 1) * sizeof(T) + 255) & ~(size_t) 255;
    }
};

/// At least `bytes` in p, whose contents are not kept: what is there when that is enough and not far
/// more, else an allocation of its own.  (A build's two dozen allocations took 1.5 ms of a 4 ms build.)
cudaError_t
ensure_bytes(void*& p, size_t& have, size_t bytes) {
    if (p && have >= bytes && have / 4 <= bytes) return cudaSuccess;
    cudaFree(p);
    p             = nullptr;
    have          = 0;
    cudaError_t e = cudaMalloc(&p, bytes);
    if (e == cudaSuccess) have = bytes;
    else p = nullptr;
    return e;
}

/// Device buffers freed on scope exit.
struct Scratch {
    std::vector<void*> ptrs;
    template<typename T>
    cudaError_t
    alloc(mqi_ctx* c, T*& p, uint64_t n) {
        cudaError_t e = device_alloc(c, p, std::max<uint64_t>(n, 1) * sizeof(T));
        if (e == cudaSuccess) ptrs.push_back(p);
        return e;
    }
    ~Scratch() {
        for (void* p : ptrs) cudaFree(p);
    }
};

ScorerHost*
dij_scorer(mqi_ctx* c, int id, const char* who) {
    if (!valid_ctx(c)) {
        fail(c, MQI_ERR_INVALID, std::string(who) + ": ctx is NULL");
        return nullptr;
    }
    if (id < 0 || id >= (int) c->scorers.size() || c->scorers[id].type != MQI_SCORER_DIJ) {
        fail(c, MQI_ERR_INVALID, std::string(who) + ": not a Dij scorer");
        return nullptr;
    }
    return &c->scorers[id];
}

}   // namespace

namespace mqi_gpu
{

void
dij_drop_matrix(ScorerHost& s) {
    free_csr(s.csr);
}

/// Called by mqi_destroy / mqi_reset_tallies.
void
dij_release(ScorerHost& s) {
    cudaFree(s.hit_log);
    cudaFree(s.hit_count);
    s.hit_log   = nullptr;
    s.hit_count = nullptr;
    s.hit_cap   = 0;
    free_csr(s.csr);
    cudaFree(s.dij);
    cudaFree(s.dij_count);
    s.dij = nullptr;
    s.dij_count = nullptr;
}

cudaError_t
dij_reset(ScorerHost& s, int sms, cudaStream_t st) {
    s.csr.built = false;
    if (s.csr.slab_bytes > kKeepScratch) free_csr(s.csr);   // a smaller one is kept for the next build
    cudaError_t e = dij_clear(s.dij, s.dij_cap, sms, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(s.dij_count, 0, sizeof(unsigned long long), st);
    return e;
}

}   // namespace mqi_gpu

extern "C" {

int
mqi_add_dij_scorer(mqi_ctx* c, int child_id, int roi_method, uint32_t roi_length, const uint32_t* roi_start,
                   const uint32_t* roi_stride, const uint32_t* roi_acc, uint64_t capacity, int* scorer_id) {
    if (!valid_ctx(c)) return fail(c, MQI_ERR_INVALID, "mqi_add_dij_scorer: ctx is NULL");
    if (c->n_scen > 1) return fail(c, MQI_ERR_UNSUPPORTED, "mqi_add_dij_scorer: not with robust scenarios");
    if (capacity == 0) capacity = 1ull << 26;
    if (capacity > (1ull << 32)) return fail(c, MQI_ERR_INVALID, "mqi_add_dij_scorer: at most 2^32 slots");
    uint64_t cap = 1;
    while (cap < capacity) cap <<= 1;
    // the dense-scorer path validates the child and the ROI and allocates the ROI arrays
    int id = -1;
    int rc = mqi_add_scorer(c, child_id, MQI_SCORER_EDEP, roi_method, roi_length, roi_start, roi_stride, roi_acc, &id);
    if (rc != MQI_OK) return rc;
    ScorerHost& s = c->scorers[id];
    DeviceGuard g(c->device);
    cudaFree(s.tally);   // a Dij scorer has no dense tally
    s.tally     = nullptr;
    s.tally_len = 0;
    s.type      = MQI_SCORER_DIJ;
    s.dij_cap   = cap;
    cudaError_t e = device_alloc(c, s.dij, cap * sizeof(DijSlot));
    if (e == cudaSuccess) e = device_alloc(c, s.dij_count, sizeof(unsigned long long));
    if (e == cudaSuccess) e = dij_reset(s, c->num_sms, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) {
        dij_release(s);
        cudaFree(s.start); cudaFree(s.stride); cudaFree(s.acc); cudaFree(s.roi_words);
        c->scorers.pop_back();
        return cuda_fail(c, e, "mqi_add_dij_scorer");
    }
    if (scorer_id) *scorer_id = id;
    return MQI_OK;
}

int
mqi_dij_record_hits(mqi_ctx* c, int id, uint64_t capacity) {
    ScorerHost* sp = dij_scorer(c, id, "mqi_dij_record_hits");
    if (!sp) return MQI_ERR_INVALID;
    ScorerHost& s = *sp;
    DeviceGuard g(c->device);
    MQI_CUDA(c, cudaStreamSynchronize(c->stream), "mqi_dij_record_hits");
    cudaFree(s.hit_log);
    cudaFree(s.hit_count);
    s.hit_log   = nullptr;
    s.hit_count = nullptr;
    s.hit_cap   = 0;
    if (capacity == 0) return MQI_OK;
    cudaError_t e = device_alloc(c, s.hit_log, capacity * sizeof(DijHit));
    if (e == cudaSuccess) e = device_alloc(c, s.hit_count, sizeof(unsigned long long));
    if (e == cudaSuccess) e = cudaMemsetAsync(s.hit_count, 0, sizeof(unsigned long long), c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) {
        cudaFree(s.hit_log);
        cudaFree(s.hit_count);
        s.hit_log   = nullptr;
        s.hit_count = nullptr;
        return cuda_fail(c, e, "mqi_dij_record_hits");
    }
    s.hit_cap = capacity;
    return MQI_OK;
}

int
mqi_dij_get_hits(mqi_ctx* c, int id, uint32_t* voxel, uint32_t* spot, double* value, uint64_t* n_out) {
    ScorerHost* sp = dij_scorer(c, id, "mqi_dij_get_hits");
    if (!sp) return MQI_ERR_INVALID;
    ScorerHost& s = *sp;
    if (!n_out) return fail(c, MQI_ERR_INVALID, "mqi_dij_get_hits: n_out is NULL");
    if (!s.hit_log) return fail(c, MQI_ERR_STATE, "mqi_dij_get_hits: recording is off (mqi_dij_record_hits)");
    DeviceGuard g(c->device);
    unsigned long long count = 0;
    MQI_CUDA(c, cudaMemcpyAsync(&count, s.hit_count, sizeof(count), cudaMemcpyDeviceToHost, c->stream),
             "mqi_dij_get_hits");
    MQI_CUDA(c, cudaStreamSynchronize(c->stream), "mqi_dij_get_hits");
    const uint64_t n = std::min<uint64_t>(count, s.hit_cap);
    *n_out = n;
    if (count > s.hit_cap)
        return fail(c, MQI_ERR_OVERFLOW, "mqi_dij_get_hits: more insertions than the log holds (" +
                                             std::to_string(count) + " > " + std::to_string(s.hit_cap) + ")");
    if (!voxel && !spot && !value) return MQI_OK;
    std::vector<DijHit> h(n);
    if (n) {
        MQI_CUDA(c, cudaMemcpyAsync(h.data(), s.hit_log, n * sizeof(DijHit), cudaMemcpyDeviceToHost, c->stream),
                 "mqi_dij_get_hits");
        MQI_CUDA(c, cudaStreamSynchronize(c->stream), "mqi_dij_get_hits");
    }
    for (uint64_t i = 0; i < n; ++i) {
        if (voxel) voxel[i] = h[i].voxel;
        if (spot) spot[i] = h[i].spot;
        if (value) value[i] = h[i].value;
    }
    return MQI_OK;
}

int
mqi_dij_build(mqi_ctx* c, int id, uint32_t n_spots, double scale, uint64_t* nnz_out) {
    ScorerHost* sp = dij_scorer(c, id, "mqi_dij_build");
    if (!sp) return MQI_ERR_INVALID;
    ScorerHost& s = *sp;
    if (n_spots == 0) n_spots = c->n_plan_spots;
    if (n_spots == 0) return fail(c, MQI_ERR_INVALID, "mqi_dij_build: n_spots is 0 and no spot plan is set");
    const ChildHost& ch = c->children[s.child];
    const uint64_t nvox = (uint64_t) ch.nx * ch.ny * ch.nz;
    DeviceGuard g(c->device);
    cudaStream_t st = c->stream;
    s.csr.built = false;
    unsigned long long count = 0;
    MQI_CUDA(c, dij_count(s.dij, s.dij_cap, s.dij_count, c->num_sms, st), "mqi_dij_build: count");
    MQI_CUDA(c, cudaMemcpyAsync(&count, s.dij_count, sizeof(count), cudaMemcpyDeviceToHost, st), "mqi_dij_build");
    MQI_CUDA(c, cudaStreamSynchronize(st), "mqi_dij_build");
    const uint64_t n = count;
    const int      vbits = bit_length(nvox - 1), sbits = bit_length((uint64_t) n_spots - 1);

    // the sort's buffers
    unsigned long long *keys, *keys_alt, *cursor;
    uint32_t *vals, *vals_alt, *hist, *offs, *scan, *bad;
    auto lay_out_scratch = [&](Carve cv) {
        const uint64_t hw = radix_hist_words(n);
        cv.take(keys, n + 1);
        cv.take(keys_alt, n + 1);
        cv.take(vals, n);
        cv.take(vals_alt, n);
        cv.take(hist, hw);
        cv.take(offs, hw);
        cv.take(scan, scan_scratch_words(hw));
        cv.take(cursor, 1);
        cv.take(bad, 1);
        return cv.used;
    };
    const size_t scratch_bytes = lay_out_scratch(Carve{});
    struct Trim {   // gives it back at the end, when it is large
        mqi_ctx* c;
        ~Trim() {
            if (c->build_scratch_bytes <= kKeepScratch) return;
            cudaFree(c->build_scratch);
            c->build_scratch       = nullptr;
            c->build_scratch_bytes = 0;
        }
    } trim{ c };

    // the matrix: segments of the backward are bounded by whole ones and one more per row, voxel rows by
    // the entries and by the voxels
    DijCsr m;
    m.spot16 = n_spots <= 65536;
    const uint64_t segment = dij_segment(n, c->num_sms);
    const uint64_t max_seg = n / segment + std::min<uint64_t>(n_spots, n), max_vrows = std::min(n, nvox);
    const uint64_t n_runs  = (n + kFwdEntries - 1) / kFwdEntries;
    auto lay_out = [&](Carve cv) {
        cv.take(m.s_indptr, (uint64_t) n_spots + 1);
        // entry arrays padded to whole groups of eight: the products read them in 16-byte pieces
        unsigned char* v_spot = nullptr;
        cv.take(m.s_voxel, n + 8);
        cv.take(m.s_value, n + 8);
        cv.take(v_spot, (n + 8) * (m.spot16 ? sizeof(uint16_t) : sizeof(uint32_t)));
        cv.take(m.v_value, n + 8);
        cv.take(m.v_row, max_vrows);
        cv.take(m.v_off, max_vrows);
        m.v_spot = v_spot;
        cv.take(m.seg_start, max_seg + 1);
        cv.take(m.row_seg, (uint64_t) n_spots + 1);
        cv.take(m.seg_order, max_seg);
        cv.take(m.partial, max_seg);
        cv.take(m.bwd_cursor, 1);
        cv.take(m.fwd_row_first, n_runs + 1);
        cv.take(m.fwd_run_k, n_runs + 1);
        return cv.used;
    };
    const size_t csr_bytes = lay_out(Carve{});
    // products queued on any stream may still read the last matrix
    if (s.csr.slab) MQI_CUDA(c, cudaDeviceSynchronize(), "mqi_dij_build");
    auto allocate = [&] {
        const cudaError_t e = ensure_bytes(c->build_scratch, c->build_scratch_bytes, scratch_bytes);
        return e == cudaSuccess ? ensure_bytes(s.csr.slab, s.csr.slab_bytes, csr_bytes) : e;
    };
    cudaError_t e = allocate();
    if (e == cudaErrorMemoryAllocation && give_back(c)) {   // which takes both of them too
        (void) cudaGetLastError();
        e = allocate();
    }
    MQI_CUDA(c, e, "mqi_dij_build: allocation");
    lay_out_scratch(Carve{ static_cast<char*>(c->build_scratch) });
    lay_out(Carve{ static_cast<char*>(s.csr.slab) });
    m.slab       = s.csr.slab;
    m.slab_bytes = s.csr.slab_bytes;
    m.n_spots    = n_spots;
    m.n_voxels   = nvox;
    m.nnz        = n;

    // 1. the table's entries, in any order
    MQI_CUDA(c, dij_compact(s.dij, s.dij_cap, vbits, n_spots, scale, keys, vals, n, cursor, bad, c->num_sms, st),
             "mqi_dij_build: compact");
    unsigned long long got = 0;
    uint32_t           is_bad = 0;
    MQI_CUDA(c, cudaMemcpyAsync(&got, cursor, sizeof(got), cudaMemcpyDeviceToHost, st), "mqi_dij_build");
    MQI_CUDA(c, cudaMemcpyAsync(&is_bad, bad, sizeof(is_bad), cudaMemcpyDeviceToHost, st), "mqi_dij_build");
    MQI_CUDA(c, cudaStreamSynchronize(st), "mqi_dij_build");
    if (got != n) return fail(c, MQI_ERR_DEVICE, "mqi_dij_build: occupied slots disagree with the insertion count");
    if (is_bad) return fail(c, MQI_ERR_INVALID, "mqi_dij_build: the table holds a spot index >= n_spots");

    // 2. voxel rows, spots ascending: by spot, then (stable) by voxel
    MQI_CUDA(c, radix_sort_pairs(keys, vals, keys_alt, vals_alt, n, vbits, sbits, hist, offs, scan, st), "mqi_dij_build: sort");
    MQI_CUDA(c, radix_sort_pairs(keys, vals, keys_alt, vals_alt, n, 0, vbits, hist, offs, scan, st), "mqi_dij_build: sort");
    MQI_CUDA(c, dij_count_rows(keys, n, vbits, offs, hist, scan, st), "mqi_dij_build");
    uint32_t tail[2] = { 0, 0 };
    if (n) {
        const uint64_t last = (n - 1) / kRowTile;
        MQI_CUDA(c, cudaMemcpyAsync(&tail[0], offs + last, sizeof(uint32_t), cudaMemcpyDeviceToHost, st), "mqi_dij_build");
        MQI_CUDA(c, cudaMemcpyAsync(&tail[1], hist + last, sizeof(uint32_t), cudaMemcpyDeviceToHost, st), "mqi_dij_build");
        MQI_CUDA(c, cudaStreamSynchronize(st), "mqi_dij_build");
    }
    m.n_vrows = (uint64_t) tail[0] + tail[1];
    // the forward runs' first rows are found from the rows' first entries, in the sort's spare buffer
    uint64_t* indptr_v = reinterpret_cast<uint64_t*>(keys_alt);
    if (n == 0) MQI_CUDA(c, cudaMemsetAsync(indptr_v, 0, sizeof(uint64_t), st), "mqi_dij_build");
    // the forward multiplies whole groups: spot 0 past the end
    MQI_CUDA(c, cudaMemsetAsync(static_cast<char*>(m.v_spot) + n * (m.spot16 ? 2 : 4), 0, 8 * (m.spot16 ? 2 : 4), st),
             "mqi_dij_build");
    MQI_CUDA(c, cudaMemsetAsync(m.v_value + n, 0, 8 * sizeof(float), st), "mqi_dij_build");
    MQI_CUDA(c, dij_voxel_rows(keys, vals, n, vbits, offs, m.v_row, m.v_off, indptr_v, m.v_spot, m.spot16, m.v_value, st),
             "mqi_dij_build");
    MQI_CUDA(c, dij_forward_blocks(indptr_v, m.n_vrows, n, m.fwd_row_first, m.fwd_run_k, &m.n_fwd_blocks, st),
             "mqi_dij_build");

    // 3. spot rows, voxels ascending: those sorted (stable) by spot
    MQI_CUDA(c, radix_sort_pairs(keys, vals, keys_alt, vals_alt, n, vbits, sbits, hist, offs, scan, st), "mqi_dij_build: sort");
    MQI_CUDA(c, dij_row_bounds(keys, n, vbits, n_spots, m.s_indptr, st), "mqi_dij_build");
    MQI_CUDA(c, dij_spot_rows(keys, vals, n, vbits, m.s_voxel, m.s_value, st), "mqi_dij_build");
    std::vector<uint64_t> indptr(n_spots + 1);
    MQI_CUDA(c, cudaMemcpyAsync(indptr.data(), m.s_indptr, indptr.size() * sizeof(uint64_t), cudaMemcpyDeviceToHost, st),
             "mqi_dij_build");
    MQI_CUDA(c, cudaStreamSynchronize(st), "mqi_dij_build");
    if (indptr[n_spots] != n) return fail(c, MQI_ERR_DEVICE, "mqi_dij_build: the sorted rows do not hold every entry");
    // backward segments: each row cut into runs of at most `segment` entries, and their work
    // order: by the voxel of their first entry (the sort buffers are free now)
    {
        std::vector<uint64_t> seg;
        std::vector<uint32_t> row_seg(n_spots + 1);
        for (uint32_t r = 0; r < n_spots; ++r) {
            row_seg[r] = (uint32_t) seg.size();
            for (uint64_t b = indptr[r]; b < indptr[r + 1]; b += segment) seg.push_back(b);
        }
        row_seg[n_spots] = (uint32_t) seg.size();
        m.n_seg = seg.size();
        seg.push_back(n);
        MQI_CUDA(c, cudaMemsetAsync(m.bwd_cursor, 0, sizeof(uint32_t), st), "mqi_dij_build");
        MQI_CUDA(c, cudaMemcpyAsync(m.seg_start, seg.data(), seg.size() * sizeof(uint64_t), cudaMemcpyHostToDevice, st),
                 "mqi_dij_build");
        MQI_CUDA(c, cudaMemcpyAsync(m.row_seg, row_seg.data(), row_seg.size() * sizeof(uint32_t), cudaMemcpyHostToDevice,
                                    st), "mqi_dij_build");
        if (m.n_seg) {
            MQI_CUDA(c, dij_seg_order_keys(m.seg_start, (uint32_t) m.n_seg, m.s_voxel, keys, vals, st), "mqi_dij_build");
            MQI_CUDA(c, radix_sort_pairs(keys, vals, keys_alt, vals_alt, m.n_seg, 0, vbits, hist, offs, scan, st),
                     "mqi_dij_build: sort");
            MQI_CUDA(c, cudaMemcpyAsync(m.seg_order, vals, m.n_seg * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st),
                     "mqi_dij_build");
        }
        MQI_CUDA(c, cudaStreamSynchronize(st), "mqi_dij_build");   // the host vectors are copied from
    }

    m.built = true;
    s.csr   = m;
    if (nnz_out) *nnz_out = n;
    return MQI_OK;
}

int
mqi_dij_get_csr(mqi_ctx* c, int id, uint64_t* indptr, uint32_t* indices, float* data, int on_device) {
    ScorerHost* sp = dij_scorer(c, id, "mqi_dij_get_csr");
    if (!sp) return MQI_ERR_INVALID;
    const DijCsr& m = sp->csr;
    if (!m.built) return fail(c, MQI_ERR_STATE, "mqi_dij_get_csr: call mqi_dij_build first");
    DeviceGuard g(c->device);
    const cudaMemcpyKind k = on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost;
    if (indptr) MQI_CUDA(c, cudaMemcpyAsync(indptr, m.s_indptr, (m.n_spots + 1) * sizeof(uint64_t), k, c->stream), "mqi_dij_get_csr");
    if (indices && m.nnz) MQI_CUDA(c, cudaMemcpyAsync(indices, m.s_voxel, m.nnz * sizeof(uint32_t), k, c->stream), "mqi_dij_get_csr");
    if (data && m.nnz) MQI_CUDA(c, cudaMemcpyAsync(data, m.s_value, m.nnz * sizeof(float), k, c->stream), "mqi_dij_get_csr");
    MQI_CUDA(c, cudaStreamSynchronize(c->stream), "mqi_dij_get_csr");
    return MQI_OK;
}

int
mqi_dij_info(mqi_ctx* c, int id, uint64_t* table_slots, uint64_t* occupied, uint64_t* nnz, uint64_t* n_voxel_rows) {
    ScorerHost* sp = dij_scorer(c, id, "mqi_dij_info");
    if (!sp) return MQI_ERR_INVALID;
    DeviceGuard g(c->device);
    unsigned long long occ = 0;
    MQI_CUDA(c, dij_count(sp->dij, sp->dij_cap, sp->dij_count, c->num_sms, c->stream), "mqi_dij_info");
    MQI_CUDA(c, cudaMemcpyAsync(&occ, sp->dij_count, sizeof(occ), cudaMemcpyDeviceToHost, c->stream), "mqi_dij_info");
    MQI_CUDA(c, cudaStreamSynchronize(c->stream), "mqi_dij_info");
    if (table_slots) *table_slots = sp->dij_cap;
    if (occupied) *occupied = occ;
    if (nnz) *nnz = sp->csr.built ? sp->csr.nnz : 0;
    if (n_voxel_rows) *n_voxel_rows = sp->csr.built ? sp->csr.n_vrows : 0;
    return MQI_OK;
}

int
mqi_dij_matvec(mqi_ctx* c, int id, const void* w, void* dose, int fp64, int on_device) {
    ScorerHost* sp = dij_scorer(c, id, "mqi_dij_matvec");
    if (!sp) return MQI_ERR_INVALID;
    const DijCsr& m = sp->csr;
    if (!m.built) return fail(c, MQI_ERR_STATE, "mqi_dij_matvec: call mqi_dij_build first");
    if (!w || !dose) return fail(c, MQI_ERR_INVALID, "mqi_dij_matvec: NULL buffer");
    DeviceGuard g(c->device);
    const size_t es = fp64 ? sizeof(double) : sizeof(float);
    Scratch sc;
    const void* dw = w;
    void*       dd = dose;
    if (!on_device) {
        char *tw, *td;
        MQI_CUDA(c, sc.alloc(c, tw, m.n_spots * es), "mqi_dij_matvec");
        MQI_CUDA(c, sc.alloc(c, td, m.n_voxels * es), "mqi_dij_matvec");
        MQI_CUDA(c, cudaMemcpyAsync(tw, w, m.n_spots * es, cudaMemcpyHostToDevice, c->stream), "mqi_dij_matvec");
        dw = tw;
        dd = td;
    }
    MQI_CUDA(c, cudaMemsetAsync(dd, 0, m.n_voxels * es, c->stream), "mqi_dij_matvec");
    MQI_CUDA(c, dij_forward(m.v_row, m.v_off, m.fwd_row_first, m.fwd_run_k, m.n_fwd_blocks, m.v_spot, m.spot16,
                            m.v_value, dw, dd, fp64, c->counters + 3, c->num_sms, c->stream), "mqi_dij_matvec");
    if (!on_device) {
        uint32_t flag = 0;
        MQI_CUDA(c, cudaMemcpyAsync(dose, dd, m.n_voxels * es, cudaMemcpyDeviceToHost, c->stream), "mqi_dij_matvec");
        MQI_CUDA(c, cudaMemcpyAsync(&flag, c->counters + 3, sizeof(flag), cudaMemcpyDeviceToHost, c->stream),
                 "mqi_dij_matvec");
        MQI_CUDA(c, cudaStreamSynchronize(c->stream), "mqi_dij_matvec");
        if (flag & 8u) return fail(c, MQI_ERR_DEVICE, "mqi_dij_matvec: a bulk copy did not complete");
    }
    return MQI_OK;
}

int
mqi_dij_rmatvec(mqi_ctx* c, int id, const void* gin, void* grad, int fp64, int on_device) {
    ScorerHost* sp = dij_scorer(c, id, "mqi_dij_rmatvec");
    if (!sp) return MQI_ERR_INVALID;
    const DijCsr& m = sp->csr;
    if (!m.built) return fail(c, MQI_ERR_STATE, "mqi_dij_rmatvec: call mqi_dij_build first");
    if (!gin || !grad) return fail(c, MQI_ERR_INVALID, "mqi_dij_rmatvec: NULL buffer");
    DeviceGuard g(c->device);
    const size_t es = fp64 ? sizeof(double) : sizeof(float);
    Scratch sc;
    const void* dg = gin;
    void*       dr = grad;
    if (!on_device) {
        char *tg, *tr;
        MQI_CUDA(c, sc.alloc(c, tg, m.n_voxels * es), "mqi_dij_rmatvec");
        MQI_CUDA(c, sc.alloc(c, tr, m.n_spots * es), "mqi_dij_rmatvec");
        MQI_CUDA(c, cudaMemcpyAsync(tg, gin, m.n_voxels * es, cudaMemcpyHostToDevice, c->stream), "mqi_dij_rmatvec");
        dg = tg;
        dr = tr;
    }
    MQI_CUDA(c, dij_backward(m.seg_order, m.seg_start, (uint32_t) m.n_seg, m.row_seg, m.n_spots, m.s_voxel, m.s_value,
                             m.partial, m.bwd_cursor, dg, dr, fp64, c->num_sms, c->stream), "mqi_dij_rmatvec");
    if (!on_device) {
        MQI_CUDA(c, cudaMemcpyAsync(grad, dr, m.n_spots * es, cudaMemcpyDeviceToHost, c->stream), "mqi_dij_rmatvec");
        MQI_CUDA(c, cudaStreamSynchronize(c->stream), "mqi_dij_rmatvec");
    }
    return MQI_OK;
}

}   // extern "C"
