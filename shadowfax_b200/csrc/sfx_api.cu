/*
 * C-ABI front end of the sfxflux library: contexts, mesh upload (VorTess
 * face-list contract -> device structure-of-arrays), state transfer, the
 * step driver and the parity entry points.  See include/sfxflux.h.
 */
#include <cuda_runtime.h>

#include <cstdio>
#include <atomic>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <new>
#include <unordered_map>
#include <utility>
#include <vector>

#include "sfx_internal.h"

/* A context outlives its meshes: sfx_ctx_destroy on a context that still has
 * meshes only marks it, and the last sfx_mesh_free releases it.  Callers that
 * free in any order (garbage-collected bindings) stay safe. */
struct sfx_ctx {
    sfx_config cfg;
    sfx_solver_params sp;
    cudaStream_t own_stream = nullptr;
    cudaStream_t stream = nullptr;
    int live_meshes = 0;
    bool closing = false;
    /* Keeps one of the driver's 2 MB chunks for small allocations in use from the
     * first block of less than a megabyte on: a mesh is one block, and with no
     * chunk in use making and freeing a small one waits 600 us for a chunk to be
     * mapped and unmapped (a clone of 2,000 cells in 2D 630 us, 14 with it). */
    void* chunk = nullptr;
};

struct sfx_mesh {
    sfx_ctx* ctx = nullptr;
    sfx_dmesh d;
    std::vector<void*> allocs;
    /* split pass: the mesh as a one-member launch group, so that a mesh
     * stepped alone runs the same kernels, and so the same arithmetic, as
     * in a group with other meshes */
    sfx_group_entry* self_tab = nullptr;
    int32_t* self_pre = nullptr;
    float self_dt = 0.f; /* time step held in self_tab (0: none yet) */
    bool clone = false;  /* geometry shared with the base mesh */
    /* split meshes: the CSR entries that name the other copy of a periodic face
     * pair (sfx_mesh_upload), as {position, the cell's own face} */
    std::shared_ptr<const std::vector<std::pair<int64_t, int32_t>>> merged;
    /* a plain-FP64 clone of a split mesh has a CSR of its own; the split one, for
     * split clones of it in turn */
    int32_t* split_idx = nullptr;
    int2* split_ent = nullptr;
    unsigned long long* d_smin = nullptr; /* local time steps: smallest new step */
    /* room for d.vgen, d.newpos and d.vel in the block of a small mesh (keeps_moving) */
    double *kept_vgen = nullptr, *kept_newpos = nullptr, *kept_vel = nullptr;
};

namespace {

int cuda_ok(cudaError_t e) {
    return e == cudaSuccess ? SFX_OK : SFX_ERR_CUDA;
}

#define SFX_TRY(x)                       \
    do {                                 \
        int _rc = (x);                   \
        if(_rc != SFX_OK) return _rc;    \
    } while(0)

template <typename T>
int dalloc(sfx_mesh* m, T** p, size_t count) {
    *p = nullptr;
    if(count == 0) count = 1;
    void* q = nullptr;
    cudaError_t e = cudaMalloc(&q, count * sizeof(T));
    if(e != cudaSuccess) {
        cudaGetLastError();
        return e == cudaErrorMemoryAllocation ? SFX_ERR_NOMEM : SFX_ERR_CUDA;
    }
    m->allocs.push_back(q);
    *p = (T*)q;
    return SFX_OK;
}

template <typename T>
int h2d(T* dst, const T* src, size_t count, cudaStream_t s) {
    if(count == 0) return SFX_OK;
    return cuda_ok(cudaMemcpyAsync(dst, src, count * sizeof(T), cudaMemcpyHostToDevice, s));
}

/* the status of an error record, its index into st */
int read_err(const sfx_dev_error& e, sfx_stats* st) {
    int status = SFX_OK;
    if(st) {
        st->bad_face = -1;
        st->bad_cell = -1;
    }
    if(e.face_key != ~0ull) {
        status = (int)(e.face_key & 0xff);
        if(st) st->bad_face = (int32_t)(e.face_key >> 8);
    } else if(e.cell_key != ~0ull) {
        status = (int)(e.cell_key & 0xff);
        if(st) st->bad_cell = (int32_t)(e.cell_key >> 8);
    }
    if(st) st->status = status;
    return status;
}

int check_err(sfx_mesh* m, sfx_stats* st) {
    sfx_dev_error e;
    cudaStream_t s = m->ctx->stream;
    SFX_TRY(cuda_ok(cudaMemcpyAsync(&e, m->d.err, sizeof e, cudaMemcpyDeviceToHost, s)));
    SFX_TRY(cuda_ok(cudaStreamSynchronize(s)));
    return read_err(e, st);
}

/* the error record and the totals of a call of `steps` steps, in one copy */
int collect_stats(sfx_mesh* m, int steps, sfx_stats* st) {
    std::memset(st, 0, sizeof *st);
    st->steps_done = -1;
    double t[7];
    const int S = m->d.S;
    SFX_TRY(sfx_fp64_totals(&m->d, t, m->ctx->stream));
    sfx_dev_error e;
    std::memcpy(&e.face_key, &t[S], sizeof e.face_key);
    std::memcpy(&e.cell_key, &t[S + 1], sizeof e.cell_key);
    const int rc = read_err(e, st);
    if(rc == SFX_OK) st->steps_done = steps;
    std::memcpy(st->totals, t, sizeof(double) * S);
    return rc;
}

/* host rows [n][w] -> device field-major [w][n], through the device array
 * stage; the host array may be reused on return when it is pageable */
int rows_in(double* dst, const double* src, int64_t n, int w, double* stage, cudaStream_t s) {
    SFX_TRY(h2d(stage, src, (size_t)n * w, s));
    return sfx_from_rows(stage, n, w, dst, s);
}

/* one phase of a step: 0 gradients, 1 face fluxes, 2 update */
/* queued slow faces per mesh: room for every face, so the face kernel never
 * has to run Brent's method itself (and carries none of its code) */
int32_t slowq_capacity(int64_t n_faces) {
    return (int32_t)(n_faces > 0 ? n_faces : 1);
}

/* doubles of the split pass's dQ per face (store_dq, sfx_split.cu) */
int64_t split_dq_doubles(int dim) {
    return dim == 3 ? 4 : 3;
}

/* a one-member group's prefix sums and, last, the word behind them */
constexpr int kSelfPre = 7;

/* device table of a split mesh as a one-member launch group */
int setup_self(sfx_mesh* m, cudaStream_t s) {
    sfx_group_entry e;
    std::memset(&e, 0, sizeof e);
    e.m = m->d;
    m->self_dt = 0.f;
    SFX_TRY(cuda_ok(cudaMemsetAsync(m->self_pre, 0, kSelfPre * sizeof(int32_t), s)));
    /* pageable source: staged before the call returns */
    return h2d(m->self_tab, &e, 1, s);
}

/* doubles of one of the plain-FP64 pass's records */
size_t rec_doubles(int dim, int what) {
    return (size_t)sfx_fp64_record_bytes(dim, what) / sizeof(double);
}

int run_phase(sfx_mesh* m, int phase, double dt, int write_branch, cudaStream_t s) {
    sfx_ctx* c = m->ctx;
    if(c->cfg.precision == SFX_PREC_SPLIT) {
        const float fdt = (float)dt;
        if(phase == 1 && fdt != m->self_dt) {
            m->self_dt = fdt;
            SFX_TRY(h2d(&m->self_tab->dt, &m->self_dt, 1, s));
        }
        sfx_group_dev g;
        std::memset(&g, 0, sizeof g);
        g.tab = m->self_tab;
        g.pre = m->self_pre;
        g.n_meshes = 1;
        g.dim = m->d.dim;
        g.lanes = m->d.lanes;
        g.face_variant = m->d.face_variant;
        g.moving = m->d.vel != nullptr ? 1 : 0; /* split meshes get face velocities
                                                   only from sfx_step_moving */
        sfx_split_blocks(m->d.dim, m->d.lanes, m->d.n_cells, m->d.n_faces, g.blocks);
        if(m->d.ranged) {
            /* one part of a mesh: the phases' own ranges */
            int32_t b[3];
            sfx_split_blocks(m->d.dim, m->d.lanes, sfx_grad_cells(m->d), sfx_flux_faces(m->d), b);
            g.blocks[0] = b[0];
            g.blocks[1] = b[1];
            sfx_split_blocks(m->d.dim, m->d.lanes, sfx_update_cells(m->d), 0, b);
            g.blocks[2] = b[2];
            if(phase == 0 && g.blocks[0] == 0) {
                /* no gradient launch to empty the queue (a part without cells) */
                SFX_TRY(cuda_ok(cudaMemsetAsync(m->d.slowq_n, 0, sizeof(int32_t), s)));
                SFX_TRY(cuda_ok(cudaMemsetAsync(m->self_pre + kSelfPre - 1, 0, sizeof(int32_t), s)));
            }
        }
        return sfx_split_group_phase(&g, phase, &c->sp, s);
    }
    switch(phase) {
    case 0:
        return sfx_fp64_gradients(&m->d, &c->sp, s);
    case 1:
        return sfx_fp64_faces(&m->d, &c->sp, dt, write_branch, s);
    default:
        return sfx_fp64_apply(&m->d, &c->sp, s);
    }
}

int reset_err_on(sfx_mesh* m, cudaStream_t s) {
    return cuda_ok(cudaMemsetAsync(m->d.err, 0xff, sizeof(sfx_dev_error), s)); /* ~0 keys */
}

int reset_err(sfx_mesh* m) {
    return reset_err_on(m, m->ctx->stream);
}

/* Arrays carved from one device block (256-byte aligned each): a mesh has
 * about thirty, and an allocation of its own for each cost more than the
 * copies that fill them on small meshes. */
struct Carver {
    struct Slot {
        void** p;
        size_t bytes;
    };
    std::vector<Slot> slots;
    template <typename T>
    void add(T** p, size_t count) {
        slots.push_back({(void**)p, (count ? count : 1) * sizeof(T)});
    }
    int allocate(sfx_mesh* m) {
        size_t total = 0;
        for(const Slot& sl : slots) total = ((total + 255) & ~(size_t)255) + sl.bytes;
        uint8_t* block = nullptr;
        SFX_TRY(dalloc(m, &block, total));
        void** chunk = &m->ctx->chunk; /* beside this block, where it is a small one */
        if(total < (1 << 20) && !*chunk && cudaMalloc(chunk, 256) != cudaSuccess) {
            cudaGetLastError();
            *chunk = nullptr;
        }
        size_t off = 0;
        for(const Slot& sl : slots) {
            off = (off + 255) & ~(size_t)255;
            *sl.p = block + off;
            off += sl.bytes;
        }
        return SFX_OK;
    }
};

/* The staging rows: a state, and for plain FP64 at least one row of gradients and
 * all of a small mesh's; a second state on its way in goes through the dQ scratch
 * (dq doubles) when that holds it, otherwise behind the first. */
size_t stage_doubles(int64_t n, int dim, bool split, size_t dq) {
    const size_t ns = (size_t)n * (dim + 2), row = (size_t)dim * (dim + 2);
    const size_t rows = split ? 0 : std::max(row, std::min<size_t>(n * row, 16384));
    return std::max(dq >= ns ? ns : 2 * ns, rows);
}

void add_stage(Carver& arrays, sfx_dmesh& d, bool split, size_t dq) {
    arrays.add(&d.stage, stage_doubles(d.n_cells, d.dim, split, dq));
}

void set_stage(sfx_dmesh& d, bool split, size_t dq) {
    const size_t ns = (size_t)d.n_cells * d.S;
    d.stage2 = dq < ns ? d.stage + ns : split ? d.dq : d.dQf;
}

/* Whether an upload sets aside the arrays of a moving step: a mesh whose first
 * step_moving allocates them pays 250 to 350 us for it and as much when it is
 * freed, more than the step; they are at most a megabyte here. */
bool keeps_moving(int dim, int64_t n, int64_t F) {
    return 8 * dim * (2 * n + F) <= 1 << 20;
}

/* a plain-FP64 mesh's state and per-step scratch: the pass's records, or without
 * them the field-major gradients and dQ of its caller-owned form */
void add_fp64_state(Carver& arrays, sfx_dmesh& d, bool records) {
    const size_t n = (size_t)d.n_cells, F = (size_t)d.n_faces;
    d.grad = d.ws = d.grec = d.dQf = nullptr;
    d.listed = d.listed_n = nullptr;
    if(!records) {
        arrays.add(&d.grad, n * d.dim * d.S);
        arrays.add(&d.dQf, F * d.S);
        return;
    }
    arrays.add(&d.ws, n * rec_doubles(d.dim, SFX_REC_WS));
    arrays.add(&d.grec, n * rec_doubles(d.dim, SFX_REC_GREC));
    arrays.add(&d.dQf, F * rec_doubles(d.dim, SFX_REC_DQ));
    arrays.add(&d.listed, (size_t)sfx_fp64_list_room(F));
    arrays.add(&d.listed_n, 1);
}

/* doubles of a mesh's dQ scratch */
size_t dq_doubles(const sfx_dmesh& d, bool split, bool records) {
    const size_t F = (size_t)d.n_faces;
    return F * (split ? split_dq_doubles(d.dim)
                      : records ? rec_doubles(d.dim, SFX_REC_DQ) : (size_t)d.S);
}

/* the arrays that add(arrays, records) names: with the plain-FP64 records, or,
 * where those do not fit on the device, without (3D: 1,220 bytes per cell
 * instead of 3,470; the same bits from the kernels of caller-owned arrays: 419 us
 * a step instead of 172 on 65,537 cells in 3D with HLLC, 838 instead of 376 with
 * the exact solver, 181 instead of 128 on 150,001 cells in 2D with HLLC) */
template <typename Add>
int allocate_fp64(sfx_mesh* m, bool records, Add add) {
    for(;; records = false) {
        Carver arrays;
        add(arrays, records);
        const int rc = arrays.allocate(m);
        if(rc != SFX_ERR_NOMEM || !records) return rc;
    }
}

/* The CSR with each cell's faces in ascending order, when `idx` does not list
 * them so (empty otherwise): the reference adds each face's dQ to its cells in
 * its face loop (src/VorTessManager.cpp:198-212), while a cell's gradient walks
 * the cell's own face list (src/VorCell.cpp:464-530) */
std::vector<int32_t> ascending_csr(const int32_t* off, const std::vector<int32_t>& idx,
                                   int64_t n) {
    std::vector<int32_t> out;
    bool ascending = true;
    for(int64_t i = 0; i < n && ascending; ++i)
        for(int64_t j = off[i] + 1; j < off[i + 1]; ++j)
            if((idx[j] & 0x7fffffff) < (idx[j - 1] & 0x7fffffff)) {
                ascending = false;
                break;
            }
    if(ascending) return out;
    out = idx;
    for(int64_t i = 0; i < n; ++i)
        std::sort(out.begin() + off[i], out.begin() + off[i + 1],
                  [](int32_t a, int32_t b) { return (a & 0x7fffffff) < (b & 0x7fffffff); });
    return out;
}

/* What a plain-FP64 clone of a split mesh cannot share: the pass's face records
 * (formed here from the base's geometry) and a CSR in which every cell names
 * its own copy of a periodic face, in the FP64 update's order */
int fill_fp64_geometry(sfx_mesh* m, cudaStream_t s) {
    sfx_dmesh& d = m->d;
    std::vector<int32_t> off((size_t)d.n_cells + 1), idx((size_t)d.nnz);
    SFX_TRY(cuda_ok(cudaMemcpyAsync(off.data(), d.off, off.size() * sizeof(int32_t),
                                    cudaMemcpyDeviceToHost, s)));
    SFX_TRY(cuda_ok(cudaMemcpyAsync(idx.data(), m->split_idx, idx.size() * sizeof(int32_t),
                                    cudaMemcpyDeviceToHost, s)));
    SFX_TRY(cuda_ok(cudaStreamSynchronize(s)));
    if(m->merged)
        for(const auto& e : *m->merged) idx[(size_t)e.first] = e.second;
    const std::vector<int32_t> aidx = ascending_csr(off.data(), idx, d.n_cells);
    SFX_TRY(h2d(d.idx, idx.data(), idx.size(), s));
    SFX_TRY(h2d(d.aidx, (aidx.empty() ? idx : aidx).data(), idx.size(), s));
    if(d.ws) {
        SFX_TRY(sfx_fp64_csr_neighbours(&d, s));
        SFX_TRY(sfx_fp64_face_records(&d, s));
    }
    return cuda_ok(cudaStreamSynchronize(s)); /* the host vectors end here */
}

/* a state on base's geometry: one device block carved into the arrays,
 * set up on stream s (waited for when `wait`) */
int clone_impl(sfx_ctx* ctx, sfx_mesh* base, cudaStream_t s, bool wait, sfx_mesh** out) {
    if(!ctx || !base || !out) return SFX_ERR_INVALID;
    *out = nullptr;
    const sfx_dmesh& b = base->d;
    const bool split = ctx->cfg.precision == SFX_PREC_SPLIT;
    if(ctx->cfg.dim != b.dim || ctx->closing) return SFX_ERR_INVALID;
    if(split && !b.fg) return SFX_ERR_INVALID; /* base has no split geometry */
    if(cudaSetDevice(ctx->cfg.device) != cudaSuccess) return SFX_ERR_CUDA;
    sfx_mesh* m = new(std::nothrow) sfx_mesh;
    if(!m) return SFX_ERR_NOMEM;
    m->ctx = ctx;
    ctx->live_meshes++;
    m->d = b; /* geometry pointers shared with the base */
    m->clone = true;
    m->merged = base->merged;
    m->d.vgen = m->d.newpos = nullptr;
    m->d.tstart = m->d.tend = nullptr;
    m->d_smin = nullptr;
    sfx_dmesh& d = m->d;
    const int64_t n = d.n_cells, F = d.n_faces;
    const int S = d.S, dim = d.dim;
    d.W = d.Q = d.stage = d.stage2 = d.grad = d.dQf = d.ws = d.grec = nullptr;
    d.listed = d.listed_n = nullptr;
    d.branch = nullptr;
    d.err = nullptr;
    d.totals_scratch = nullptr;
    d.cw = d.cg = d.cdw = nullptr;
    d.dq = nullptr;
    d.slowq = nullptr;
    d.slowq_n = nullptr;
    d.slowq_cap = 0;
    if(split) {
        /* of an FP64 clone of a split mesh: that mesh's CSR again */
        d.ggeo = d.fgeo = nullptr;
        if(base->split_idx) {
            d.idx = base->split_idx;
            d.ent = base->split_ent;
        }
    }
    const bool geometry = !split && b.fg && !b.ggeo; /* the base is split */
    if(!split) {
        m->split_idx = geometry && !base->split_idx ? d.idx : base->split_idx;
        m->split_ent = geometry && !base->split_ent ? d.ent : base->split_ent;
    }
    int rc = allocate_fp64(m, !split && (geometry || b.ggeo), [&](Carver& arrays, bool records) {
        auto A = [&](auto** p, size_t c) { arrays.add(p, c); };
        A(&d.W, n * S);
        A(&d.Q, n * S);
        add_stage(arrays, d, split, dq_doubles(d, split, records));
        A(&d.err, 1);
        A(&d.totals_scratch, (size_t)(S + 1) * 1024);
        if(split) {
            A(&d.cw, 2 * n);
            A(&d.cg, (size_t)sfx_split_grad_vec4(dim) * n);
            A(&d.cdw, (size_t)sfx_split_dwdt_vec4(dim) * n);
            A(&d.dq, split_dq_doubles(dim) * F);
            d.slowq_cap = slowq_capacity(F);
            A(&d.slowq, (size_t)d.slowq_cap);
            A(&d.slowq_n, 1);
            A(&m->self_tab, 1);
            A(&m->self_pre, kSelfPre);
            return;
        }
        add_fp64_state(arrays, d, records);
        A(&d.branch, F);
        if(geometry) {
            if(records) {
                A(&d.ggeo, F * rec_doubles(dim, SFX_REC_GGEO));
                A(&d.fgeo, F * rec_doubles(dim, SFX_REC_FGEO));
                A(&d.ent, d.nnz);
            }
            A(&d.idx, d.nnz);
            A(&d.aidx, d.nnz);
        }
    });
    if(!rc) set_stage(d, split, dq_doubles(d, split, d.ws != nullptr));
    if(!rc) rc = reset_err_on(m, s);
    if(!rc && split) rc = cuda_ok(cudaMemsetAsync(d.slowq_n, 0, sizeof(int32_t), s));
    if(!rc && split) rc = setup_self(m, s);
    if(!rc && geometry) rc = fill_fp64_geometry(m, s);
    if(!rc && wait) rc = cuda_ok(cudaStreamSynchronize(s));
    if(rc) {
        sfx_mesh_free(m);
        return rc;
    }
    *out = m;
    return SFX_OK;
}

}  // namespace

sfx_dmesh* sfx_mesh_dev(sfx_mesh* m) {
    return &m->d;
}
int sfx_mesh_last_status(sfx_mesh* m, int32_t* bad_index) {
    sfx_stats st;
    std::memset(&st, 0, sizeof st);
    const int rc = check_err(m, &st);
    if(bad_index) *bad_index = st.bad_face >= 0 ? st.bad_face : st.bad_cell;
    return rc;
}
sfx_ctx* sfx_mesh_ctx(sfx_mesh* m) {
    return m->ctx;
}
void* sfx_ctx_stream(sfx_ctx* c) {
    return (void*)c->stream;
}
const sfx_config* sfx_ctx_config(sfx_ctx* c) {
    return &c->cfg;
}
const sfx_solver_params* sfx_ctx_params(sfx_ctx* c) {
    return &c->sp;
}

namespace {
std::atomic<long long> g_launches{0};
thread_local bool t_capturing = false;
}  // namespace

void sfx_count_launches(int n) {
    if(!t_capturing) g_launches.fetch_add(n, std::memory_order_relaxed);
}

void sfx_launch_capture(bool on) {
    t_capturing = on;
}

extern "C" {

int64_t sfx_launch_count(void) {
    return g_launches.load(std::memory_order_relaxed);
}

const char* sfx_version(void) {
    return "sfxflux 0.1 (sm_100a)";
}

int sfx_ctx_create(const sfx_config* cfg, sfx_ctx** out) {
    if(!cfg || !out) return SFX_ERR_INVALID;
    *out = nullptr;
    if(cfg->dim != 2 && cfg->dim != 3) return SFX_ERR_INVALID;
    if(cfg->solver != SFX_SOLVER_EXACT && cfg->solver != SFX_SOLVER_HLLC)
        return SFX_ERR_UNSUPPORTED;
    if(cfg->precision != SFX_PREC_FP64 && cfg->precision != SFX_PREC_SPLIT)
        return SFX_ERR_INVALID;
    if(!(cfg->gamma > 1.)) return SFX_ERR_INVALID;
    int ndev = 0;
    if(cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return SFX_ERR_CUDA;
    }
    if(cfg->device < 0 || cfg->device >= ndev) return SFX_ERR_INVALID;
    SFX_TRY(cuda_ok(cudaSetDevice(cfg->device)));
    sfx_ctx* c = new(std::nothrow) sfx_ctx;
    if(!c) return SFX_ERR_NOMEM;
    c->cfg = *cfg;
    sfx_solver_params_init(&c->sp, cfg->solver, cfg->gamma, cfg->tolerance, cfg->cutoff);
    if(cudaStreamCreateWithFlags(&c->own_stream, cudaStreamNonBlocking) != cudaSuccess) {
        delete c;
        return SFX_ERR_CUDA;
    }
    c->stream = c->own_stream;
    *out = c;
    return SFX_OK;
}

static void ctx_release(sfx_ctx* ctx) {
    cudaSetDevice(ctx->cfg.device);
    if(ctx->own_stream) {
        cudaStreamSynchronize(ctx->own_stream);
        cudaStreamDestroy(ctx->own_stream);
    }
    if(ctx->chunk) cudaFree(ctx->chunk);
    delete ctx;
}

int sfx_ctx_destroy(sfx_ctx* ctx) {
    if(!ctx || ctx->closing) return SFX_ERR_INVALID;
    ctx->closing = true;
    if(ctx->live_meshes > 0) return SFX_OK; /* released with the last mesh */
    ctx_release(ctx);
    return SFX_OK;
}

int sfx_ctx_set_stream(sfx_ctx* ctx, void* stream) {
    if(!ctx) return SFX_ERR_INVALID;
    ctx->stream = stream ? (cudaStream_t)stream : ctx->own_stream;
    return SFX_OK;
}

int sfx_ctx_synchronize(sfx_ctx* ctx) {
    if(!ctx) return SFX_ERR_INVALID;
    return cuda_ok(cudaStreamSynchronize(ctx->stream));
}

int64_t sfx_mesh_device_bytes(int32_t dim, int32_t n_cells, int32_t n_faces,
                              int64_t nnz, int32_t precision) {
    const int64_t S = dim + 2, n = n_cells, F = n_faces;
    const bool split = precision == SFX_PREC_SPLIT;
    const size_t dq = (size_t)F * (split ? split_dq_doubles(dim) : rec_doubles(dim, SFX_REC_DQ));
    int64_t cells = n * (8 * (2 * dim + 2 + 2 * S) + 4) + 4 +
                    8 * (int64_t)stage_doubles(n, dim, split, dq);
    int64_t faces = F * (8 * (1 + 2 * dim) + 4 * 4);
    int64_t bytes = cells + faces + nnz * 4 + 8 * 8 * 1024 + 4096;
    if(precision != SFX_PREC_SPLIT) {
        /* the records; the update's CSR copy (cells not in ascending face
         * order); face velocities */
        auto rec = [&](int what) { return (int64_t)sfx_fp64_record_bytes(dim, what); };
        bytes += n * (rec(SFX_REC_WS) + rec(SFX_REC_GREC)) +
                 F * (rec(SFX_REC_DQ) + rec(SFX_REC_GGEO) + rec(SFX_REC_FGEO) + 8 * dim) +
                 4 * sfx_fp64_list_room(F) + nnz * 4;
    } else {
        bytes += F * 8 * (dim + S); /* face velocities, dQf */
    }
    if(precision == SFX_PREC_SPLIT) {
        /* fg, fr, an, dq, queue; cw, cg, cx, self table */
        bytes += F * (32 + 4 * 12 + 8 * dim + 8 * split_dq_doubles(dim)) +
                 4 * slowq_capacity(F) + 4;
        bytes += n * (32 + 16 * (sfx_split_grad_vec4((int)dim) + sfx_split_dwdt_vec4((int)dim)) +
                      16) + 256;
    }
    bytes += nnz * 8; /* ent */
    if(keeps_moving(dim, n, F)) bytes += 16 * dim * n;
    return bytes;
}

namespace {

/* The host checks of a face list (sfx_mesh_check, and sfx_mesh_upload before
 * it allocates anything): every index a kernel will dereference, so device
 * code needs no bounds checks on mesh indices, and the one geometric
 * condition the split kernels rely on. */
int check_desc(const sfx_mesh_desc* desc, int precision) {
    const int dim = desc->dim;
    const int64_t n = desc->n_cells, F = desc->n_faces;
    if(n <= 0 || F < 0) return SFX_ERR_INVALID;
    if(!desc->cell_pos || !desc->cell_centroid || !desc->cell_volume ||
       !desc->cell_total_area || !desc->cell_face_offset || !desc->cell_face_index ||
       (F && (!desc->face_area || !desc->face_midpoint || !desc->face_left ||
              !desc->face_right || !desc->face_kind || !desc->face_right_pos)))
        return SFX_ERR_INVALID;
    const int32_t* off = desc->cell_face_offset;
    if(off[0] != 0) return SFX_ERR_BOUNDS;
    for(int64_t i = 0; i < n; ++i)
        if(off[i + 1] < off[i]) return SFX_ERR_BOUNDS;
    for(int64_t f = 0; f < F; ++f) {
        int L = desc->face_left[f], R = desc->face_right[f], k = desc->face_kind[f];
        if(L < 0 || L >= n) return SFX_ERR_BOUNDS;
        if(k == SFX_FACE_REAL || k == SFX_FACE_PERIODIC) {
            if(R < 0 || R >= n) return SFX_ERR_BOUNDS;
        } else if(k != SFX_FACE_MIRROR) {
            return SFX_ERR_BOUNDS;
        }
    }
    /* a cell lists the faces it owns and the real faces it is the right side of */
    for(int64_t i = 0; i < n; ++i)
        for(int64_t j = off[i]; j < off[i + 1]; ++j) {
            const int32_t f = desc->cell_face_index[j];
            if(f < 0 || f >= F) return SFX_ERR_BOUNDS;
            if(desc->face_left[f] != i &&
               !(desc->face_right[f] == i && desc->face_kind[f] == SFX_FACE_REAL))
                return SFX_ERR_BOUNDS;
        }
    if(precision == SFX_PREC_SPLIT) {
        /* the split kernels apply a periodic image's offset as one whole unit
         * box per axis (a code per axis: 0, +1 or -1); a mesh of another box
         * is refused rather than computed with the wrong offset */
        for(int64_t f = 0; f < F; ++f) {
            if(desc->face_kind[f] != SFX_FACE_PERIODIC) continue;
            for(int l = 0; l < dim; ++l) {
                const double a = std::fabs(desc->face_right_pos[f * dim + l] -
                                           desc->cell_pos[(int64_t)desc->face_right[f] * dim + l]);
                if(!(a <= 1e-9 || std::fabs(a - 1.) <= 1e-9)) return SFX_ERR_UNSUPPORTED;
            }
        }
    }
    return SFX_OK;
}

}  // namespace

int sfx_mesh_check(const sfx_mesh_desc* desc, int32_t precision) {
    if(!desc || (desc->dim != 2 && desc->dim != 3) ||
       (precision != SFX_PREC_FP64 && precision != SFX_PREC_SPLIT))
        return SFX_ERR_INVALID;
    return check_desc(desc, precision);
}

int sfx_mesh_upload(sfx_ctx* ctx, const sfx_mesh_desc* desc, sfx_mesh** out) {
    if(!ctx || !desc || !out) return SFX_ERR_INVALID;
    *out = nullptr;
    const int dim = desc->dim;
    if(dim != ctx->cfg.dim) return SFX_ERR_INVALID;
    SFX_TRY(check_desc(desc, ctx->cfg.precision));
    const int64_t n = desc->n_cells, F = desc->n_faces;
    const int32_t* off = desc->cell_face_offset;
    const int64_t nnz = off[n];
    std::vector<int32_t> idx(nnz);
    for(int64_t i = 0; i < n; ++i) {
        for(int64_t j = off[i]; j < off[i + 1]; ++j) {
            int32_t f = desc->cell_face_index[j];
            if(f < 0 || f >= F) return SFX_ERR_BOUNDS;
            if(desc->face_left[f] == i) {
                idx[j] = f;
            } else if(desc->face_right[f] == i && desc->face_kind[f] == SFX_FACE_REAL) {
                idx[j] = (int32_t)((uint32_t)f | 0x80000000u);
            } else {
                return SFX_ERR_BOUNDS;
            }
        }
    }
    /* The builder's cells list their faces in ascending order and one CSR serves
     * both passes; otherwise the plain-FP64 update gets a sorted copy, so that
     * its sums round as the reference's. */
    std::vector<int32_t> aidx;
    if(ctx->cfg.precision == SFX_PREC_FP64) aidx = ascending_csr(off, idx, n);
    /* Split pass only: a face across a periodic boundary is listed twice, once
     * owned by each cell (the reference computes it twice and lets each copy
     * update only its owner, src/VorFace.cpp:913-955).  The split pass
     * applies one copy's flux to both cells: the other copy's owner takes its
     * negated flux (the CSR entry names the kept copy with the right-side
     * bit), so mass and energy leave one cell exactly as they enter the other.
     * Both copies are still solved; the dropped copy's flux reaches no cell
     * and only the per-face export reads it.  The copy kept is chosen by
     * geometry, not by face number: the one whose image shift has the smaller
     * code.  Any numbering of the same faces -- a part of the mesh
     * (shadowfax_b200/partition.py) renumbers them -- then applies the same
     * copy with the same rounding. */
    std::vector<uint8_t> skip;
    std::vector<int32_t> idx_split;
    std::vector<std::pair<int64_t, int32_t>> merged;
    if(ctx->cfg.precision == SFX_PREC_SPLIT) {
        skip.assign(F, 0);
        idx_split = idx;
        auto shcode = [&](int64_t f) {
            int code = 0;
            for(int l = 0; l < dim; ++l) {
                double s = desc->face_right_pos[f * dim + l] -
                           desc->cell_pos[(int64_t)desc->face_right[f] * dim + l];
                int c = s > 0.5 ? 1 : (s < -0.5 ? 2 : 0);
                code = code * 3 + c;
            }
            return code;
        };
        auto negcode = [&](int code) {
            int out = 0, mul = 1;
            for(int l = 0; l < dim; ++l) {
                int c = code % 3;
                code /= 3;
                out += (c == 1 ? 2 : (c == 2 ? 1 : 0)) * mul;
                mul *= 3;
            }
            return out;
        };
        auto key = [](int64_t L, int64_t R, int code) {
            return ((uint64_t)L * 0x9E3779B97F4A7C15ull) ^ ((uint64_t)R << 20) ^ (uint64_t)code;
        };
        std::unordered_multimap<uint64_t, int64_t> per;
        for(int64_t f = 0; f < F; ++f)
            if(desc->face_kind[f] == SFX_FACE_PERIODIC)
                per.emplace(key(desc->face_left[f], desc->face_right[f], shcode(f)), f);
        std::vector<int32_t> twin(F, -1);
        for(int64_t g = 0; g < F; ++g) {
            if(desc->face_kind[g] != SFX_FACE_PERIODIC) continue;
            const int64_t L = desc->face_left[g], R = desc->face_right[g];
            const int want = negcode(shcode(g));
            auto rng = per.equal_range(key(R, L, want));
            for(auto it = rng.first; it != rng.second; ++it) {
                const int64_t f = it->second;
                if(desc->face_left[f] == R && desc->face_right[f] == L && shcode(f) == want &&
                   f < g && twin[f] < 0) {
                    twin[f] = (int32_t)g;
                    twin[g] = (int32_t)f;
                    if(want > shcode(g)) /* f has the larger code */
                        skip[f] = 1;
                    else
                        skip[g] = 1;
                    break;
                }
            }
        }
        for(int64_t i = 0; i < n; ++i)
            for(int64_t j = off[i]; j < off[i + 1]; ++j) {
                const int32_t g = desc->cell_face_index[j];
                if(skip[g]) {
                    idx_split[j] = (int32_t)((uint32_t)twin[g] | 0x80000000u);
                    merged.emplace_back(j, idx[j]);
                }
            }
    }
    SFX_TRY(cuda_ok(cudaSetDevice(ctx->cfg.device)));
    if(ctx->closing) return SFX_ERR_INVALID;
    sfx_mesh* m = new(std::nothrow) sfx_mesh;
    if(!m) return SFX_ERR_NOMEM;
    m->ctx = ctx;
    ctx->live_meshes++;
    if(!merged.empty())
        m->merged = std::make_shared<const std::vector<std::pair<int64_t, int32_t>>>(
                std::move(merged));
    sfx_dmesh& d = m->d;
    std::memset(&d, 0, sizeof d);
    d.dim = dim;
    d.S = dim + 2;
    d.n_cells = (int32_t)n;
    d.n_faces = (int32_t)F;
    d.nnz = nnz;
    d.has_velocity = desc->face_velocity != nullptr;
    d.lanes = sfx_default_lanes(dim);
    /* the plain-FP64 gradients compute a face's terms once for both of its
     * cells when the right cell of every local face sits at the face's right
     * position, bit for bit */
    d.gshare = 1;
    for(int64_t f = 0; f < F && d.gshare; ++f)
        if(desc->face_kind[f] == SFX_FACE_REAL &&
           std::memcmp(desc->face_right_pos + f * dim,
                       desc->cell_pos + (int64_t)desc->face_right[f] * dim,
                       sizeof(double) * dim) != 0)
            d.gshare = 0;
    const int S = d.S;
    const bool split = ctx->cfg.precision == SFX_PREC_SPLIT;
    if(split && d.has_velocity) {
        sfx_mesh_free(m);
        return SFX_ERR_UNSUPPORTED; /* the split pass is for static meshes */
    }
    int rc = allocate_fp64(m, !split, [&](Carver& arrays, bool records) {
        auto A = [&](auto** p, size_t c) { arrays.add(p, c); };
        A(&d.pos, n * dim);
        A(&d.cen, n * dim);
        A(&d.vol, n);
        A(&d.tarea, n);
        A(&d.off, n + 1);
        A(&d.idx, nnz);
        if(!aidx.empty()) A(&d.aidx, nnz);
        A(&d.W, n * S);
        A(&d.Q, n * S);
        add_stage(arrays, d, split, dq_doubles(d, split, records));
        A(&d.area, F);
        A(&d.mid, F * dim);
        A(&d.left, F);
        A(&d.right, F);
        A(&d.kind, F);
        A(&d.rpos, F * dim);
        if(d.has_velocity) A(&d.vel, F * dim);
        if(keeps_moving(dim, n, F)) {
            A(&m->kept_vgen, n * dim);
            A(&m->kept_newpos, n * dim);
            if(!d.has_velocity) A(&m->kept_vel, F * dim);
        }
        A(&d.branch, F);
        A(&d.err, 1);
        A(&d.totals_scratch, (size_t)(S + 1) * 1024);
        if(split || records) A(&d.ent, nnz);
        if(!split) {
            add_fp64_state(arrays, d, records);
            if(records) {
                A(&d.ggeo, F * rec_doubles(dim, SFX_REC_GGEO));
                A(&d.fgeo, F * rec_doubles(dim, SFX_REC_FGEO));
            }
            return;
        }
        A(&d.dQf, F * S);
        A(&d.fg, 2 * F);
        A(&d.fr, 12 * F);
        A(&d.cw, 2 * n);
        A(&d.cg, (size_t)sfx_split_grad_vec4(dim) * n);
        A(&d.cdw, (size_t)sfx_split_dwdt_vec4(dim) * n);
        A(&d.cx, n);
        A(&d.an, (size_t)dim * F);
        A(&d.dq, split_dq_doubles(dim) * F);
        d.slowq_cap = slowq_capacity(F);
        A(&d.slowq, (size_t)d.slowq_cap);
        A(&d.slowq_n, 1);
        A(&m->self_tab, 1);
        A(&m->self_pre, kSelfPre);
    });
    if(rc != SFX_OK) {
        sfx_mesh_free(m);
        return rc;
    }
    set_stage(d, split, dq_doubles(d, split, d.ws != nullptr));
    cudaStream_t s = ctx->stream;
    /* the dQ scratch holds dim doubles per face, the state staging per cell */
    double* fstage = split ? d.dq : d.dQf;
    rc = rows_in(d.pos, desc->cell_pos, n, dim, d.stage, s);
    if(!rc) rc = rows_in(d.cen, desc->cell_centroid, n, dim, d.stage, s);
    if(!rc) rc = rows_in(d.mid, desc->face_midpoint, F, dim, fstage, s);
    if(!rc) rc = rows_in(d.rpos, desc->face_right_pos, F, dim, fstage, s);
    if(!rc && d.has_velocity) rc = rows_in(d.vel, desc->face_velocity, F, dim, fstage, s);
    if(!rc) rc = h2d(d.vol, desc->cell_volume, n, s);
    if(!rc) rc = h2d(d.tarea, desc->cell_total_area, n, s);
    if(!rc) rc = h2d(d.off, off, n + 1, s);
    if(!rc) rc = h2d(d.idx, split ? idx_split.data() : idx.data(), nnz, s);
    if(!rc && !aidx.empty()) rc = h2d(d.aidx, aidx.data(), nnz, s);
    if(aidx.empty()) d.aidx = d.idx;
    if(!rc) rc = h2d(d.area, desc->face_area, F, s);
    if(!rc) rc = h2d(d.left, desc->face_left, F, s);
    if(!rc) rc = h2d(d.right, desc->face_right, F, s);
    if(!rc) rc = h2d(d.kind, desc->face_kind, F, s);
    if(!rc) rc = cuda_ok(cudaMemsetAsync(d.W, 0, sizeof(double) * n * S, s));
    if(!rc) rc = cuda_ok(cudaMemsetAsync(d.Q, 0, sizeof(double) * n * S, s));
    if(!rc) rc = reset_err(m);
    if(!rc && split) rc = cuda_ok(cudaMemsetAsync(d.slowq_n, 0, sizeof(int32_t), s));
    if(!rc && d.ent) rc = sfx_fp64_csr_neighbours(&d, s);
    if(!rc && split) rc = sfx_split_prepare(&d, s);
    if(!rc && split) rc = setup_self(m, s);
    if(!rc && d.ws) rc = sfx_fp64_face_records(&d, s);
    if(!rc && d.ws)
        rc = cuda_ok(cudaMemsetAsync(d.ws, 0, sizeof(double) * n * rec_doubles(dim, SFX_REC_WS), s));
    /* host staging buffers go out of scope: wait for the copies */
    if(!rc) rc = cuda_ok(cudaStreamSynchronize(s));
    if(rc != SFX_OK) {
        sfx_mesh_free(m);
        return rc;
    }
    *out = m;
    return SFX_OK;
}

int sfx_mesh_free(sfx_mesh* m) {
    if(!m) return SFX_ERR_INVALID;
    sfx_ctx* ctx = m->ctx;
    if(ctx) {
        cudaSetDevice(ctx->cfg.device);
        /* cudaFree waits for the device; a caller stream may already be gone */
        cudaStreamSynchronize(ctx->own_stream);
    }
    for(void* p : m->allocs) cudaFree(p);
    delete m;
    if(ctx && --ctx->live_meshes == 0 && ctx->closing) ctx_release(ctx);
    return SFX_OK;
}

int sfx_state_upload_W(sfx_mesh* m, const double* W) {
    if(!m || !W) return SFX_ERR_INVALID;
    SFX_TRY(sfx_mesh_upload_W_async(m, W, m->ctx->stream));
    return check_err(m, nullptr);
}

int sfx_state_upload_WQ(sfx_mesh* m, const double* W, const double* Q) {
    if(!m || !W || !Q) return SFX_ERR_INVALID;
    const int64_t n = m->d.n_cells;
    cudaStream_t s = m->ctx->stream;
    const sfx_dmesh& d = m->d;
    SFX_TRY(reset_err(m));
    const size_t ns = (size_t)n * d.S;
    SFX_TRY(h2d(d.stage, W, ns, s));
    SFX_TRY(h2d(d.stage2, Q, ns, s));
    if(m->ctx->cfg.precision == SFX_PREC_SPLIT)
        SFX_TRY(sfx_split_load_state(&d, d.stage, d.stage2, s));
    else
        SFX_TRY(sfx_fp64_load_rows(&d, d.stage, d.stage2, s));
    return cuda_ok(cudaStreamSynchronize(s));
}

/* States of at most this many doubles are transposed on the host: 1,200 doubles of
 * W and of Q take 24 us so (plain FP64, both in one copy) and 45 with two copies
 * and the transposing launches; 8,000 take 41 (12,000 with the launches 60). */
constexpr size_t kSmallState = 8192;

static int download_small(sfx_mesh* m, double* W, double* Q) {
    const sfx_dmesh& d = m->d;
    const size_t n = (size_t)d.n_cells, ns = n * d.S;
    cudaStream_t s = m->ctx->stream;
    double t[2 * kSmallState + 64];
    const bool split = m->ctx->cfg.precision == SFX_PREC_SPLIT;
    /* plain FP64: W and Q, neighbours in the mesh's block, in one copy */
    const double* from = split ? d.Q : d.W;
    const size_t at = (size_t)(d.Q - from);
    if(split) {
        SFX_TRY(sfx_split_W_rows(&d, d.stage, s));
        SFX_TRY(cuda_ok(cudaMemcpyAsync(W, d.stage, sizeof(double) * ns, cudaMemcpyDeviceToHost, s)));
    }
    SFX_TRY(cuda_ok(cudaMemcpyAsync(t, from, sizeof(double) * (at + ns), cudaMemcpyDeviceToHost, s)));
    SFX_TRY(cuda_ok(cudaStreamSynchronize(s)));
    for(size_t i = 0; i < n; ++i)
        for(int k = 0; k < d.S; ++k) {
            if(!split) W[i * d.S + k] = t[k * n + i];
            Q[i * d.S + k] = t[at + k * n + i];
        }
    return SFX_OK;
}

int sfx_state_download(sfx_mesh* m, double* W, double* Q) {
    if(!m) return SFX_ERR_INVALID;
    cudaStream_t s = m->ctx->stream;
    if(W && Q && (size_t)m->d.n_cells * m->d.S <= kSmallState) return download_small(m, W, Q);
    SFX_TRY(sfx_mesh_download_async(m, W, Q, s));
    return cuda_ok(cudaStreamSynchronize(s));
}

int sfx_step(sfx_mesh* m, double dt, int32_t nsteps, sfx_stats* st) {
    if(!m || nsteps < 0 || !(dt > 0.)) return SFX_ERR_INVALID;
    sfx_ctx* c = m->ctx;
    cudaStream_t s = c->stream;
    SFX_TRY(reset_err(m));
    for(int t = 0; t < nsteps; ++t)
        for(int ph = 0; ph < 3; ++ph) SFX_TRY(run_phase(m, ph, dt, 0, s));
    if(!st) return SFX_OK;
    return collect_stats(m, nsteps, st);
}

int sfx_step_moving(sfx_mesh* m, double dt, int32_t periodic, double* positions,
                    sfx_stats* st) {
    if(!m || !(dt > 0.)) return SFX_ERR_INVALID;
    sfx_ctx* c = m->ctx;
    if(m->clone || m->d.ranged) return SFX_ERR_UNSUPPORTED;
    const bool split = c->cfg.precision == SFX_PREC_SPLIT;
    cudaStream_t s = c->stream;
    sfx_dmesh& d = m->d;
    const int64_t n = d.n_cells, F = d.n_faces;
    const int D = d.dim;
    const bool fresh = d.vel == nullptr;
    if(!d.vgen) d.vgen = m->kept_vgen;
    if(!d.newpos) d.newpos = m->kept_newpos;
    if(!d.vel) d.vel = m->kept_vel;
    Carver first; /* one allocation: a moving mesh takes one step per tessellation */
    if(!d.vgen) first.add(&d.vgen, (size_t)D * n);
    if(!d.newpos) first.add(&d.newpos, (size_t)D * n);
    if(!d.vel) first.add(&d.vel, (size_t)D * F);
    if(!first.slots.empty()) SFX_TRY(first.allocate(m));
    d.has_velocity = 1;
    SFX_TRY(reset_err(m));
    /* the split pass keeps the state in FP32 cell records: the FP64 W the
     * velocity kernels read is exported from them first; the device copy of
     * the mesh (the one-member group table) learns the face velocities */
    if(split) SFX_TRY(sfx_split_export_W(&d, s));
    if(split && fresh) SFX_TRY(setup_self(m, s));
    SFX_TRY(sfx_fp64_move_velocities(&d, c->cfg.gamma, dt, periodic ? 1 : 0, 1, s));
    for(int ph = 0; ph < 3; ++ph) SFX_TRY(run_phase(m, ph, dt, 0, s));
    SFX_TRY(sfx_fp64_drift(&d, dt, s));
    if(positions) {
        SFX_TRY(sfx_to_rows(d.newpos, n, D, d.stage, s));
        SFX_TRY(cuda_ok(cudaMemcpyAsync(positions, d.stage, sizeof(double) * D * n,
                                        cudaMemcpyDeviceToHost, s)));
    }
    sfx_stats local;
    return collect_stats(m, 1, st ? st : &local);
}

/* local time steps: per-cell integer step bounds and generator velocities
 * (all zero at first) */
static int ensure_local(sfx_mesh* m) {
    sfx_dmesh& d = m->d;
    cudaStream_t s = m->ctx->stream;
    const size_t n = (size_t)d.n_cells;
    if(!d.tstart) {
        SFX_TRY(dalloc(m, &d.tstart, n));
        SFX_TRY(dalloc(m, &d.tend, n));
        SFX_TRY(cuda_ok(cudaMemsetAsync(d.tstart, 0, sizeof(uint64_t) * n, s)));
        SFX_TRY(cuda_ok(cudaMemsetAsync(d.tend, 0, sizeof(uint64_t) * n, s)));
    }
    if(!d.vgen) {
        double* vgen = m->kept_vgen;
        if(!vgen) SFX_TRY(dalloc(m, &vgen, (size_t)d.dim * n));
        d.vgen = vgen;
        SFX_TRY(cuda_ok(cudaMemsetAsync(d.vgen, 0, sizeof(double) * d.dim * n, s)));
    }
    if(!m->d_smin) SFX_TRY(dalloc(m, &m->d_smin, 1));
    return SFX_OK;
}

/* local time steps: plain FP64 meshes, and split meshes that are not
 * clones (a clone is a request instance of the server) */
static bool local_ok(const sfx_mesh* m) {
    if(m->d.ranged) return false;
    return m->ctx->cfg.precision == SFX_PREC_FP64 || !m->clone;
}

int sfx_mesh_set_timesteps(sfx_mesh* m, const uint64_t* start, const uint64_t* end) {
    if(!m || !start || !end) return SFX_ERR_INVALID;
    if(!local_ok(m)) return SFX_ERR_UNSUPPORTED;
    const int64_t n = m->d.n_cells;
    for(int64_t i = 0; i < n; ++i)
        if(end[i] < start[i] || end[i] > SFX_TIMELINE_TICKS) return SFX_ERR_INVALID;
    SFX_TRY(ensure_local(m));
    cudaStream_t s = m->ctx->stream;
    SFX_TRY(h2d(m->d.tstart, start, (size_t)n, s));
    SFX_TRY(h2d(m->d.tend, end, (size_t)n, s));
    return cuda_ok(cudaStreamSynchronize(s));
}

int sfx_mesh_get_timesteps(sfx_mesh* m, uint64_t* start, uint64_t* end) {
    if(!m || !start || !end) return SFX_ERR_INVALID;
    if(!local_ok(m)) return SFX_ERR_UNSUPPORTED;
    SFX_TRY(ensure_local(m));
    cudaStream_t s = m->ctx->stream;
    const size_t n = (size_t)m->d.n_cells;
    SFX_TRY(cuda_ok(cudaMemcpyAsync(start, m->d.tstart, sizeof(uint64_t) * n,
                                    cudaMemcpyDeviceToHost, s)));
    SFX_TRY(cuda_ok(cudaMemcpyAsync(end, m->d.tend, sizeof(uint64_t) * n,
                                    cudaMemcpyDeviceToHost, s)));
    return cuda_ok(cudaStreamSynchronize(s));
}

/* host gradients [n][dim*S] from or to the mesh's records (gradients [l][k] first) or
 * field-major arrays, through the staging rows, as many cells at a time as fit (a copy of
 * the records with the host picking the gradients out took 920 us to set and 680
 * to get for 30,000 cells in 2D; these take 128 and 178) */
static int move_gradients(sfx_mesh* m, double* out, const double* in) {
    const sfx_dmesh& d = m->d;
    if(m->ctx->cfg.precision != SFX_PREC_FP64) return SFX_ERR_UNSUPPORTED;
    cudaStream_t s = m->ctx->stream;
    const int w = d.dim * d.S;
    const int64_t n = d.n_cells;
    /* on their way in through the dQ scratch when that holds them all */
    const size_t dq = dq_doubles(d, false, d.ws != nullptr);
    const bool whole = in && dq >= (size_t)(n * w);
    double* rows = whole ? d.dQf : d.stage;
    const int64_t part = whole ? n : (int64_t)(stage_doubles(n, d.dim, false, dq) / w);
    const int64_t rs = d.grec ? (int64_t)rec_doubles(d.dim, SFX_REC_GREC) : 1;
    const int64_t cs = d.grec ? 1 : n;
    double* g = d.grec ? d.grec : d.grad;
    for(int64_t i = 0; i < n; i += part) {
        const int64_t count = std::min(part, n - i);
        const size_t bytes = sizeof(double) * (size_t)(count * w);
        if(in) SFX_TRY(h2d(rows, in + i * w, (size_t)(count * w), s));
        SFX_TRY(sfx_strided_rows(g + i * rs, rs, cs, count, w, rows, in != nullptr, s));
        if(out)
            SFX_TRY(cuda_ok(cudaMemcpyAsync(out + i * w, rows, bytes, cudaMemcpyDeviceToHost, s)));
    }
    return cuda_ok(cudaStreamSynchronize(s));
}

int sfx_mesh_set_gradients(sfx_mesh* m, const double* grad) {
    if(!m || !grad) return SFX_ERR_INVALID;
    return move_gradients(m, nullptr, grad); /* the records' dW/dt stays */
}

int sfx_mesh_get_gradients(sfx_mesh* m, double* grad) {
    if(!m || !grad) return SFX_ERR_INVALID;
    return move_gradients(m, grad, nullptr);
}

int sfx_step_window(sfx_mesh* m, double t_total, uint64_t t_now, uint64_t t_next,
                    int32_t periodic, sfx_stats* st) {
    if(!m || !(t_total > 0.) || t_next <= t_now || t_next > SFX_TIMELINE_TICKS)
        return SFX_ERR_INVALID;
    if(!local_ok(m)) return SFX_ERR_UNSUPPORTED;
    SFX_TRY(ensure_local(m));
    sfx_ctx* c = m->ctx;
    cudaStream_t s = c->stream;
    sfx_dmesh& d = m->d;
    const bool split = c->cfg.precision == SFX_PREC_SPLIT;
    d.local = 1;
    d.t_now = t_now;
    d.t_next = t_next;
    d.t_total = t_total;
    int rc = reset_err(m);
    /* the cells starting a step set their generator velocity (the mesh
     * stays); a split mesh's FP32 states are exported to its FP64 W first */
    if(!rc && split) rc = sfx_split_export_W(&d, s);
    if(!rc) rc = sfx_fp64_move_velocities(&d, c->cfg.gamma, 0., periodic ? 1 : 0, 0, s);
    /* a split mesh's kernels read the window from its device table */
    if(!rc && split) rc = setup_self(m, s);
    for(int ph = 0; ph < 3 && !rc; ++ph) rc = run_phase(m, ph, 1., 0, s);
    d.local = 0;
    if(split) {
        const int r2 = setup_self(m, s);
        if(!rc) rc = r2;
    }
    if(rc) return rc;
    sfx_stats local;
    return collect_stats(m, 1, st ? st : &local);
}

int sfx_timestep_bins(sfx_mesh* m, double t_total, double cfl, uint64_t max_step,
                      uint64_t min_step, uint64_t t_next, uint64_t* system_step) {
    if(!m || !(t_total > 0.) || !(cfl > 0.) || max_step == 0 || max_step > SFX_TIMELINE_TICKS ||
       min_step > max_step || !system_step)
        return SFX_ERR_INVALID;
    if(!local_ok(m)) return SFX_ERR_UNSUPPORTED;
    SFX_TRY(ensure_local(m));
    sfx_ctx* c = m->ctx;
    cudaStream_t s = c->stream;
    sfx_dmesh& d = m->d;
    d.t_next = t_next;
    d.t_total = t_total;
    SFX_TRY(reset_err(m));
    const unsigned long long smax = max_step;
    SFX_TRY(h2d(m->d_smin, &smax, 1, s));
    /* a split mesh: the CFL steps from its FP32 states, exported to FP64 */
    if(c->cfg.precision == SFX_PREC_SPLIT) SFX_TRY(sfx_split_export_W(&d, s));
    SFX_TRY(sfx_fp64_timestep_bins(&d, c->cfg.gamma, cfl, max_step, min_step, m->d_smin, s));
    unsigned long long out = 0;
    SFX_TRY(cuda_ok(cudaMemcpyAsync(&out, m->d_smin, sizeof out, cudaMemcpyDeviceToHost, s)));
    SFX_TRY(cuda_ok(cudaStreamSynchronize(s)));
    SFX_TRY(check_err(m, nullptr));
    *system_step = out;
    return SFX_OK;
}

int sfx_step_timed(sfx_mesh* m, double dt, int32_t nsteps, float* kernel_ms,
                   int32_t* launches) {
    if(!m || nsteps < 0 || !(dt > 0.) || !kernel_ms) return SFX_ERR_INVALID;
    sfx_ctx* c = m->ctx;
    cudaStream_t s = c->stream;
    cudaEvent_t ev[4];
    for(auto& e : ev)
        if(cudaEventCreate(&e) != cudaSuccess) return SFX_ERR_CUDA;
    double acc[3] = {0., 0., 0.};
    int rc = reset_err(m);
    const int64_t l0 = sfx_launch_count();
    for(int t = 0; t < nsteps && rc == SFX_OK; ++t) {
        cudaEventRecord(ev[0], s);
        rc = run_phase(m, 0, dt, 0, s);
        cudaEventRecord(ev[1], s);
        if(!rc) rc = run_phase(m, 1, dt, 0, s);
        cudaEventRecord(ev[2], s);
        if(!rc) rc = run_phase(m, 2, dt, 0, s);
        cudaEventRecord(ev[3], s);
        if(!rc) rc = cuda_ok(cudaEventSynchronize(ev[3]));
        for(int k = 0; k < 3 && !rc; ++k) {
            float ms = 0.f;
            rc = cuda_ok(cudaEventElapsedTime(&ms, ev[k], ev[k + 1]));
            acc[k] += ms;
        }
    }
    for(auto& e : ev) cudaEventDestroy(e);
    for(int k = 0; k < 3; ++k) kernel_ms[k] = (float)acc[k];
    if(launches) *launches = (int32_t)(sfx_launch_count() - l0);
    if(rc) return rc;
    return check_err(m, nullptr);
}

int sfx_flux_pass(sfx_mesh* m, double dt, double* grad, double* dQ_face,
                  int32_t* branch, sfx_stats* st) {
    if(!m || !(dt > 0.)) return SFX_ERR_INVALID;
    sfx_ctx* c = m->ctx;
    cudaStream_t s = c->stream;
    const int64_t n = m->d.n_cells, F = m->d.n_faces;
    const int S = m->d.S, D = m->d.dim;
    const bool split = c->cfg.precision == SFX_PREC_SPLIT;
    if(!m->d.dQf) return SFX_ERR_UNSUPPORTED; /* a split clone keeps no FP64 dQ */
    SFX_TRY(reset_err(m));
    SFX_TRY(run_phase(m, 0, dt, 1, s));
    SFX_TRY(run_phase(m, 1, dt, 1, s));
    if(split) SFX_TRY(sfx_split_export_dQ(&m->d, s));
    if(grad && split) {
        /* FP32 gradient records [n][G float4] */
        const int G = sfx_split_grad_vec4(D);
        std::vector<float> tf((size_t)n * G * 4);
        SFX_TRY(cuda_ok(cudaMemcpyAsync(tf.data(), m->d.cg, sizeof(float) * tf.size(),
                                        cudaMemcpyDeviceToHost, s)));
        SFX_TRY(cuda_ok(cudaStreamSynchronize(s)));
        for(int64_t i = 0; i < n; ++i)
            for(int q = 0; q < D * S; ++q) grad[i * D * S + q] = tf[(size_t)i * G * 4 + q];
    }
    if(branch && split && F) SFX_TRY(cuda_ok(cudaMemsetAsync(m->d.branch, 0, 4 * F, s)));
    /* dQ: rows as they are (split, and the 2D records), or formed through the staging
     * rows from the 3D records or field-major arrays */
    if(dQ_face && (split || (m->d.ws && D == 2))) {
        SFX_TRY(cuda_ok(cudaMemcpyAsync(dQ_face, m->d.dQf, sizeof(double) * (size_t)F * S,
                                        cudaMemcpyDeviceToHost, s)));
    } else if(dQ_face) {
        const int64_t rs = m->d.ws ? (int64_t)rec_doubles(D, SFX_REC_DQ) : 1;
        const int64_t cs = m->d.ws ? 1 : F;
        const size_t dq = dq_doubles(m->d, split, m->d.ws != nullptr);
        const int64_t part = (int64_t)stage_doubles(n, D, split, dq) / S;
        for(int64_t f = 0; f < F; f += part) {
            const int64_t count = std::min(part, F - f);
            SFX_TRY(sfx_strided_rows(m->d.dQf + f * rs, rs, cs, count, S, m->d.stage, 0, s));
            SFX_TRY(cuda_ok(cudaMemcpyAsync(dQ_face + f * S, m->d.stage,
                                            sizeof(double) * (size_t)(count * S),
                                            cudaMemcpyDeviceToHost, s)));
        }
    }
    if(branch && F)
        SFX_TRY(cuda_ok(cudaMemcpyAsync(branch, m->d.branch, sizeof(int32_t) * F,
                                        cudaMemcpyDeviceToHost, s)));
    SFX_TRY(cuda_ok(cudaStreamSynchronize(s)));
    if(grad && !split) SFX_TRY(sfx_mesh_get_gradients(m, grad));
    sfx_stats local;
    return check_err(m, st ? st : &local);
}

int sfx_riemann_eval(sfx_ctx* c, int32_t n, const double* WL, const double* WR,
                     const double* normal, int32_t reflective, double* half,
                     double* flux, int32_t* branch) {
    if(!c || n < 0 || (n && (!WL || !WR || !normal || !flux || !branch)))
        return SFX_ERR_INVALID;
    if(n == 0) return SFX_OK;
    const int D = c->cfg.dim, S = D + 2;
    cudaStream_t s = c->stream;
    double *dWL = nullptr, *dWR = nullptr, *dn = nullptr, *dh = nullptr, *df = nullptr;
    int32_t* dc = nullptr;
    int rc = SFX_OK;
    auto al = [&](auto** p, size_t bytes) {
        if(rc == SFX_OK && cudaMalloc((void**)p, bytes) != cudaSuccess) rc = SFX_ERR_CUDA;
    };
    al(&dWL, sizeof(double) * n * S);
    al(&dWR, sizeof(double) * n * S);
    al(&dn, sizeof(double) * n * D);
    al(&dh, sizeof(double) * n * S);
    al(&df, sizeof(double) * n * S);
    al(&dc, sizeof(int32_t) * n);
    if(!rc) rc = h2d(dWL, WL, (size_t)n * S, s);
    if(!rc) rc = h2d(dWR, WR, (size_t)n * S, s);
    if(!rc) rc = h2d(dn, normal, (size_t)n * D, s);
    if(!rc) rc = sfx_fp64_riemann(D, &c->sp, n, dWL, dWR, dn, reflective, dh, df, dc, s);
    if(!rc && half)
        rc = cuda_ok(cudaMemcpyAsync(half, dh, sizeof(double) * n * S, cudaMemcpyDeviceToHost, s));
    if(!rc)
        rc = cuda_ok(cudaMemcpyAsync(flux, df, sizeof(double) * n * S, cudaMemcpyDeviceToHost, s));
    if(!rc)
        rc = cuda_ok(cudaMemcpyAsync(branch, dc, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, s));
    if(!rc) rc = cuda_ok(cudaStreamSynchronize(s));
    cudaFree(dWL);
    cudaFree(dWR);
    cudaFree(dn);
    cudaFree(dh);
    cudaFree(df);
    cudaFree(dc);
    return rc;
}

int sfx_mesh_clone(sfx_ctx* ctx, sfx_mesh* base, sfx_mesh** out) {
    return clone_impl(ctx, base, ctx ? ctx->stream : nullptr, true, out);
}

int64_t sfx_mesh_clone_bytes(sfx_mesh* base, int32_t precision) {
    if(!base) return -1;
    const sfx_dmesh& b = base->d;
    const int64_t n = b.n_cells, F = b.n_faces, S = b.S, D = b.dim;
    const bool split = precision == SFX_PREC_SPLIT;
    const size_t dq = (size_t)F * (split ? split_dq_doubles((int)D) : rec_doubles((int)D, SFX_REC_DQ));
    int64_t bytes = n * S * 16 + 8 * (int64_t)stage_doubles(n, (int)D, split, dq) +
                    (S + 1) * 1024 * 8 + 64;
    if(precision == SFX_PREC_SPLIT)
        bytes += n * 32 + n * 16 * (sfx_split_grad_vec4((int)D) + sfx_split_dwdt_vec4((int)D)) +
                 F * 8 * split_dq_doubles((int)D) +
                 4 * (int64_t)slowq_capacity(F) + 4 + (int64_t)sizeof(sfx_group_entry) + 28;
    else {
        auto rec = [&](int what) { return (int64_t)sfx_fp64_record_bytes((int)D, what); };
        bytes += n * (rec(SFX_REC_WS) + rec(SFX_REC_GREC)) + F * (4 + rec(SFX_REC_DQ)) +
                 4 * sfx_fp64_list_room(F) + 512;
        if(b.fg && !b.ggeo) /* of a split mesh: face records and CSR of its own */
            bytes += F * (rec(SFX_REC_GGEO) + rec(SFX_REC_FGEO)) + (int64_t)b.nnz * 16 + 1280;
    }
    return bytes;
}

int sfx_mesh_set_lanes(sfx_mesh* m, int32_t lanes) {
    if(!m || (lanes != 1 && lanes != 2 && lanes != 4 && lanes != 8 && lanes != 16))
        return SFX_ERR_INVALID;
    m->d.lanes = lanes;
    return SFX_OK;
}

int sfx_mesh_set_face_variant(sfx_mesh* m, int32_t variant) {
    if(!m || variant < 0 || variant >= SFX_FACE_VARIANTS) return SFX_ERR_INVALID;
    m->d.face_variant = variant;
    return SFX_OK;
}

int sfx_mesh_set_ranges(sfx_mesh* m, int32_t grad_cells, int32_t flux_faces,
                        int32_t update_cells) {
    if(!m) return SFX_ERR_INVALID;
    const bool split = m->ctx->cfg.precision == SFX_PREC_SPLIT;
    if(split && m->clone) return SFX_ERR_UNSUPPORTED;
    sfx_dmesh& d = m->d;
    if(update_cells < 0 || update_cells > grad_cells || grad_cells > d.n_cells ||
       flux_faces < 0 || flux_faces > d.n_faces)
        return SFX_ERR_INVALID;
    d.ranged = 1;
    d.r_grad = grad_cells;
    d.r_flux = flux_faces;
    d.r_upd = update_cells;
    /* a split mesh's kernels read the ranges from its device table */
    if(split) return setup_self(m, m->ctx->stream);
    return SFX_OK;
}

int sfx_mesh_pack_cells(sfx_mesh* m, const int32_t* idx, int32_t count, double* out,
                        void* stream) {
    if(!m || count < 0 || (count > 0 && (!idx || !out))) return SFX_ERR_INVALID;
    if(m->ctx->cfg.precision == SFX_PREC_SPLIT)
        return sfx_split_pack_cells(&m->d, idx, count, out,
                                    stream ? stream : (void*)m->ctx->stream);
    return sfx_fp64_pack_cells(&m->d, idx, count, out,
                               stream ? stream : (void*)m->ctx->stream);
}

int sfx_mesh_unpack_cells(sfx_mesh* m, const int32_t* idx, int32_t count, const double* in,
                          void* stream) {
    if(!m || count < 0 || (count > 0 && (!idx || !in))) return SFX_ERR_INVALID;
    if(m->ctx->cfg.precision == SFX_PREC_SPLIT)
        return sfx_split_unpack_cells(&m->d, idx, count, in,
                                      stream ? stream : (void*)m->ctx->stream);
    return sfx_fp64_unpack_cells(&m->d, idx, count, in,
                                 stream ? stream : (void*)m->ctx->stream);
}

int sfx_mesh_totals(sfx_mesh* m, double* totals) {
    if(!m || !totals) return SFX_ERR_INVALID;
    double t[7];
    SFX_TRY(sfx_fp64_totals(&m->d, t, m->ctx->stream));
    std::memcpy(totals, t, sizeof(double) * m->d.S);
    return SFX_OK;
}

}  // extern "C"

/* internal transfers (C++ linkage) */
int sfx_mesh_upload_W_async(sfx_mesh* m, const double* W, void* stream) {
    if(!m || !W) return SFX_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    SFX_TRY(reset_err_on(m, s));
    SFX_TRY(h2d(m->d.stage, W, (size_t)m->d.n_cells * m->d.S, s));
    SFX_TRY(sfx_fp64_init_Q(&m->d, &m->ctx->sp, m->d.stage, s));
    if(m->ctx->cfg.precision == SFX_PREC_SPLIT) SFX_TRY(sfx_split_load_state(&m->d, nullptr, nullptr, s));
    return SFX_OK;
}

int sfx_mesh_download_async(sfx_mesh* m, double* W, double* Q, void* stream) {
    if(!m) return SFX_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    const sfx_dmesh& d = m->d;
    const size_t bytes = sizeof(double) * (size_t)d.n_cells * d.S;
    /* one after the other through the staging rows: the stream orders them */
    if(W) {
        if(m->ctx->cfg.precision == SFX_PREC_SPLIT)
            SFX_TRY(sfx_split_W_rows(&d, d.stage, s));
        else
            SFX_TRY(sfx_to_rows(d.W, d.n_cells, d.S, d.stage, s));
        SFX_TRY(cuda_ok(cudaMemcpyAsync(W, d.stage, bytes, cudaMemcpyDeviceToHost, s)));
    }
    if(Q) {
        SFX_TRY(sfx_to_rows(d.Q, d.n_cells, d.S, d.stage, s));
        SFX_TRY(cuda_ok(cudaMemcpyAsync(Q, d.stage, bytes, cudaMemcpyDeviceToHost, s)));
    }
    return SFX_OK;
}

int sfx_mesh_clone_async(sfx_ctx* ctx, sfx_mesh* base, void* stream, sfx_mesh** out) {
    return clone_impl(ctx, base, (cudaStream_t)stream, false, out);
}
