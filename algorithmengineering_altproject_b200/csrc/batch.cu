// Batched designs: many designs of uneven grid size advance together, one launch per kernel of the inner
// PCG iteration for all of them.
//
// Layout.  The members' buffers are carved from one device arena (sized by a first, counting creation of each
// member).  Each member keeps its own context -- grid, MG hierarchy, FP32/FP64 vectors, reduction slots and
// scalars -- so everything outside the inner solve runs per member on the member's own host thread and stream
// (SIMP, MG rebuild, the FP64 defect correction, compliance, sensitivities, filter, OC): see "the engine".
//
// Work list.  Every kernel of the FP32 MG-PCG iteration is one persistent launch over (instance, logical
// block) items (kernels.hpp, "batched launches"): the logical blocks of an instance are the blocks of the
// launch the member would make alone, so each member's arithmetic and reduction order are those of its own
// launch and its results are identical to a solo run with the same parameters.  Per-instance convergence
// masks: a member whose inner solve has converged or spent its budget (S->done, set on the device) skips its
// items for the rest of that iteration, and a compaction kernel at the end of every iteration drops it from
// the work lists, so finished members cost nothing while the others go on.  BATCH_CHUNK iterations are
// captured once in a CUDA graph and replayed; the host polls the members' done flags (gathered into one
// array) after each replay.
//
// The FP64 defect-correction loop around each inner solve is the single-design one (mixed_solve in context.cu),
// run by the member's thread, so members do not wait for one another between inner solves.
#include <atomic>
#include <chrono>
#include <cmath>
#include <condition_variable>
#include <cstring>
#include <memory>
#include <mutex>
#include <thread>

#include "context.hpp"

namespace t3d {

namespace {

constexpr int BATCH_CHUNK = 16;      // inner PCG iterations per graph replay
constexpr int BATCH_MAX_OUTER = 64;  // defect-correction passes (as the single-design solve)

struct LaunchList {      // one batched launch: per-instance arguments and the active-instance list on the device
    void* args = nullptr;
    int* act = nullptr;   // n, positions, block prefix sums (kernels.hpp)
    int n = 0;            // instances in the list
    int64_t blocks = 0;   // logical blocks with every instance active
};

}  // namespace

struct Job {
    t3d_context* c = nullptr;
    int steps = 0;
    bool release = false;               // submitted: leaves the batch when finished
    std::vector<t3d_iter_record> recs;
    int rc = T3D_OK;
    std::string err;
    int phase = 0;                      // 0 own work, 1 inner solve requested, 2 in the batched solve, 3 solved
    PcgScalars init{};
    bool started = false, finished = false;
    std::thread th;
};

struct Batch {
    int dev = 0;
    std::vector<t3d_context*> m;
    Arena arena;
    cudaStream_t st = nullptr;
    int variant = T3D_BATCH_TILE - 1;
    int mv_grid = 0;
    ModalKe kh{};
    std::vector<void*> dallocs;
    bool standard = false;       // the members' V-cycle (all the same): Standard, else Adapted
    LaunchList mv, up, dir, p0, co, mv1, mv2;
    LaunchList rs0[8], rs1[8], pr[8], lsp[8], lnd[8], pa[8];   // level products: split levels, levels by nodes
    int maxL = 0, coarse_max = 0;
    CUtensorMap* maps = nullptr;
    std::vector<BatchCompact> compact;   // one compaction job per launch list
    BatchCompact* dcompact = nullptr;
    PcgScalars** dS = nullptr;
    int* dflags = nullptr;
    int* err = nullptr;
    int* hflags = nullptr;       // pinned
    PcgScalars* hS = nullptr;    // pinned
    double* hscal = nullptr;     // pinned
    cudaGraphExec_t graph = nullptr;
    int64_t launches = 0;
    int iter_kernels = 0;
    int64_t iter_blocks = 0;
    int n_arena = 0;             // members 0 .. n_arena-1 live in the arena (created with the batch)
    bool dirty = true;           // membership changed: the launch lists and the graph are rebuilt before use
    // the engine (batch.cu "the engine"): jobs, their handshake with the scheduler, submitted work
    std::mutex mu;
    std::condition_variable cv;
    std::vector<std::unique_ptr<Job>> jobs;   // running or finished, not yet collected
    std::vector<std::unique_ptr<Job>> incoming;   // submitted, not yet members
    std::thread sched;           // the scheduler thread of submitted work
    bool stop = false;
    bool failed = false;
    std::string fail_msg;

    template <class T>
    int dalloc(T** p, size_t n) {
        void* q = nullptr;
        cudaError_t e = cudaMalloc(&q, std::max<size_t>(n, 1) * sizeof(T));
        if (e != cudaSuccess) return set_cuda_error(e, "cudaMalloc", __FILE__, __LINE__);
        dallocs.push_back(q);
        *p = static_cast<T*>(q);
        return T3D_OK;
    }

    // the launch lists, the graph and the polling buffers (rebuilt when membership changes)
    void free_lists() {
        if (graph) cudaGraphExecDestroy(graph);
        graph = nullptr;
        for (void* q : dallocs) cudaFree(q);
        dallocs.clear();
        if (hflags) cudaFreeHost(hflags);
        if (hS) cudaFreeHost(hS);
        if (hscal) cudaFreeHost(hscal);
        hflags = nullptr;
        hS = nullptr;
        hscal = nullptr;
        maps = nullptr;
        compact.clear();
        dcompact = nullptr;
        dS = nullptr;
        dflags = nullptr;
        err = nullptr;
        mv = up = dir = p0 = co = mv1 = mv2 = LaunchList{};
        for (int l = 0; l < 8; ++l) rs0[l] = rs1[l] = pr[l] = lsp[l] = lnd[l] = pa[l] = LaunchList{};
    }

    ~Batch() {
        cudaSetDevice(dev);
        if (st) cudaStreamSynchronize(st);
        for (t3d_context* c : m) {
            if (!c) continue;
            cudaStreamSynchronize(c->st);
            delete c;
        }
        free_lists();
        if (arena.base) cudaFree(arena.base);
        if (st) cudaStreamDestroy(st);
    }
};

namespace {

// uploads one launch list: args[k] with blocks[k] logical blocks each and scalars S[k]; the active list starts
// with every instance and its compaction job is queued
template <class T>
int make_list(Batch* B, const std::vector<T>& a, const std::vector<int>& blocks, const std::vector<PcgScalars*>& S,
              LaunchList* L) {
    const int N = (int)a.size();
    L->n = N;
    L->blocks = 0;
    if (N == 0) return T3D_OK;
    std::vector<int> act(2 * (size_t)N + 2, 0);
    act[0] = N;
    for (int k = 0; k < N; ++k) {
        if (blocks[k] <= 0) return set_error(T3D_ERR_INVALID, "batched launch with an empty instance");
        act[1 + k] = k;
        act[2 + N + k] = act[1 + N + k] + blocks[k];
    }
    L->blocks = act[1 + 2 * N];
    T* da = nullptr;
    int* db = nullptr;
    PcgScalars** dS = nullptr;
    CHECK(B->dalloc(&da, a.size()));
    CHECK(B->dalloc(&L->act, act.size()));
    CHECK(B->dalloc(&db, blocks.size()));
    CHECK(B->dalloc(&dS, S.size()));
    T3D_CUDA_OK(cudaMemcpyAsync(da, a.data(), a.size() * sizeof(T), cudaMemcpyHostToDevice, B->st));
    T3D_CUDA_OK(cudaMemcpyAsync(L->act, act.data(), act.size() * sizeof(int), cudaMemcpyHostToDevice, B->st));
    T3D_CUDA_OK(cudaMemcpyAsync(db, blocks.data(), blocks.size() * sizeof(int), cudaMemcpyHostToDevice, B->st));
    T3D_CUDA_OK(cudaMemcpyAsync(dS, S.data(), S.size() * sizeof(PcgScalars*), cudaMemcpyHostToDevice, B->st));
    L->args = da;
    B->compact.push_back(BatchCompact{dS, db, N, L->act});
    return T3D_OK;
}

}  // namespace

// ------------------------------------------------------------------ creation
static int batch_members_check(Batch* B) {
    const t3d_context* c0 = B->m[0];
    for (size_t i = 0; i < B->m.size(); ++i) {
        const t3d_context* c = B->m[i];
        const std::string who = "batch member " + std::to_string(i) + ": ";
        if (!c->mixed) return set_error(T3D_ERR_INVALID, who + "batched designs need precision T3D_MIXED");
        if (c->standard != c0->standard) return set_error(T3D_ERR_INVALID, who + "members must share one V-cycle");
        if (c->ncases != 1) return set_error(T3D_ERR_INVALID, who + "batched designs have one load case");
        if (c->nlev < 2) return set_error(T3D_ERR_INVALID, who + "batched designs need two MG levels at least");
        if (!c->modal || c->mt.variant != B->variant || !modal_fused_available(c->mt))
            return set_error(T3D_ERR_INVALID, who + "the batched K(E)p needs the modal TMA tile shape");
        if (c->dev != c0->dev) return set_error(T3D_ERR_INVALID, who + "members must share one device");
        if (std::memcmp(&c->kh, &c0->kh, sizeof c->kh) != 0)
            return set_error(T3D_ERR_INVALID, who + "members must share one element stiffness (E0, nu)");
    }
    return T3D_OK;
}

// the launch lists of one batched PCG iteration (all arguments are fixed for the life of the batch: the
// members' buffers never move)
static int batch_lists(Batch* B) {
    T3D_CUDA_OK(cudaStreamSynchronize(B->st));
    B->free_lists();
    B->dirty = true;
    const int n = (int)B->m.size();
    if (n == 0) return T3D_OK;
    B->standard = B->m[0]->standard;
    // tensor maps per member: the PCG product (p, E); the Standard cycle's level-0 products (z, E_mg), (Ap, E_mg)
    const int per = B->standard ? 6 : 2;
    std::vector<CUtensorMap> maps((size_t)per * n);
    for (int i = 0; i < n; ++i) {
        const t3d_context* c = B->m[i];
        CUtensorMap* q = &maps[(size_t)per * i];
        bool ok = modal_tensor_maps_for(B->variant, c->g, c->p32, c->E32, q, q + 1);
        if (B->standard)
            ok = ok && modal_tensor_maps_for(B->variant, c->g, c->z32, c->E_mg32, q + 2, q + 3) &&
                 modal_tensor_maps_for(B->variant, c->g, c->Ap32, c->E_mg32, q + 4, q + 5);
        if (!ok) return set_error(T3D_ERR_CUDA, "batch member " + std::to_string(i) + ": tensor maps could not be encoded");
    }
    CHECK(B->dalloc(&B->maps, maps.size()));
    T3D_CUDA_OK(cudaMemcpyAsync(B->maps, maps.data(), maps.size() * sizeof(CUtensorMap), cudaMemcpyHostToDevice, B->st));

    B->maxL = 0;
    B->coarse_max = 0;
    B->iter_kernels = 0;
    B->iter_blocks = 0;
    for (const t3d_context* c : B->m) {
        B->maxL = std::max(B->maxL, c->nlev);
        B->coarse_max = std::max(B->coarse_max, c->Nc);
    }
    // one list: the arguments f(c, i) of the members that `take` (c, i), with their block counts
    auto list = [&](LaunchList* L, auto take, auto f, auto blocks) -> int {
        using A = decltype(f(B->m[0], 0));
        std::vector<A> a;
        std::vector<int> bl;
        std::vector<PcgScalars*> S;
        for (int i = 0; i < n; ++i) {
            t3d_context* c = B->m[i];
            if (!take(c)) continue;
            a.push_back(f(c, i));
            bl.push_back(blocks(a.back()));
            S.push_back(c->S32);
        }
        CHECK(make_list(B, a, bl, S, L));
        B->iter_kernels += L->n > 0;
        B->iter_blocks += L->blocks;
        return T3D_OK;
    };
    auto all = [](const t3d_context*) { return true; };
    auto mvb = [](const BatchMatvec& a) { return a.t.grid; };
    CHECK(list(&B->mv, all, [&](t3d_context* c, int i) {
        const CUtensorMap* q = B->maps + (size_t)per * i;
        return BatchMatvec{c->g, c->mt, c->mask0, c->Ap32, c->slot[0], c->S32, q, q + 1, nullptr, nullptr, 0.f};
    }, mvb));
    CHECK(list(&B->up, all, [](t3d_context* c, int) {
        return BatchUpdate{c->g.NNp, c->r32, c->Ap32, c->slot[1], c->S32, c->lv32[0].diag,
                           c->standard ? c->z32 : nullptr, c->prm.mg_standard_weight};
    }, [](const BatchUpdate& a) { return batch_blocks_update(a.NNp); }));
    CHECK(list(&B->dir, all, [](t3d_context* c, int) {
        return BatchDirection{c->g.NNp, c->z32, c->p32, c->d32, c->S32};
    }, [](const BatchDirection& a) { return batch_blocks_update(a.NNp); }));
    CHECK(list(&B->co, all, [](t3d_context* c, int) {
        return BatchCoarse{c->lv32[c->nlev - 1], c->Xc, c->Nc, c->chol_status, c->S32};
    }, [](const BatchCoarse& a) { return batch_blocks_coarse(a); }));
    const int norm = B->standard ? 0 : 1;
    for (int l = 0; l + 1 < B->maxL; ++l) {
        auto below = [l](const t3d_context* c) { return c->nlev - 1 > l; };
        auto rs = [&, l](t3d_context* c, int) {
            const float* src = B->standard ? (l == 0 ? c->Ap32 : c->vtmp32[l]) : (l == 0 ? c->r32 : c->lv32[l].r);
            // the Standard cycle starts the coarse level in the same kernel (the coarsest level is solved instead)
            float* x0 = B->standard && l + 2 < c->nlev ? c->lv32[l + 1].x : nullptr;
            return BatchRestrict{c->lv32[l + 1], c->lv32[l], src, c->ra1_32, c->lv32[l + 1].r, c->S32, norm, x0,
                                 c->prm.mg_standard_weight};
        };
        CHECK(list(&B->rs0[l], below, rs, [](const BatchRestrict& a) { return batch_blocks_restrict(a, 0); }));
        CHECK(list(&B->rs1[l], [&, l](const t3d_context* c) {
            return c->nlev - 1 > l && c->lv32[l + 1].span == 4;
        }, rs, [](const BatchRestrict& a) { return batch_blocks_restrict(a, 1); }));
        if (!B->standard) {
            if (l >= 1)
                CHECK(list(&B->pr[l], below, [l](t3d_context* c, int) {
                    return BatchProlong{c->lv32[l + 1], c->lv32[l], c->prm.mg_weight, c->S32};
                }, [](const BatchProlong& a) { return batch_blocks_prolong(a); }));
            continue;
        }
        // the Standard cycle's prolongations and level products; a level's corrected x is in its vtmp32
        CHECK(list(&B->pa[l], below, [l](t3d_context* c, int) {
            const MgLevel32 &Lc = c->lv32[l + 1], &Lf = c->lv32[l];
            const float* xc = l + 2 < c->nlev ? c->vtmp32[l + 1] : Lc.x;
            return l == 0 ? BatchProlongAdd{Lc, Lf, xc, c->z32, c->Ap32, c->S32}
                          : BatchProlongAdd{Lc, Lf, xc, Lf.x, Lf.x, c->S32};
        }, [](const BatchProlongAdd& a) { return batch_blocks_prolong_add(a); }));
        if (l >= 1) {
            auto op = [l](t3d_context* c, int) {
                const MgLevel32& L = c->lv32[l];
                return BatchLevelOp{L, c->Kel32[l], L.x, L.r, c->vtmp32[l], c->prm.mg_standard_weight, c->S32};
            };
            for (const bool split : {true, false}) {
                LaunchList* L = split ? &B->lsp[l] : &B->lnd[l];
                CHECK(list(L, [&](t3d_context* c) { return below(c) && batch_level_split(op(c, 0)) == split; }, op,
                           [](const BatchLevelOp& a) { return batch_blocks_level_op(a); }));
                // each level product runs twice per cycle (down and up)
                B->iter_kernels += L->n > 0;
                B->iter_blocks += L->blocks;
            }
        }
    }
    if (B->standard) {
        CHECK(list(&B->mv1, all, [&](t3d_context* c, int i) {
            const CUtensorMap* q = B->maps + (size_t)per * i + 2;
            return BatchMatvec{c->g, c->mt, c->mask0, c->Ap32, RedSlot{nullptr, nullptr}, c->S32, q, q + 1, c->r32,
                               nullptr, c->prm.mg_standard_weight};
        }, mvb));
        CHECK(list(&B->mv2, all, [&](t3d_context* c, int i) {
            const CUtensorMap* q = B->maps + (size_t)per * i + 4;
            return BatchMatvec{c->g, c->mt, c->mask0, c->z32, c->slot[2], c->S32, q, q + 1, c->r32, c->lv32[0].diag,
                               c->prm.mg_standard_weight};
        }, mvb));
    } else {
        CHECK(list(&B->p0, all, [](t3d_context* c, int) {
            return BatchProlong0{c->lv32[1], c->lv32[0], c->r32, c->z32, c->prm.mg_weight, c->slot[2], c->S32};
        }, [](const BatchProlong0& a) { return batch_blocks_prolong0(a); }));
    }
    std::vector<PcgScalars*> S;
    for (const t3d_context* c : B->m) S.push_back(c->S32);
    CHECK(B->dalloc(&B->dcompact, B->compact.size()));
    T3D_CUDA_OK(cudaMemcpyAsync(B->dcompact, B->compact.data(), B->compact.size() * sizeof(BatchCompact),
                                cudaMemcpyHostToDevice, B->st));
    B->iter_kernels += 1;   // the compaction
    CHECK(B->dalloc(&B->dS, S.size()));
    T3D_CUDA_OK(cudaMemcpyAsync(B->dS, S.data(), S.size() * sizeof(PcgScalars*), cudaMemcpyHostToDevice, B->st));
    CHECK(B->dalloc(&B->dflags, (size_t)n));
    CHECK(B->dalloc(&B->err, 1));
    T3D_CUDA_OK(cudaMemsetAsync(B->err, 0, sizeof(int), B->st));
    T3D_CUDA_OK(cudaMallocHost(&B->hflags, (size_t)n * sizeof(int)));
    T3D_CUDA_OK(cudaMallocHost(&B->hS, (size_t)n * sizeof(PcgScalars)));
    T3D_CUDA_OK(cudaMallocHost(&B->hscal, (size_t)n * sizeof(double)));
    CHECK(modal_batched_grid(B->variant, B->dev, &B->mv_grid));
    B->dirty = false;
    return T3D_OK;
}

static int batch_create(int n, const int* dims, const t3d_params* params, const t3d_problem* problems, Batch* B) {
    if (n <= 0 || !dims) return set_error(T3D_ERR_INVALID, "batch needs n > 0 members and their dims");
    std::vector<t3d_params> P((size_t)n);
    std::vector<t3d_problem> Q((size_t)n);
    for (int i = 0; i < n; ++i) {
        if (params) P[(size_t)i] = params[i];
        else {
            t3d_params_default(&P[(size_t)i]);
            P[(size_t)i].precision = T3D_MIXED;
        }
        P[(size_t)i].matvec32_tile = T3D_BATCH_TILE;
        if (problems) Q[(size_t)i] = problems[i];
        else {
            std::memset(&Q[(size_t)i], 0, sizeof(t3d_problem));
            Q[(size_t)i].load_case = T3D_LOAD_TIP_LINE;
        }
    }
    B->dev = P[0].device;
    T3D_CUDA_OK(cudaSetDevice(B->dev));
    // pass 1: the device bytes each member carves (created and released one at a time)
    size_t total = 0;
    for (int i = 0; i < n; ++i) {
        std::unique_ptr<t3d_context> t(new t3d_context());
        CHECK(create(dims[3 * i], dims[3 * i + 1], dims[3 * i + 2], &P[(size_t)i], &Q[(size_t)i], t.get()));
        total += t->carved;
    }
    // pass 2: the members inside one arena
    T3D_CUDA_OK(cudaMalloc(reinterpret_cast<void**>(&B->arena.base), total));
    B->arena.size = total;
    for (int i = 0; i < n; ++i) {
        t3d_context* c = new t3d_context();
        B->m.push_back(c);
        c->arena = &B->arena;
        const int rc = create(dims[3 * i], dims[3 * i + 1], dims[3 * i + 2], &P[(size_t)i], &Q[(size_t)i], c);
        c->arena = nullptr;
        if (rc != T3D_OK) return rc;
    }
    CHECK(batch_members_check(B));
    B->kh = B->m[0]->kh;
    B->n_arena = n;
    T3D_CUDA_OK(cudaStreamCreateWithFlags(&B->st, cudaStreamNonBlocking));
    return batch_lists(B);
}

// ------------------------------------------------------------------ the batched inner solve
template <class T>
static const T* args_of(const LaunchList& L) {
    return static_cast<const T*>(L.args);
}

static void batch_restrict(Batch* B, int l) {
    if (B->rs0[l].n) launch_batch_restrict32(args_of<BatchRestrict>(B->rs0[l]), B->rs0[l].act, B->rs0[l].n, 0, B->st);
    if (B->rs1[l].n) launch_batch_restrict32(args_of<BatchRestrict>(B->rs1[l]), B->rs1[l].act, B->rs1[l].n, 1, B->st);
}

static void batch_level_op(Batch* B, int l, bool correct) {
    for (const bool split : {true, false}) {
        const LaunchList& L = split ? B->lsp[l] : B->lnd[l];
        if (L.n) launch_batch_level_op32(args_of<BatchLevelOp>(L), L.act, L.n, split, correct, B->st);
    }
}

static void batch_product(Batch* B, int mode, const LaunchList& L) {
    launch_batch_matvec32(B->variant, mode, args_of<BatchMatvec>(L), L.act, L.n, B->kh, B->mv_grid, B->err, B->st);
}

// vcycle32 (context.cu) for every member: the Adapted cycle, or the Standard one (vcycle32_standard) with its
// level-0 residual and correction fused into the TMA products and its start z = w r / D into the update before
static void batch_vcycle(Batch* B) {
    if (!B->standard) {
        for (int l = 0; l + 1 < B->maxL; ++l) batch_restrict(B, l);
        launch_batch_coarse32(args_of<BatchCoarse>(B->co), B->co.act, B->co.n, B->coarse_max, B->st);
        for (int l = B->maxL - 2; l >= 1; --l)
            if (B->pr[l].n) launch_batch_prolong32(args_of<BatchProlong>(B->pr[l]), B->pr[l].act, B->pr[l].n, B->st);
        launch_batch_prolong0_32(args_of<BatchProlong0>(B->p0), B->p0.act, B->p0.n, B->st);
        return;
    }
    for (int l = 0; l + 1 < B->maxL; ++l) {
        if (l == 0) batch_product(B, 1, B->mv1);                       // t = r - K x
        else batch_level_op(B, l, false);
        batch_restrict(B, l);                                          // r' = P^T t, x' = w r' / D'
    }
    launch_batch_coarse32(args_of<BatchCoarse>(B->co), B->co.act, B->co.n, B->coarse_max, B->st);
    for (int l = B->maxL - 2; l >= 1; --l) {
        const LaunchList& pa = B->pa[l];
        if (!pa.n) continue;
        launch_batch_prolong_add32(args_of<BatchProlongAdd>(pa), pa.act, pa.n, B->st);        // x += P x'
        batch_level_op(B, l, true);                                                           // t = x + w (r - K x) / D
    }
    launch_batch_prolong_add32(args_of<BatchProlongAdd>(B->pa[0]), B->pa[0].act, B->pa[0].n, B->st);   // T = z + P x'
    batch_product(B, 2, B->mv2);                                      // z = T + w (r - K T) / D, with r.z
}

// one PCG iteration of every member (pcg32_iteration in context.cu, batched)
static void batch_iteration(Batch* B) {
    batch_product(B, 0, B->mv);
    launch_batch_update32(args_of<BatchUpdate>(B->up), B->up.act, B->up.n, B->st);
    batch_vcycle(B);
    launch_batch_direction32(args_of<BatchDirection>(B->dir), B->dir.act, B->dir.n, B->st);
    // members whose solve ended in this iteration (their last step applied above) leave the work lists
    launch_batch_compact(B->dcompact, (int)B->compact.size(), B->st);
}

static int batch_graph(Batch* B) {
    if (B->graph) return T3D_OK;
    cudaGraph_t graph;
    T3D_CUDA_OK(cudaStreamBeginCapture(B->st, cudaStreamCaptureModeThreadLocal));
    for (int k = 0; k < BATCH_CHUNK; ++k) batch_iteration(B);
    T3D_CUDA_OK(cudaStreamEndCapture(B->st, &graph));
    cudaError_t e = cudaGraphInstantiate(&B->graph, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) return set_cuda_error(e, "cudaGraphInstantiate", __FILE__, __LINE__);
    return T3D_OK;
}

// While the batch stream runs the members' solve, every member context issues its own launches there too (its
// stream is idle: the host synchronised it before); restored on exit.
// ------------------------------------------------------------------ the engine
//
// Members advance independently.  Each job (a member and a number of design iterations) runs on its own host
// thread and stream: SIMP, MG rebuild, the FP64 defect-correction loop (true residual, stop test,
// accumulation) and compliance, sensitivities, filter and OC.  Its inner FP32 MG-PCG is handed to the
// scheduler, which owns the batch stream: between chunks it starts the requested inner solves (scalars, the
// first V-cycle, p = z), then replays the graph of batched iterations for every member whose inner solve is
// running, and hands each finished one back to its thread.  A member's scalars are written only by the
// scheduler, between chunks, so the batched kernels never see them change inside a chunk; outside its inner
// solves a member's scalars say done and the batched launches skip it.

namespace {

// one inner solve through the scheduler: blocks until the batched iterations of this member have ended
int request_inner(Batch* B, Job* J, const PcgScalars& init) {
    std::unique_lock<std::mutex> lk(B->mu);
    J->init = init;
    J->phase = 1;
    B->cv.notify_all();
    B->cv.wait(lk, [&] { return J->phase == 3 || B->failed; });
    if (J->phase != 3) return set_error(T3D_ERR_CUDA, "batched inner solve: " + B->fail_msg);
    J->phase = 0;
    return T3D_OK;
}

// mixed_solve (context.cu) with the inner solve batched: same stop test, inner target max(stop, 1e-5 |r64|) and
// budget, so the same iterates.  *iters: inner iterations, or cg_max_it when the budget ran out unconverged.
int job_solve(Batch* B, Job* J, int* iters) {
    t3d_context* c = J->c;
    const Grid& g = c->g;
    const double tol = (double)c->prm.cg_tol;
    const int maxit = c->prm.cg_max_it;
    launch_cells_to32(g, c->E, c->E32, c->st);
    launch_dot(g, 3, c->b, c->b, c->slot[3], c->scal + 5, c->st);
    c->launches += 2;
    T3D_CUDA_OK(cudaMemcpyAsync(c->scal_h + 5, c->scal + 5, sizeof(double), cudaMemcpyDeviceToHost, c->st));
    CHECK(sync(c));
    const double nb = std::sqrt(c->scal_h[5]);
    const double stop = (1.0e-30 < nb ? nb : 1.0e-30) * tol;
    int budget = maxit, used = 0, outer = 0;
    bool converged = false;
    for (; outer < BATCH_MAX_OUTER; ++outer) {
        c->launches += 1 + matvec64(c, c->u, c->Ap, RedSlot{nullptr, nullptr}, nullptr);
        launch_mixed_residual(g, c->b, c->Ap, c->r32, c->d32, c->slot[3], c->scal + 6, c->st);
        CHECK(launch_check("mixed residual"));
        T3D_CUDA_OK(cudaMemcpyAsync(c->scal_h + 6, c->scal + 6, sizeof(double), cudaMemcpyDeviceToHost, c->st));
        CHECK(sync(c));
        const double rn = std::sqrt(c->scal_h[6]);
        if (rn < stop) {
            converged = true;
            break;
        }
        if (budget <= 0) break;
        PcgScalars init{};
        init.stop = std::max(stop, 1e-5 * rn);
        init.tol = tol;
        init.first = 1;
        init.maxit = budget;
        CHECK(request_inner(B, J, init));
        launch_mixed_accumulate(g, c->u, c->d32, c->st);
        c->launches += 1;
        T3D_CUDA_OK(cudaMemcpyAsync(c->S_h, c->S32, sizeof(PcgScalars), cudaMemcpyDeviceToHost, c->st));
        CHECK(sync(c));
        used += c->S_h->it;
        budget -= c->S_h->it;
    }
    c->last_outer = outer;
    *iters = converged ? used : maxit;
    return T3D_OK;
}

void job_main(Batch* B, Job* J) {
    cudaSetDevice(B->dev);
    t3d_context* c = J->c;
    int rc = T3D_OK;
    for (int k = 0; k < J->steps && rc == T3D_OK; ++k) {
        rc = design_pre(c);
        int its = 0;
        if (rc == T3D_OK) rc = job_solve(B, J, &its);
        if (rc == T3D_OK) {
            launch_compliance64(c->g, c->Ke, c->E, c->u, c->ce, c->slot[0], c->scal + 0, c->st);
            c->launches += 1;
            t3d_iter_record r{};
            rc = design_post(c, its, &r);
            if (rc == T3D_OK) J->recs.push_back(r);
        }
    }
    std::lock_guard<std::mutex> lk(B->mu);
    J->rc = rc;
    if (rc != T3D_OK) J->err = t3d_last_error();
    J->finished = true;
    B->cv.notify_all();
}

int member_index(const Batch* B, const t3d_context* c) {
    for (size_t i = 0; i < B->m.size(); ++i)
        if (B->m[i] == c) return (int)i;
    return -1;
}

// the scheduler's start of one member's inner solve (solve loop of mixed_solve: scalars, z = M r, p = z), issued
// on the batch stream with the member's own kernels
int start_inner(Batch* B, Job* J) {
    t3d_context* c = J->c;
    T3D_CUDA_OK(cudaMemcpyAsync(c->S32, &J->init, sizeof(PcgScalars), cudaMemcpyHostToDevice, B->st));
    const cudaStream_t own = c->st;
    c->st = B->st;
    const int rc = member_vcycle32(c, c->r32, c->z32, c->S32, c->slot[2]);
    c->st = own;
    CHECK(rc);
    T3D_CUDA_OK(cudaMemcpyAsync(c->p32, c->z32, 3 * c->g.NNp * sizeof(float), cudaMemcpyDeviceToDevice, B->st));
    return launch_check("batched solve start");
}

}  // namespace

// masks member c out of the batched launches until its first inner solve starts
static int mask_member(Batch* B, t3d_context* c) {
    PcgScalars h{};
    h.done = 1;
    T3D_CUDA_OK(cudaMemcpyAsync(c->S32, &h, sizeof h, cudaMemcpyHostToDevice, B->st));
    return T3D_OK;
}

// The scheduler.  Between chunks: adds submitted members (and starts their threads) and drops finished
// submitted ones, rebuilds the launch lists and the graph when membership changed, starts the requested
// inner solves, then replays one chunk for the members solving and hands the finished ones back to their
// threads.  Returns when every job has finished (`submitted` false: the jobs of t3d_batch_run) or, for
// submitted work, once stop is set and nothing is left to run.
static int schedule(Batch* B, bool submitted) {
    for (;;) {
        std::vector<Job*> starting, adding, dropping;
        bool solving = false;
        {
            std::unique_lock<std::mutex> lk(B->mu);
            auto any = [&](auto pred) {
                for (auto& j : B->jobs)
                    if (pred(*j)) return true;
                return false;
            };
            auto done = [&] {
                const bool running = any([](const Job& j) { return !j.finished; });
                return submitted ? (B->stop && !running && B->incoming.empty()) : !running;
            };
            auto work = [&] {
                return any([](const Job& j) { return j.phase == 1 || j.phase == 2; }) || !B->incoming.empty() ||
                       any([&](const Job& j) { return j.finished && j.release && member_index(B, j.c) >= 0; }) ||
                       done();
            };
            B->cv.wait(lk, work);
            if (!any([](const Job& j) { return j.phase == 1 || j.phase == 2; }) && B->incoming.empty() &&
                !any([&](const Job& j) { return j.finished && j.release && member_index(B, j.c) >= 0; }) && done())
                return T3D_OK;
            for (auto& j : B->incoming) {
                adding.push_back(j.get());
                B->jobs.push_back(std::move(j));
            }
            B->incoming.clear();
            for (auto& j : B->jobs) {
                if (j->finished && j->release && member_index(B, j->c) >= 0) dropping.push_back(j.get());
                if (j->phase == 1) {
                    j->phase = 2;
                    starting.push_back(j.get());
                }
                solving = solving || j->phase == 2;
            }
        }
        // membership
        for (Job* J : dropping) {
            if (J->th.joinable()) J->th.join();
            B->m.erase(B->m.begin() + member_index(B, J->c));
            B->dirty = true;
        }
        for (Job* J : adding) {
            B->m.push_back(J->c);
            int rc = batch_members_check(B);
            if (rc == T3D_OK) rc = mask_member(B, J->c);
            if (rc != T3D_OK) {
                B->m.pop_back();
                std::lock_guard<std::mutex> lk(B->mu);
                J->rc = rc;
                J->err = t3d_last_error();
                J->finished = true;
                continue;
            }
            if (B->m.size() == 1) B->kh = J->c->kh;
            B->dirty = true;
            J->started = true;
            J->th = std::thread(job_main, B, J);
        }
        if (!dropping.empty()) {
            std::lock_guard<std::mutex> lk(B->mu);
            B->cv.notify_all();   // finished submitted jobs are now collectable
        }
        if (B->dirty) CHECK(batch_lists(B));
        for (Job* J : starting) CHECK(start_inner(B, J));
        if (!solving) continue;
        CHECK(batch_graph(B));
        launch_batch_compact(B->dcompact, (int)B->compact.size(), B->st);   // the members solving in this chunk
        T3D_CUDA_OK(cudaGraphLaunch(B->graph, B->st));
        B->launches += (int64_t)BATCH_CHUNK * B->iter_kernels + 2;
        const int n = (int)B->m.size();
        launch_batch_flags(B->dS, n, B->dflags, B->st);
        T3D_CUDA_OK(cudaMemcpyAsync(B->hflags, B->dflags, (size_t)n * sizeof(int), cudaMemcpyDeviceToHost, B->st));
        T3D_CUDA_OK(cudaStreamSynchronize(B->st));
        std::lock_guard<std::mutex> lk(B->mu);
        for (auto& j : B->jobs) {
            if (j->phase != 2) continue;
            const int i = member_index(B, j->c);
            if (i >= 0 && B->hflags[i]) j->phase = 3;
        }
        B->cv.notify_all();
    }
}

static void fail(Batch* B, int rc) {
    std::lock_guard<std::mutex> lk(B->mu);
    B->failed = true;
    B->fail_msg = t3d_last_error();
    (void)rc;
    B->cv.notify_all();
}

static int check_batch_tma(Batch* B) {
    if (!B->err) return T3D_OK;
    int e = 0;
    T3D_CUDA_OK(cudaMemcpy(&e, B->err, sizeof(int), cudaMemcpyDeviceToHost));
    if (e) return set_error(T3D_ERR_CUDA, "batched TMA-staged K(E)p: an mbarrier wait timed out");
    return T3D_OK;
}

// steps[i] design iterations of member i, every member on its own thread, the inner solves batched;
// recs: the members' records one after another (steps[0] of member 0, then member 1's, ...)
static int batch_run(Batch* B, const int* steps, t3d_iter_record* recs) {
    if (B->sched.joinable()) return set_error(T3D_ERR_INVALID, "the batch is serving submitted work");
    if (B->m.empty()) return T3D_OK;
    if (B->dirty) CHECK(batch_lists(B));
    for (t3d_context* c : B->m) CHECK(mask_member(B, c));
    T3D_CUDA_OK(cudaStreamSynchronize(B->st));
    for (t3d_context* c : B->m) {
        std::unique_ptr<Job> J(new Job());
        J->c = c;
        J->steps = steps ? steps[B->jobs.size()] : 1;
        B->jobs.push_back(std::move(J));
    }
    for (auto& J : B->jobs) {
        J->started = true;
        J->th = std::thread(job_main, B, J.get());
    }
    int rc = schedule(B, false);
    if (rc != T3D_OK) fail(B, rc);
    for (auto& J : B->jobs)
        if (J->th.joinable()) J->th.join();
    std::string msg;
    int jrc = T3D_OK;
    size_t k = 0;
    for (size_t i = 0; i < B->jobs.size(); ++i) {
        Job& J = *B->jobs[i];
        if (J.rc != T3D_OK && jrc == T3D_OK) {
            jrc = J.rc;
            msg = "batch member " + std::to_string(i) + ": " + J.err;
        }
        if (recs)
            for (const t3d_iter_record& r : J.recs) recs[k++] = r;
    }
    B->jobs.clear();
    const bool failed = B->failed;
    B->failed = false;
    if (rc != T3D_OK) return rc;
    if (failed) return set_error(T3D_ERR_CUDA, B->fail_msg);
    if (jrc != T3D_OK) return set_error(jrc, msg);
    return check_batch_tma(B);
}

}  // namespace t3d

// ====================================================================== C-ABI
struct t3d_batch : public t3d::Batch {};

extern "C" {

int t3d_batch_create(int n, const int* dims, const t3d_params* params, const t3d_problem* problems, t3d_batch** out) {
    if (!out) return t3d::set_error(T3D_ERR_INVALID, "null argument");
    *out = nullptr;
    t3d_batch* b = new (std::nothrow) t3d_batch();
    if (!b) return t3d::set_error(T3D_ERR_OOM, "host allocation failed");
    const int rc = t3d::batch_create(n, dims, params, problems, b);
    if (rc != T3D_OK) {
        delete b;
        return rc;
    }
    *out = b;
    return T3D_OK;
}

int t3d_batch_open(int device, t3d_batch** out) {
    if (!out) return t3d::set_error(T3D_ERR_INVALID, "null argument");
    *out = nullptr;
    t3d_batch* b = new (std::nothrow) t3d_batch();
    if (!b) return t3d::set_error(T3D_ERR_OOM, "host allocation failed");
    b->dev = device;
    cudaError_t e = cudaSetDevice(device);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&b->st, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
        delete b;
        return t3d::set_cuda_error(e, "t3d_batch_open", __FILE__, __LINE__);
    }
    *out = b;
    return T3D_OK;
}

int t3d_batch_adopt(t3d_batch* b, t3d_context* ctx) {
    if (!b || !ctx) return t3d::set_error(T3D_ERR_INVALID, "null argument");
    if (b->sched.joinable()) return t3d::set_error(T3D_ERR_INVALID, "the batch is serving submitted work");
    if (!ctx->design_ready) return t3d::set_error(T3D_ERR_INVALID, "t3d_design_init not called on the context");
    for (const t3d_context* c : b->m)
        if (c == ctx) return t3d::set_error(T3D_ERR_INVALID, "context is already a batch member");
    if (cudaSetDevice(b->dev) != cudaSuccess) return t3d::set_error(T3D_ERR_CUDA, "cudaSetDevice failed");
    if (ctx->dev != b->dev) return t3d::set_error(T3D_ERR_INVALID, "context is on another device");
    b->m.push_back(ctx);
    const int rc = t3d::batch_members_check(b);
    if (rc != T3D_OK) {
        b->m.pop_back();
        return rc;
    }
    if (b->m.size() == 1) b->kh = ctx->kh;
    b->dirty = true;
    return T3D_OK;
}

int t3d_batch_release(t3d_batch* b, int i, t3d_context** out) {
    if (!b || !out || i < 0 || i >= (int)b->m.size()) return t3d::set_error(T3D_ERR_INVALID, "bad batch member");
    if (i < b->n_arena) return t3d::set_error(T3D_ERR_INVALID, "member lives in the batch arena");
    if (b->sched.joinable()) return t3d::set_error(T3D_ERR_INVALID, "the batch is serving submitted work");
    if (cudaSetDevice(b->dev) != cudaSuccess) return t3d::set_error(T3D_ERR_CUDA, "cudaSetDevice failed");
    if (cudaStreamSynchronize(b->st) != cudaSuccess) return t3d::set_error(T3D_ERR_CUDA, "batch stream failed");
    *out = b->m[(size_t)i];
    b->m.erase(b->m.begin() + i);
    b->dirty = true;
    return T3D_OK;
}

int t3d_batch_member(t3d_batch* b, int i, t3d_context** out) {
    if (!b || !out || i < 0 || i >= (int)b->m.size()) return t3d::set_error(T3D_ERR_INVALID, "bad batch member");
    *out = b->m[(size_t)i];
    return T3D_OK;
}

// One member after another, each on its own stream (a first solve also captures the member's PCG graph).
int t3d_batch_design_init(t3d_batch* b, const float* V0, double* c_solid) {
    if (!b || !V0) return t3d::set_error(T3D_ERR_INVALID, "null argument");
    if (cudaSetDevice(b->dev) != cudaSuccess) return t3d::set_error(T3D_ERR_CUDA, "cudaSetDevice failed");
    for (size_t i = 0; i < b->m.size(); ++i) {
        const int rc = t3d::design_init(b->m[i], V0[i], c_solid ? c_solid + i : nullptr);
        if (rc != T3D_OK) return t3d::set_error(rc, "batch member " + std::to_string(i) + ": " + t3d_last_error());
    }
    return T3D_OK;
}

int t3d_batch_design_step(t3d_batch* b, t3d_iter_record* recs) {
    if (!b) return t3d::set_error(T3D_ERR_INVALID, "null batch");
    if (cudaSetDevice(b->dev) != cudaSuccess) return t3d::set_error(T3D_ERR_CUDA, "cudaSetDevice failed");
    return t3d::batch_run(b, nullptr, recs);
}

int t3d_batch_run(t3d_batch* b, const int* steps, t3d_iter_record* recs) {
    if (!b || !steps) return t3d::set_error(T3D_ERR_INVALID, "null argument");
    for (size_t i = 0; i < b->m.size(); ++i)
        if (steps[i] < 0) return t3d::set_error(T3D_ERR_INVALID, "negative step count");
    if (cudaSetDevice(b->dev) != cudaSuccess) return t3d::set_error(T3D_ERR_CUDA, "cudaSetDevice failed");
    return t3d::batch_run(b, steps, recs);
}

int t3d_batch_submit(t3d_batch* b, t3d_context* ctx, int steps) {
    if (!b || !ctx || steps < 0) return t3d::set_error(T3D_ERR_INVALID, "bad argument");
    if (!ctx->design_ready) return t3d::set_error(T3D_ERR_INVALID, "t3d_design_init not called on the context");
    if (ctx->dev != b->dev) return t3d::set_error(T3D_ERR_INVALID, "context is on another device");
    std::lock_guard<std::mutex> lk(b->mu);
    if (b->stop) return t3d::set_error(T3D_ERR_INVALID, "the batch is shutting down");
    if (!b->sched.joinable() && !b->m.empty())
        return t3d::set_error(T3D_ERR_INVALID, "submitted work needs a batch without members (t3d_batch_open)");
    std::unique_ptr<t3d::Job> J(new t3d::Job());
    J->c = ctx;
    J->steps = steps;
    J->release = true;
    b->incoming.push_back(std::move(J));
    if (!b->sched.joinable()) {
        t3d::Batch* B = b;
        b->sched = std::thread([B] {
            cudaSetDevice(B->dev);
            const int rc = t3d::schedule(B, true);
            if (rc != T3D_OK) t3d::fail(B, rc);
        });
    }
    b->cv.notify_all();
    return T3D_OK;
}

int t3d_batch_collect(t3d_batch* b, int timeout_ms, t3d_context** ctx, t3d_iter_record* recs, int cap, int* nrec,
                      int* status) {
    if (!b || !ctx || !nrec || !status) return t3d::set_error(T3D_ERR_INVALID, "null argument");
    *ctx = nullptr;
    *nrec = 0;
    *status = T3D_OK;
    std::unique_lock<std::mutex> lk(b->mu);
    auto ready = [&]() -> int {
        for (size_t i = 0; i < b->jobs.size(); ++i) {
            const t3d::Job& J = *b->jobs[i];
            if (J.release && J.finished && t3d::member_index(b, J.c) < 0) return (int)i;
        }
        return -1;
    };
    int k = ready();
    if (k < 0 && !b->failed)
        b->cv.wait_for(lk, std::chrono::milliseconds(timeout_ms > 0 ? timeout_ms : 0),
                       [&] { return (k = ready()) >= 0 || b->failed; });
    if (k < 0) {
        if (b->failed) return t3d::set_error(T3D_ERR_CUDA, "batch scheduler: " + b->fail_msg);
        return T3D_OK;   // nothing finished yet
    }
    std::unique_ptr<t3d::Job> J = std::move(b->jobs[(size_t)k]);
    b->jobs.erase(b->jobs.begin() + k);
    lk.unlock();
    if (J->th.joinable()) J->th.join();
    *ctx = J->c;
    const int n = std::min<int>(cap, (int)J->recs.size());
    for (int i = 0; i < n && recs; ++i) recs[i] = J->recs[(size_t)i];
    *nrec = n;
    *status = J->rc;
    if (J->rc != T3D_OK) t3d::set_error(J->rc, J->err);
    return T3D_OK;
}

int t3d_batch_info(t3d_batch* b, int64_t* info) {
    if (!b || !info) return t3d::set_error(T3D_ERR_INVALID, "null argument");
    int64_t member = 0;
    for (const t3d_context* c : b->m) member += c->launches;
    info[0] = (int64_t)b->arena.size;
    info[1] = (int64_t)b->m.size();
    info[2] = b->launches;
    info[3] = b->iter_kernels;
    info[4] = b->iter_blocks;
    info[5] = member;
    return T3D_OK;
}

int t3d_batch_destroy(t3d_batch* b) {
    if (!b) return T3D_OK;
    if (b->sched.joinable()) {   // submitted work: let the running jobs finish, then stop the scheduler
        {
            std::lock_guard<std::mutex> lk(b->mu);
            b->stop = true;
            b->cv.notify_all();
        }
        b->sched.join();
        for (auto& J : b->jobs) {
            if (J->th.joinable()) J->th.join();
            if (t3d::member_index(b, J->c) < 0) delete J->c;   // finished and released, never collected
        }
        for (auto& J : b->incoming) delete J->c;
    }
    delete b;
    return T3D_OK;
}

}  // extern "C"
