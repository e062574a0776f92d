// gdp_context.h -- host-side propagation context (device layout + drivers).
#pragma once

#include <cuda_runtime.h>

#include <exception>
#include <functional>
#include <initializer_list>
#include <new>
#include <string>
#include <vector>

#include "gdp_ext.h"
#include "gdp_internal.h"
#include "gdp_mlp.h"

namespace gdp {

void set_error(const std::string &msg);
const char *last_error();

// Owns device allocations. Released blocks go to a process-wide cache of
// device memory that later arenas draw from, so contexts of one problem size
// can be created and destroyed without cudaMalloc / cudaFree (each costs up
// to milliseconds for blocks of hundreds of MB).
struct Arena {
    struct Block {
        void *p;
        size_t bytes;
        int dev;
    };
    std::vector<Block> blocks;
    struct Piece {
        void **dst;
        size_t bytes;
    };
    ~Arena();
    void *alloc_bytes(size_t bytes);
    bool carve(std::initializer_list<Piece> pieces);  // one block for all pieces, 256-byte aligned
    void release();  // waits for the device, then returns every block to the cache
};

// What a context needs besides device memory: two streams (its own, and one
// for uploads during the build), events, and page-locked memory for the round
// flags and a stage for small uploads. Taken from and given back to a bounded
// process-wide pool.
struct HostResources {
    static constexpr size_t kFlagBytes = 4096;
    static constexpr size_t kStageBytes = 1 << 20;
    int device = 0;
    cudaStream_t stream = nullptr, upload = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr, uploaded = nullptr;
    void *pinned = nullptr;
};
static_assert(3 * sizeof(RoundFlags) <= HostResources::kFlagBytes, "the flags fit their part");
HostResources *take_resources(int device, cudaError_t *err);
void give_resources(HostResources *r);
void release_kept_resources();  // destroys the sets that the pool keeps

// Frees the cached device memory of released arenas (all devices).
void release_cached_memory();

GDP_RETCODE autotune(int m, int n, int nnz, const int *col, const int *row_ptr, const double *val,
                     const double *lhs, const double *rhs, const double *lbs, const double *ubs,
                     const int *vartype, const gdp_options *base, int repeats, gdp_options *best,
                     double *best_ms, gdp_tune_trial *trials, int max_trials, int *n_trials);
GDP_RETCODE autotune_clear_cache();

GDP_RETCODE validate_csr(int m, int n, int nnz, const int *col, const int *row_ptr,
                         const double *val, const int *vartype);

// The reference's CALL_AND_HANDLE (src/interface.cu:7-16): exceptions become
// GDP_ERROR; here with the message kept for gdp_last_error().
template <class F>
GDP_RETCODE guarded(F &&f) {
    try {
        return f();
    } catch (const std::bad_alloc &) {
        set_error("host allocation failed");
        return GDP_ERROR;
    } catch (const std::exception &e) {
        set_error(e.what());
        return GDP_ERROR;
    } catch (...) {
        set_error("unknown exception");
        return GDP_ERROR;
    }
}

class Context {
public:
    ~Context();
    GDP_RETCODE init(int m, int n, int nnz, const int *col, const int *row_ptr, const double *val,
                     const double *lhs, const double *rhs, const int *vartype, const gdp_options *o);
    // Host bounds (an output may be its input); a failed call leaves the inputs
    // in the outputs.
    GDP_RETCODE propagate_host(const double *lbs_in, const double *ubs_in, double *lbs_out, double *ubs_out,
                               gdp_stats *st);
    GDP_RETCODE propagate_device(double *d_lbs, double *d_ubs, cudaStream_t s, gdp_stats *st);
    // Loop driver, resident CTAs per SM (0: as many as fit) and megakernel CTA
    // size of later propagations; the layout stays.
    GDP_RETCODE set_schedule(int sync_type, int ctas_per_sm, int cta_threads);
    // Gives the streams, events and page-locked memory back: a batch member's
    // context is only a layout once it is built.
    void release_host_resources();
    // Learned marking with model m (NULL: off), logit threshold and the
    // shortest row length the model decides for.
    GDP_RETCODE set_model(const Mlp *m, float threshold, int min_len);
    // Trace propagation: exact marking, logging up to `capacity` samples.
    GDP_RETCODE trace(double *lbs, double *ubs, int capacity, float *x_out, float *y_out, int *n_out,
                      gdp_stats *st);

    int m = 0, n = 0, nnz = 0;
    gdp_options opts{};
    HostResources *res = nullptr;
    cudaStream_t stream = nullptr;  // this and the next three: res's
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    RoundFlags *h_flags = nullptr;  // pinned
    Arena arena;
    DevProblem P{};
    double *d_lb = nullptr, *d_ub = nullptr;  // staging for host bounds (alloc_staging)
    int n_sms = 0, vec_blocks = 1, act_blocks = 1, cand_blocks = 1, mega_grid = 1, learned_grid = 1;
    int mega_warps = 8;  // warps per CTA of the megakernel (opts.cta_threads / 32; 16 where that is 0)
    int n_srows = 0, n_slices = 0, n_lrows = 0, n_tiles = 0;
    long long sell_elems = 0;
    // the last propagation converged feasibly: P.bnd is a fixpoint of the problem
    bool certified = false;
    bool host_direct = false;  // kernels read and write pageable host memory (coherent access)
    // GPU_LOOP graph (built on first use, reused while the context lives)
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t graph_exec = nullptr;

private:
    GDP_RETCODE run(const double *lb_in, const double *ub_in, double *lb_out, double *ub_out,
                    cudaStream_t s, gdp_stats *st);
    GDP_RETCODE build_graph();
    // meanwhile: host work to do once the first rounds are queued
    GDP_RETCODE rounds_cpu_loop(cudaStream_t s, int *launches, const std::function<void()> &meanwhile);
    GDP_RETCODE rounds_gpu_loop(cudaStream_t s);
    void copy_bounds(const double *lbs_in, const double *ubs_in, double *lbs_out, double *ubs_out) const;
    GDP_RETCODE rounds_megakernel(cudaStream_t s, int *launches);
    GDP_RETCODE rounds_learned(cudaStream_t s, int *launches);
    GDP_RETCODE alloc_learned_state();
    GDP_RETCODE alloc_staging();
};

}  // namespace gdp
