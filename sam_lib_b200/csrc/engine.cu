// GPU numeric phase of SPR for sm_100a: supernodal multifrontal LDL'
// factorisation and the forward/diagonal/back solves.
//
// Semantics follow the reference routines (file:line in src/SPR):
//   SPRF11 multifrontal loop ............ sprfc1.f:286-713
//   SPRF12/13/14 extend-add ............. sprfc1.f:716-982
//   SPRF15/SPRF17 (+LMVY18) pivots ...... sprfc1.f:985-1299, lmvy18.f
//   LMMY18 Schur update ................. lmmy18.f:5-192
//   SPRFS3/5/6 forward + diagonal ....... sprfs1.f:266-1141
//   SPRBS4/6 back substitution .......... sprbs1.f:251-574
// The arithmetic is FP64, but for large Schur updates: sums of 8-bit digit
// products whose errors are below those of FP64 multiply-adds (i8_gemm.cuh), or, in
// the mixed modes, split TF32 products (tc_gemm.cuh, x3).  The order of the
// floating-point updates differs from the reference (blocked, FMA), so results
// agree to rounding.
//
// Execution: one pass per elimination-tree level (leaves first).  Fronts of
// order <= kSmallMaxF are assembled, factored and written back by one CTA in
// shared memory (fused extend-add + LDL' + Schur update).  Larger fronts are
// assembled into dense column-major buffers in HBM and factored with a
// blocked right-looking LDL' (a launch per panel step: TRSM, the next panel's
// columns, the next diagonal block; DMMA or digit products for the other Schur
// updates), all fronts of the level batched into each launch.
#include <cuda.h>
#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <condition_variable>
#include <deque>
#include <mutex>
#include <thread>

#include "engine.h"
#include "smhash.h"

namespace sprb {

bool trace_on() {
    static const bool on = [] {
        const char* e = std::getenv("SPR_B200_TRACE");
        return e && e[0] == '1';
    }();
    return on;
}
static std::chrono::steady_clock::time_point g_trace_t0;
void trace_reset() {
    if (trace_on()) g_trace_t0 = std::chrono::steady_clock::now();
}
void trace_point(const char* what) {
    if (!trace_on()) return;
    const double ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - g_trace_t0).count();
    fprintf(stderr, "[spr_b200 trace] %9.3f ms  %s\n", ms, what);
}


// (the error is taken off the thread: after a failed allocation the next call starts clean)
#define CK(x)                                                                    \
    do {                                                                         \
        cudaError_t e_ = (x);                                                    \
        if (e_ != cudaSuccess) {                                                 \
            cudaGetLastError();                                                  \
            fprintf(stderr, "spr_b200: CUDA error %s at %s:%d\n",                \
                    cudaGetErrorString(e_), __FILE__, __LINE__);                 \
            return -4;                                                           \
        }                                                                        \
    } while (0)

constexpr int kMaxRHS = 16;          // right-hand sides per CTA of the small fronts and per residual pass
// Right-hand sides per pass over the factor.  A wider pass reads L less often and
// fills the chain of a front's blocks better; the work buffers grow with it
// (48: 3 times those of 16).  96 right-hand sides with 16, 32, 48, 64 and 96 a pass: 12^3 4.5,
// 2.4, 1.7, 1.7, 1.0 ms; 24^3 13.0, 8.6, 7.2, 7.2, 5.9; 32^3 27.1, 21.4, 19.5, 19.5, 17.6.
constexpr int kPassRHS = 48;

// NVTX range for the host timeline of a profiler (no-op without one).
struct NvtxRange {
    explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
    ~NvtxRange() { nvtxRangePop(); }
};

// ---------------------------------------------------------------------------
// Device views
// ---------------------------------------------------------------------------
struct Stats {
    int zero_count;
    int first_zero;          // smallest 0-based column with an exact zero diagonal
    int any_fail;            // exact zero diagonal found: nothing is factored (sprfc1.f:488)
    int pivot_fail;          // some pivot failed the TOL(1) test
    unsigned long long numneg;
    double tol2;             // max(a_jj / d_j), sprfc1.f:1284
    double trace;            // sum a_jj, sprfc1.f:483
    double mindpos;          // smallest positive pivot, sprfc1.f:690-697
    int tc_timeout;          // a tensor-core update CTA gave up waiting (see tc_gemm.cuh)
    unsigned long long nsing;    // SPRFC3: pivots replaced by the TOL(1)/TOL(4) rule
    unsigned long long near_piv; // pivots with |d| < near_tol |a_jj| (mixed-mode inertia guard)
    int solve_timeout;       // a triangle task of the solves gave up waiting for a block (k_*_tri)
};

struct PV {
    const int32_t *fst, *S, *F, *child_ptr, *child, *rows, *rel, *cchild, *ct, *buf_ld;
    const int64_t *lnz_off, *rel_off, *rbase, *cptr, *buf_off, *upd_off;
    double* arena;
    double* lnz;
    double* dvec;
    double* adiag;
    int32_t* sn_neg;
    int32_t* sn_fail;
    int32_t* sn_bad;         // front failed, or depends on a failed front
    double* sn_faild;
    double* sn_faila;
    Stats* st;
    const int64_t* linv_off;
    double* linv;            // inverses of the unit-lower diagonal blocks
    const int64_t* rect_off;
    const int64_t* fwd_off;
    double tol1;
    // SPRFC3 semantics (sprfc3.f:549-572, 1083-1099): a zero diagonal becomes
    // 1 and a pivot at or below TOL(1)|a_jj| is replaced instead of stopping;
    // both are recorded in DCOR(2,NEQ) (dcor[2j], dcor[2j+1])
    int fc3;
    double tol4;
    double* dcor;
    // partial factorisation: 1 for the retained supernodes (null if none)
    const uint8_t* ret;
    // inertia guard of the mixed mode: pivots with |d| < near_tol |a_jj| are
    // counted (their sign may depend on the TF32 rounding); 0 = off
    double near_tol;
    // time limit of every mbarrier wait of the tensor-core update (ns), and a
    // test switch: when set, CTA 0 of each tensor-core launch skips its first
    // operand load, so that its waits run out and the launch reports a timeout
    unsigned long long wait_ns;
    int tc_drop;
    // streamed factorisation: the original diagonal gathered on the host
    // (the pre-pass then reads it instead of LNZ, which is still uploading)
    const double* adiag_in;
    // node mask of a run split across GPUs: supernodes with skip[js] != 0 are
    // left alone (null: none)
    const uint8_t* skip;
    // per equation (sign(d) sqrt|d|, its rounding error) of the large fronts'
    // pivots, for the integer-digit updates (null: not wanted)
    double* sqd;
};

struct Engine::Dev {
    // plan arrays
    int32_t *fst = nullptr, *S = nullptr, *F = nullptr, *child_ptr = nullptr, *child = nullptr,
            *rows = nullptr, *rel = nullptr, *cchild = nullptr, *ct = nullptr, *buf_ld = nullptr;
    int64_t *lnz_off = nullptr, *rel_off = nullptr, *rbase = nullptr, *cptr = nullptr,
            *buf_off = nullptr, *upd_off = nullptr;
    Job* jobs = nullptr;
    int64_t* linv_off = nullptr;
    double* linv = nullptr;
    int32_t* task_map = nullptr;
    int64_t* rect_off = nullptr;
    int64_t* fwd_off = nullptr;
    double* pbuf = nullptr;                      // rectangle partial sums of the solves
    int32_t* level_nodes = nullptr;              // small nodes of every level, concatenated
    std::vector<int64_t> small_begin;            // per level offset into level_nodes
    // work
    double* arena = nullptr;
    double* adiag = nullptr;
    int32_t* sn_neg = nullptr;
    int32_t* sn_fail = nullptr;
    int32_t* sn_bad = nullptr;
    uint8_t* ret = nullptr;                      // retained supernodes (partial factorisation)
    double* sn_faild = nullptr;
    double* sn_faila = nullptr;
    Stats* st = nullptr;
    double* vbuf = nullptr;                      // update vectors of the forward sweep
    double* ybuf = nullptr;                      // solved rows of the large fronts
    int64_t vbuf_rhs = 0;                        // right-hand sides that vbuf, ybuf and pbuf hold
    int64_t pass_rhs = kPassRHS;                 // right-hand sides per pass (kMaxRHS once kPassRHS did not fit)
    uint8_t* skip = nullptr;                     // node mask of a split run
    bool skip_on = false;
    int32_t* tri_tasks = nullptr;                // the solves' triangle tasks (node, block)
    int32_t* tri_sync = nullptr;                 // per level a task counter and an abort word
    std::vector<void*> owned;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    // page-locked, device-mapped mailbox for the few words the host reads
    // after each call (the factorisation's Stats, a hash, the solve's
    // timeout flag): a kernel writes them over the bus, so the read does not
    // queue on the copy engine behind a streamed factorisation's downloads
    unsigned long long* mbox = nullptr;         // host address
    unsigned long long* mbox_dev = nullptr;     // its device address
    unsigned long long* hbuf = nullptr;          // result of k_sm_hash
    // tensor-core (mixed) updates: operand slabs and the TMA map over them
    float* slab = nullptr;
    alignas(64) CUtensorMap slab_map;
    float* slab_far = nullptr;                   // slabs of the side-stream launches
    int32_t* tc_off = nullptr;                   // fronts left out, per supernode: launches on the stream, side-stream ones
    alignas(64) CUtensorMap slab_map_far;
    // integer-digit updates: digit slabs, row scales, the TMA maps over the slabs
    uint8_t* i8_slab = nullptr;
    double* i8_scales = nullptr;
    alignas(64) CUtensorMap i8_map_a, i8_map_b;
    double* sqd = nullptr;                       // (sqrt|d| with d's sign, its rounding error) per equation
    cudaStream_t side = nullptr;                 // side stream: trailing updates beyond the next super-panel
    cudaStream_t ahead = nullptr;                // look-ahead stream: in-super-panel columns after the next two panels
    cudaStream_t wbs = nullptr;                  // early writes of final super-panels to LNZ (streamed copies)
    std::vector<cudaEvent_t> evpool;             // fork/join events of one factorisation
};

template <typename T>
static int dev_upload(std::vector<void*>& owned, T** dst, const std::vector<T>& src) {
    size_t n = std::max<size_t>(src.size(), 1);
    CK(cudaMalloc((void**)dst, n * sizeof(T)));
    owned.push_back(*dst);
    if (!src.empty()) CK(cudaMemcpy(*dst, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice));
    return 0;
}

// ---------------------------------------------------------------------------
// Small device helpers
// ---------------------------------------------------------------------------
__device__ __forceinline__ void atomic_max_double(double* addr, double v) {
    unsigned long long* a = reinterpret_cast<unsigned long long*>(addr);
    unsigned long long old = *a;
    while (__longlong_as_double((long long)old) < v) {
        unsigned long long assumed = old;
        old = atomicCAS(a, assumed, (unsigned long long)__double_as_longlong(v));
        if (old == assumed) break;
    }
}

__device__ __forceinline__ int64_t find_job(const Job* jobs, int64_t n, int64_t t) {
    int64_t lo = 0, hi = n - 1;
    while (lo < hi) {
        int64_t mid = (lo + hi + 1) >> 1;
        if (jobs[mid].task0 <= t) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// job of a task: one load from the launch's task map, or a binary search
// over the jobs' first tasks when no map is given
__device__ __forceinline__ const Job& job_of(const Job* jobs, int64_t njobs, const int32_t* tmap, int64_t t) {
    return tmap ? jobs[tmap[t]] : jobs[find_job(jobs, njobs, t)];
}

// packed lower, column-major, order F: column j holds rows j..F-1
__device__ __forceinline__ int pk(int i, int j, int F) { return j * F - ((j * (j - 1)) >> 1) + (i - j); }

__host__ __device__ __forceinline__ int64_t lnz_col(int64_t j, int64_t F) { return j * F - (j * (j - 1)) / 2; }

// record a failed pivot (sprfc1.f:1274-1279): first failure per supernode wins
// A failed front poisons its ancestors only: fronts earlier in postorder than
// the first failure are still factored, so NUMNEG matches the reference's count
// of negative pivots met before it stops (sprfc1.f:610-616).
__device__ void record_fail(const PV& P, int js, int col, double d, double ad) {
    P.sn_fail[js] = col;
    P.sn_faild[js] = d;
    P.sn_faila[js] = ad;
    P.sn_bad[js] = 1;
    atomicExch(&P.st->pivot_fail, 1);
}

// A retained supernode of a partial factorisation (MSPAR(57) > 0, SUPSUP > 0):
// assembled but not eliminated (sprfc1.f:587), skipped by the solves
// (sprfs1.f:371, sprbs1.f:347).
__device__ __forceinline__ bool is_retained(const PV& P, int js) { return P.ret != nullptr && P.ret[js] != 0; }

// SPRF37 (sprfc3.f:1083-1099): the pivot d of a column with original
// diagonal ad becomes sign(TOL(1) max(1, |TOL(4) ad|), d) when |d| <= TOL(1)|ad|.
__device__ __forceinline__ double fc3_pivot(const PV& P, double d, double ad) {
    return fabs(d) <= P.tol1 * fabs(ad) ? copysign(fabs(P.tol1 * fmax(1.0, fabs(P.tol4 * ad))), d) : d;
}

// DCOR entries of column col (0-based) for the pivot d0 before and dn after
// the replacement: DCOR(1) = d0 on a replacement, else (or if d0 == 0) dn when
// dn < 0; DCOR(2) = dn on a replacement.  One thread per column.
__device__ __forceinline__ void fc3_record(const PV& P, int col, double d0, double dn) {
    const bool sing = fabs(d0) <= P.tol1 * fabs(P.adiag[col]);
    double* dc = P.dcor + 2 * (int64_t)col;
    double c1 = sing ? d0 : 0.0;
    if (dn < 0.0 && c1 == 0.0) c1 = dn;
    if (sing || dn < 0.0) dc[0] = c1;
    if (sing) {
        dc[1] = dn;
        atomicAdd(&P.st->nsing, 1ull);
    }
}

// a supernode another GPU handles (split runs)
__device__ __forceinline__ bool node_off(const PV& P, int js) { return P.skip != nullptr && P.skip[js] != 0; }

__device__ __forceinline__ bool children_bad(const PV& P, int js) {
    for (int k = P.child_ptr[js]; k < P.child_ptr[js + 1]; ++k)
        if (P.sn_bad[P.child[k]]) return true;
    return false;
}

// ---------------------------------------------------------------------------
// Pre-pass: original diagonal, zero test, trace (sprfc1.f:465-488)
// ---------------------------------------------------------------------------
__global__ void k_prepass(PV P, int64_t nsuper) {
    const int lane = threadIdx.x & 31;
    for (int64_t js = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; js < nsuper;
         js += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        const int s = P.S[js], f = P.F[js], fst = P.fst[js];
        double* col = P.lnz + P.lnz_off[js];
        if (is_retained(P, js)) {                     // D stays 0 (sprfc1.f:463-467, sprfc3.f:551-554)
            for (int j = lane; j < s; j += 32) {
                P.adiag[fst + j] = 0.0;
                P.dvec[fst + j] = 0.0;
                if (P.fc3) {
                    P.dcor[2 * (int64_t)(fst + j)] = 0.0;
                    P.dcor[2 * (int64_t)(fst + j) + 1] = 0.0;
                }
            }
            continue;
        }
        for (int j = lane; j < s; j += 32) {
            double a = P.adiag_in ? P.adiag_in[fst + j] : col[lnz_col(j, f)];
            if (P.fc3) {                                  // sprfc3.f:561-572
                double* dc = P.dcor + 2 * (int64_t)(fst + j);
                dc[0] = 0.0;
                dc[1] = 0.0;
                if (a == 0.0) {
                    a = 1.0;
                    dc[1] = 1.0;
                    col[lnz_col(j, f)] = 1.0;
                }
                P.adiag[fst + j] = a;
                continue;
            }
            P.adiag[fst + j] = a;
            if (a == 0.0) {
                atomicAdd(&P.st->zero_count, 1);
                atomicMin(&P.st->first_zero, fst + j);
                atomicExch(&P.st->any_fail, 1);
            }
        }
    }
}

// Content hash of a device array (see smhash.h): each thread sums its words'
// mixes, the partial sums meet in one 64-bit atomic add (order-free).
__global__ void k_sm_hash(const double* a, int64_t n, unsigned long long* out) {
    unsigned long long acc = 0ull;
    const uint64_t* w = reinterpret_cast<const uint64_t*>(a);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        acc += sm_mix(__ldcs(reinterpret_cast<const unsigned long long*>(w + i)), (uint64_t)i);
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(out, acc);
}

// Deterministic single-CTA reductions over a vector: sum, or min over positives.
template <bool kMinPos>
__global__ void k_reduce(const double* v, int64_t n, double* out) {
    __shared__ double red[1024];
    double acc = kMinPos ? 0.0 : 0.0;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        const double x = v[i];
        if (kMinPos) {
            if (x > 0.0 && (acc == 0.0 || x < acc)) acc = x;
        } else {
            acc += x;
        }
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) {
            const double a = red[threadIdx.x], b = red[threadIdx.x + s];
            if (kMinPos) {
                red[threadIdx.x] = (a == 0.0) ? b : ((b == 0.0) ? a : (a < b ? a : b));
            } else {
                red[threadIdx.x] = a + b;
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = red[0];
}

// ---------------------------------------------------------------------------
// Small fronts: fused extend-add + LDL' + Schur update, one CTA per front.
// Shared memory holds the packed lower front F(F+1)/2 plus one column.
// ---------------------------------------------------------------------------
// Pivot rules of the factorisation kernels: SPRF17's |d| <= TOL(1)|a| stops
// (sprfc1.f:1274), SPRF37 replaces the pivot (sprfc3.f:1083), SPRF27's
// d <= TOL(1)|a| stops the Cholesky form (sprfc2.f:1001-1008; the C C'
// factor is formed from L D L' afterwards, see k_chol_convert).
// SPRF47 (sprfc4.f:978-1000) is the Cholesky form of SPRF37: a pivot below
// -TOL(1)|a_jj| stops, one in [-TOL(1)|a_jj|, TOL(1)|a_jj|] is replaced by
// TOL(1) max(1, |TOL(4) a_jj|) and recorded in DCOR(1:2, j).
enum PivotRule { kPivotLDL = 0, kPivotReplace = 1, kPivotChol = 2, kPivotChol4 = 3 };

// 1/c for the pivots: the hardware reciprocal approximation (rcp.approx.ftz.f64)
// refined by two Newton-Raphson steps x <- x + x (1 - c x), each with fused
// multiply-adds; within one ulp of 1/c for normal c (tests compare it with
// the IEEE quotient 1.0 / c over many values).  Zero, subnormal, huge and
// non-finite c take the quotient itself.  It replaces a division on the
// pivot chain of every elimination step.
__device__ __forceinline__ double recip_nr(double c) {
    // (the approximation first, so that it does not wait for the test)
    double r;
    asm volatile("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(c));
    r = fma(r, fma(-c, r, 1.0), r);
    r = fma(r, fma(-c, r, 1.0), r);
    const unsigned e = ((unsigned)__double2hiint(c) >> 20) & 0x7ffu;
    if (e - 1u > 2044u) r = 1.0 / c;                 // biased exponents 1 .. 2045: 2^-1022 <= |c| < 2^1023
    return r;
}

// the same where c is the same in all lanes of the warp: a uniform branch
__device__ __forceinline__ double recip_nr_uniform(double c) {
    double r;
    asm volatile("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(c));
    r = fma(r, fma(-c, r, 1.0), r);
    r = fma(r, fma(-c, r, 1.0), r);
    const unsigned e = ((unsigned)__double2hiint(c) >> 20) & 0x7ffu;
    if (__any_sync(0xffffffffu, e - 1u > 2044u)) r = 1.0 / c;
    return r;
}

__global__ void k_recip_check(const double* x, int64_t n, double* out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) {
        out[2 * i] = recip_nr(x[i]);
        out[2 * i + 1] = 1.0 / x[i];
    }
}

// A NaN or infinite pivot (a NaN or Inf anywhere in SM reaches some pivot
// through the Schur updates) fails the test as well, so that the call reports
// an error instead of a factor full of NaN.
__device__ __forceinline__ bool pivot_fails(int rule, double d, double ad, double tol1) {
    if (!isfinite(d)) return true;
    if (rule == kPivotChol4) return d < -tol1 * fabs(ad);
    return rule == kPivotChol ? d <= tol1 * fabs(ad) : fabs(d) <= tol1 * fabs(ad);
}

// SPRF47's replacement of a small pivot (not a failing one): returns the
// pivot to use and records DCOR(1,j) = d, DCOR(2,j) = the replacement.
__device__ __forceinline__ double chol4_pivot(const PV& P, int col, double d, double ad, bool record) {
    if (!(d <= P.tol1 * fabs(ad)) || d < -P.tol1 * fabs(ad)) return d;
    const double dn = P.tol1 * fmax(1.0, fabs(P.tol4 * ad));
    if (record) {
        P.dcor[2 * (int64_t)col] = d;
        P.dcor[2 * (int64_t)col + 1] = dn;
        atomicAdd(&P.st->nsing, 1ull);
    }
    return dn;
}

// SPRF47 on a failing (negative) pivot: DCOR(1,j) = DCOR(2,j) = d.
__device__ __forceinline__ void chol4_fail_record(const PV& P, int col, double d) {
    P.dcor[2 * (int64_t)col] = d;
    P.dcor[2 * (int64_t)col + 1] = d;
}

// Mixed-mode inertia guard: a pivot this close to zero relative to its
// original diagonal may have its sign decided by the TF32 rounding of the
// updates that formed it.
__device__ __forceinline__ bool near_zero_pivot(const PV& P, double d, double ad) {
    return P.near_tol > 0.0 && fabs(d) < P.near_tol * fabs(ad);
}

namespace gemm {
__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(c0), "+d"(c1)
                 : "d"(a), "d"(b));
}
}  // namespace gemm

constexpr int kDG = 16;                              // columns of an elimination group
template <int V>
struct IntC {
    static constexpr int value = V;
};

// barrier of the first n warps of the CTA (barrier 1)
__device__ __forceinline__ void sync_warps(int n) { asm volatile("bar.sync 1, %0;" ::"r"(32 * n) : "memory"); }

// One 16x16 tile of a packed front: A(i, j) -= sum_{k < K} w_ik (w_jk / d_k) for
// i0 <= i < F, j0 <= j < jend, i >= j, by one warp with DMMA (2x2 tiles of 8x8,
// k ascending: DMMA chains its products in order, like a loop of multiply-adds).
// A holds the unscaled columns w, rd the reciprocal pivots.
__device__ __forceinline__ void small_tile(double* A, const double* rd, int F, int K, int i0, int j0, int jend,
                                           int lane) {
    const int fr = lane >> 2, fk = lane & 3;
    double c[2][2][2];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = i0 + 8 * a + fr, j = j0 + 8 * b + 2 * fk + h;
                c[a][b][h] = (i < F && j < jend && i >= j) ? A[pk(i, j, F)] : 0.0;
            }
    const bool vi0 = i0 + fr < F, vi1 = i0 + 8 + fr < F, vj0 = j0 + fr < F, vj1 = j0 + 8 + fr < F;
    int base = pk(0, fk, F), k = fk;                 // A[base + i] = w_ik
    for (int k4 = 0; k4 < K; k4 += 4) {
        const bool vk = k < K;
        const double r = vk ? rd[k] : 0.0;
        const double a0 = vk && vi0 ? -A[base + i0 + fr] : 0.0, a1 = vk && vi1 ? -A[base + i0 + 8 + fr] : 0.0;
        const double b0 = vk && vj0 ? A[base + j0 + fr] * r : 0.0, b1 = vk && vj1 ? A[base + j0 + 8 + fr] * r : 0.0;
        gemm::dmma(c[0][0][0], c[0][0][1], a0, b0);
        gemm::dmma(c[0][1][0], c[0][1][1], a0, b1);
        gemm::dmma(c[1][0][0], c[1][0][1], a1, b0);
        gemm::dmma(c[1][1][0], c[1][1][1], a1, b1);
        base += 4 * F - 4 * k - 10;                  // pk(0, k + 4) - pk(0, k)
        k += 4;
    }
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = i0 + 8 * a + fr, j = j0 + 8 * b + 2 * fk + h;
                if (i < F && j < jend && i >= j) A[pk(i, j, F)] = c[a][b][h];
            }
}

// The published column of an elimination step: entry j of the columns after
// the current one, for every lane of the warp.
template <int W>
__device__ __forceinline__ void read_column(const double* cb, double (&c)[kDG]) {
#pragma unroll
    for (int j = 0; j < (W + 1) / 2; ++j) {
        const double2 v = *reinterpret_cast<const double2*>(cb + 2 * j);
        c[2 * j] = v.x;
        c[2 * j + 1] = v.y;
    }
}

// Elimination of the columns c0 .. c0 + kmax - 1 of a packed front by one warp,
// without a CTA barrier: lanes 0-15 hold the group's own rows (every warp
// repeats them), and every lane one row below, 32 of them from c0 + 16 + 32 w on,
// 16 entries each in registers; the pivot goes round by a shuffle, the column
// through the warp's own shared memory cb (2 x 32).  The columns stay unscaled
// (w).  The registers move down by one each step (a[0] is always the current
// column), so that the loop over the columns is a loop and not 16 copies, which a
// kernel of one pass pays for in instruction fetches, and a step has no branch
// but the loop's (the reciprocal's is uniform): 610 clocks a step with one, about 150
// without.
// Returns the failing column or -1.
template <int PR>
__device__ __forceinline__ int small_group(const PV& P, int js, double* A, double* rd, double* dd, double* cb, int F,
                                           int c0, int kmax, int w, int sets, int lane) {
    const int fst = P.fst[js];
    const bool own = lane < kDG && c0 + lane < F;
    const int row = c0 + kDG + 32 * w + lane;
    const bool below = row < F;
    const double adr = lane < kmax ? P.adiag[fst + c0 + lane] : 0.0;
    double a[kDG], x[kDG];
#pragma unroll
    for (int j = 0; j < kDG; ++j) {
        a[j] = (own && j < kmax && j <= lane) ? A[pk(c0 + lane, c0 + j, F)] : 0.0;
        x[j] = (below && j < kmax) ? A[pk(row, c0 + j, F)] : 0.0;
    }
    if (sets > 1) sync_warps(sets);                    // all have read the own rows, which set 0 writes back
    double dmine = 1.0, rmine = 1.0;                   // lane k keeps pivot k
    double* ap = A + pk(0, c0, F);                     // the current column, row 0
    const int own_row = w == 0 && own ? c0 + lane : -1;
    double d_next = __shfl_sync(0xffffffffu, a[0], 0);
    auto step = [&](int k, auto width) -> bool {
        constexpr int W = decltype(width)::value;
        double* cbk = cb + (k & 1) * 32;
        const double a0 = a[0], x0 = x[0];
        double d = d_next;
        const double ann = __shfl_sync(0xffffffffu, a[1], (k + 1) & 31);     // the next pivot before this step
        if (PR == kPivotReplace || PR == kPivotChol4) {
            const double ad = __shfl_sync(0xffffffffu, adr, k);
            const int col = c0 + k;
            if (PR == kPivotReplace) {
                const double d0 = d;
                d = fc3_pivot(P, d0, ad);
                if (w == 0 && lane == 0) fc3_record(P, fst + col, d0, d);
            } else {
                if (pivot_fails(PR, d, ad, P.tol1)) {            // sprfc4.f:980
                    if (w == 0 && lane == 0) {
                        record_fail(P, js, col, d, ad);
                        chol4_fail_record(P, fst + col, d);
                    }
                    return false;
                }
                d = chol4_pivot(P, fst + col, d, ad, w == 0 && lane == 0);
            }
        }
        cbk[(lane - k - 1) & 31] = a0;                           // lane k + 1 + j to entry j
        const double r = recip_nr_uniform(d);
        dmine = lane == k ? d : dmine;
        rmine = lane == k ? r : rmine;
        if (own_row >= c0 + k) ap[own_row] = lane == k ? d : a0;
        if (below) ap[row] = x0;
        ap += F - (c0 + k) - 1;
        __syncwarp();
        double c[kDG];
        read_column<W>(cbk, c);
        d_next = fma(-c[0], c[0] * r, ann);                      // as lane k + 1 does below, without its shuffle
#pragma unroll
        for (int j = 0; j < W; ++j) {
            const double l = c[j] * r;
            a[j] = fma(-a0, l, a[j + 1]);
            x[j] = fma(-x0, l, x[j + 1]);
        }
        return true;
    };
    int k = 0;
    bool go = true;
#pragma unroll 1
    for (; k < min(kmax, kDG / 2) && go; ++k) go = step(k, IntC<kDG - 1>());
#pragma unroll 1
    for (; k < kmax && go; ++k) go = step(k, IntC<kDG / 2 - 1>());
    if (w == 0 && lane < kmax) {
        dd[c0 + lane] = dmine;
        rd[c0 + lane] = rmine;
    }
    if (PR == kPivotChol4) return go ? -1 : c0 + k - 1;
    if (PR == kPivotReplace || w != 0) return -1;
    // the first failing pivot (sprfc1.f:1274, sprfc2.f:1004); the steps after it
    // only computed values that are thrown away
    const unsigned m = __ballot_sync(0xffffffffu, lane < kmax && pivot_fails(PR, dmine, adr, P.tol1));
    if (!m) return -1;
    const int f = __ffs(m) - 1;
    if (lane == f) record_fail(P, js, c0 + f, dmine, adr);
    return c0 + f;
}

// The chain of S pivots and the latency of the children's loads bound a small
// front, so the columns are eliminated in groups of 16 by warps (small_group)
// after one DMMA update by everything before them, the trailing block takes
// one DMMA update at the end, and the children's data are loaded ahead.  Every
// entry takes its multiply-adds in ascending k.  One rank-1 step of all
// threads and two barriers per column before: all small fronts of 12^3 0.80
// ms, now 0.65 ms; of 512 boxes of 3^3 to 12^3 6.8 and 6.0 ms; 4^3 alone 0.42
// and 0.28 ms.
template <int PR>
__global__ void __launch_bounds__(256) k_small_front(const int32_t* nodes, PV P) {
    extern __shared__ double sh[];
    __shared__ __align__(16) double cbuf[8][64];
    __shared__ int16_t srel[2][kSmallMaxF];
    __shared__ int64_t s_rel[32], s_upd[32];
    __shared__ int s_q[32], s_ld[32];
    __shared__ int s_fail;
    if (P.st->any_fail) return;
    const int js = nodes[blockIdx.x];
    if (node_off(P, js)) return;
    const int F = P.F[js], S = P.S[js], fst = P.fst[js];
    const int kid0 = P.child_ptr[js], nkid = P.child_ptr[js + 1] - kid0;
    const int npk = F * (F + 1) / 2;
    double* A = sh;
    double* rd = sh + npk;                    // 1 / d_k of the S pivots
    double* dd = rd + F;                      // the pivots
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5;
    if (tid == 0) s_fail = F;
    // the first 32 children, last sibling first (sprfc1.f:534-584), one thread each
    auto load_kids = [&](int m0) {
        if (tid < 32 && m0 + tid < nkid) {
            const int c = P.child[kid0 + nkid - 1 - (m0 + tid)];
            s_q[tid] = P.F[c] - P.S[c];
            s_rel[tid] = P.rel_off[c];
            s_upd[tid] = P.upd_off[c];
            s_ld[tid] = P.buf_ld[c];
        }
    };
    load_kids(0);
    int bad = 0;
    for (int k = tid; k < nkid; k += blockDim.x) bad |= P.sn_bad[P.child[kid0 + k]];
    // fully-summed columns: the packed trapezoid of LNZ is the front's first SUPSZE entries
    const int supsze = F * S - (S * (S - 1)) / 2;
    const double* lnz = P.lnz + P.lnz_off[js];
    for (int i0 = tid; i0 < npk; i0 += 8 * (int)blockDim.x) {
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int i = i0 + u * (int)blockDim.x;
            v[u] = i < supsze ? lnz[i] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int i = i0 + u * (int)blockDim.x;
            if (i < npk) A[i] = v[u];
        }
    }
    if (__syncthreads_or(bad)) {              // a child failed, or depends on a failure
        if (tid == 0) P.sn_bad[js] = 1;
        return;
    }
    // extend-add: a warp takes every nwarp-th column of a child, in 32-row
    // pieces, kExt pieces at a time; the next pieces (of this child or the
    // next one) and the next child's rows are loaded while these are added
    constexpr int kExt = 8;
    struct Piece {
        int t, r0;
    };
    auto first = [&]() { return Piece{warp, warp & ~31}; };
    auto advance = [&](Piece& p, int q) {
        p.r0 += 32;
        if (p.r0 >= q) {
            p.t += nwarp;
            p.r0 = p.t & ~31;
        }
    };
    auto load = [&](int m, Piece& p, double (&u)[kExt]) {
        const int q = s_q[m], ld = s_ld[m];
        const double* U = P.arena + s_upd[m];
#pragma unroll
        for (int e = 0; e < kExt; ++e) {
            const int r = p.r0 + lane;
            u[e] = (p.t < q && r >= p.t && r < q) ? __ldcg(U + r + (int64_t)p.t * ld) : 0.0;
            advance(p, q);
        }
    };
    for (int m0 = 0; m0 < nkid; m0 += 32) {
        const int n = min(32, nkid - m0);
        if (m0) {
            __syncthreads();                   // the last child's adds are done
            load_kids(m0);
            __syncthreads();
        }
        double u[kExt];
        Piece pl = first();
        load(0, pl, u);
        if (tid < s_q[0]) srel[0][tid] = (int16_t)P.rel[s_rel[0] + tid];
        for (int m = 0; m < n; ++m) {
            const int q = s_q[m];
            const int16_t* rel = srel[m & 1];
            int next_rel = 0;
            if (m + 1 < n && tid < s_q[m + 1]) next_rel = P.rel[s_rel[m + 1] + tid];
            __syncthreads();                   // rel is there, the child before is added
            Piece pa = first();
            for (;;) {
                double un[kExt];
                const bool more = pl.t < q;
                if (more) {
                    load(m, pl, un);
                } else if (m + 1 < n) {
                    pl = first();
                    load(m + 1, pl, un);
                }
#pragma unroll
                for (int e = 0; e < kExt; ++e) {
                    const int r = pa.r0 + lane;
                    if (pa.t < q && r >= pa.t && r < q) A[pk(rel[r], rel[pa.t], F)] += u[e];
                    advance(pa, q);
                }
#pragma unroll
                for (int e = 0; e < kExt; ++e) u[e] = un[e];
                if (!more) break;
            }
            if (m + 1 < n && tid < s_q[m + 1]) srel[(m + 1) & 1][tid] = (int16_t)next_rel;
        }
    }
    __syncthreads();
    const bool ret = is_retained(P, js);       // a retained front is only assembled
    for (int c0 = 0; c0 < (ret ? 0 : S); c0 += kDG) {
        const int kmax = min(kDG, S - c0);
        if (c0 > 0) {
            for (int i0 = c0 + kDG * warp; i0 < F; i0 += kDG * nwarp) small_tile(A, rd, F, c0, i0, c0, c0 + kmax, lane);
            __syncthreads();
        }
        const int rest = F - c0 - kDG, sets = rest > 0 ? (rest + 31) / 32 : 1;
        if (warp < sets) {                        // at most 5 sets (of 8 warps), 2 (of 4) up to F = 64
            const int f = small_group<PR>(P, js, A, rd, dd, cbuf[warp], F, c0, kmax, warp, sets, lane);
            if (f >= 0 && lane == 0) s_fail = f;      // (set 0's, or every warp's the same)
        }
        __syncthreads();
        if (s_fail < F) break;
    }
    const int kend = ret ? 0 : min(S, s_fail);
    if (warp == 0) {
        // inertia and TOL(2) of the processed columns (sprfc1.f:1280-1290)
        int neg = 0, near = 0;
        double tmax = 0.0;
        for (int k = lane; k < kend; k += 32) {
            const double d = dd[k], ad = P.adiag[fst + k];
            neg += d < 0.0;
            near += near_zero_pivot(P, d, ad);
            tmax = fmax(tmax, ad / d);
        }
        for (int o = 16; o > 0; o >>= 1) {
            neg += __shfl_xor_sync(0xffffffffu, neg, o);
            near += __shfl_xor_sync(0xffffffffu, near, o);
            tmax = fmax(tmax, __shfl_xor_sync(0xffffffffu, tmax, o));
        }
        if (lane == 0) {
            P.sn_neg[js] = neg;
            if (neg) atomicAdd(&P.st->numneg, (unsigned long long)neg);
            if (near) atomicAdd(&P.st->near_piv, (unsigned long long)near);
            if (s_fail >= F) atomic_max_double(&P.st->tol2, tmax);
        }
    }
    if (s_fail < F) return;
    // write back the S columns (LNZ layout == packed layout) as L, and the pivots
    double* lnzw = P.lnz + P.lnz_off[js];
    for (int k = warp; k < S; k += nwarp) {
        const int base = pk(0, k, F);
        const double r = ret ? 1.0 : rd[k];
        for (int i = k + lane; i < F; i += 32) lnzw[base + i] = (i == k || ret) ? A[base + i] : A[base + i] * r;
    }
    if (!ret)
        for (int j = tid; j < S; j += blockDim.x) P.dvec[fst + j] = dd[j];
    const int q = F - S;
    if (q <= 0) return;
    if (!ret) {
        // the trailing (F-S)^2 block in 16x16 tiles
        const int nt = (q + kDG - 1) / kDG;
        int ti = 0, tj = warp;
        for (int t = warp; t < nt * (nt + 1) / 2; t += nwarp) {
            while (tj > ti) tj -= ++ti;
            small_tile(A, rd, F, S, S + kDG * ti, S + kDG * tj, F, lane);
            tj += nwarp;
        }
        __syncthreads();
    }
    double* U = P.arena + P.upd_off[js];
    const int ld = P.buf_ld[js];
    for (int t = warp; t < q; t += nwarp)
        for (int r = t + lane; r < q; r += 32) U[r + (int64_t)t * ld] = A[pk(S + r, S + t, F)];
}

// ---------------------------------------------------------------------------
// Large fronts
// ---------------------------------------------------------------------------

// A large front whose child failed (or depends on a failure) is skipped.
__global__ void k_poison(const Job* jobs, int64_t njobs, const int32_t* tmap, PV P) {
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= njobs) return;
    const int js = jobs[j].node;
    if (!node_off(P, js) && children_bad(P, js)) P.sn_bad[js] = 1;
}

// Extend-add into a dense column-major front: one warp per front column.
// The column is built in chunks of kAsmRows rows in shared memory: the chunk
// starts as the LNZ column (fully-summed columns) or zero, receives the
// children's update entries whose parent rows fall into it (each child's rows
// are increasing in the parent, so a per-child cursor, kept in one lane,
// advances chunk by chunk), and is written once.  Each front entry is written
// once and each child entry read once, in the same order of additions as a
// column-at-a-time scatter (deterministic, no atomics).  A column with more
// than 32 contributions (one cursor per lane) scatters into HBM instead.
constexpr int kAsmRows = 256;

__device__ __forceinline__ void asm_scatter_column(const PV& P, double* col, int j, int F, int S, const double* src,
                                                   int64_t e0, int64_t e1, int lane) {
    if (j < S) {
        int i = j + lane;
        for (; i + 96 < F; i += 128) {
            const double a0 = __ldcg(src + i), a1 = __ldcg(src + i + 32), a2 = __ldcg(src + i + 64),
                         a3 = __ldcg(src + i + 96);
            col[i] = a0;
            col[i + 32] = a1;
            col[i + 64] = a2;
            col[i + 96] = a3;
        }
        for (; i < F; i += 32) col[i] = __ldcg(src + i);
    } else {
        for (int i = j + lane; i < F; i += 32) col[i] = 0.0;
    }
    __syncwarp();
    for (int64_t e = e0; e < e1; ++e) {
        const int c = P.cchild[e], t = P.ct[e];
        const int q = P.F[c] - P.S[c];
        const int32_t* rel = P.rel + P.rel_off[c];
        const double* U = P.arena + P.upd_off[c] + (int64_t)t * P.buf_ld[c];
        for (int r = t + lane; r < q; r += 32) col[rel[r]] += U[r];
        __syncwarp();
    }
}

__global__ void __launch_bounds__(256) k_assemble(const Job* jobs, int64_t njobs, const int32_t* tmap, int64_t ntasks,
                                                  PV P) {
    __shared__ double chunk[8][kAsmRows];
    if (P.st->any_fail) return;
    const int lane = threadIdx.x & 31;
    const int64_t task = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    if (task >= ntasks) return;
    const Job& jb = job_of(jobs, njobs, tmap, task);
    const int js = jb.node;
    if (P.sn_bad[js] || node_off(P, js)) return;
    const int j = jb.c0 + (int)(task - jb.task0);
    const int F = P.F[js], S = P.S[js];
    const int ld = P.buf_ld[js];
    double* col = P.arena + P.buf_off[js] + (int64_t)j * ld;
    const double* src = (j < S) ? P.lnz + P.lnz_off[js] + lnz_col(j, F) - j : nullptr;
    const int64_t e0 = P.cptr[P.rbase[js] + j], e1 = P.cptr[P.rbase[js] + j + 1];
    const int ne = (int)(e1 - e0);
    if (ne > 32) {
        asm_scatter_column(P, col, j, F, S, src, e0, e1, lane);
        return;
    }
    // lane k holds contribution k: child, its update column, rows, cursor
    int my_c = 0, my_t = 0, my_q = 0, cur = 0;
    if (lane < ne) {
        my_c = P.cchild[e0 + lane];
        my_t = P.ct[e0 + lane];
        my_q = P.F[my_c] - P.S[my_c];
        cur = my_t;
    }
    double* acc = chunk[threadIdx.x >> 5];
    for (int lo = j; lo < F; lo += kAsmRows) {
        const int n = min(kAsmRows, F - lo), hi = lo + n;
        for (int i = lane; i < n; i += 32) acc[i] = src ? __ldcg(src + lo + i) : 0.0;
        __syncwarp();
        for (int k = 0; k < ne; ++k) {
            const int c = __shfl_sync(0xffffffffu, my_c, k);
            const int t = __shfl_sync(0xffffffffu, my_t, k);
            const int q = __shfl_sync(0xffffffffu, my_q, k);
            int r = __shfl_sync(0xffffffffu, cur, k);
            const int32_t* rel = P.rel + P.rel_off[c];
            const double* U = P.arena + P.upd_off[c] + (int64_t)t * P.buf_ld[c];
            for (;;) {
                // four 32-row steps with their loads first; the rows inside
                // [lo, hi) form a prefix (the parent rows increase)
                int ri[4];
                double u[4];
#pragma unroll
                for (int st = 0; st < 4; ++st) {
                    const int rr = r + 32 * st + lane;
                    ri[st] = rr < q ? __ldg(rel + rr) : 0x7fffffff;
                    u[st] = rr < q ? __ldcg(U + rr) : 0.0;
                }
                bool more = true;
#pragma unroll
                for (int st = 0; st < 4; ++st) {
                    if (!more) break;
                    const bool in = ri[st] < hi;
                    if (in) acc[ri[st] - lo] += u[st];
                    const unsigned m = __ballot_sync(0xffffffffu, in);
                    r += __popc(m);
                    more = (m == 0xffffffffu);
                }
                if (!more) break;
            }
            if (lane == k) cur = r;
            __syncwarp();
        }
        for (int i = lane; i < n; i += 32) col[lo + i] = acc[i];
        __syncwarp();
    }
}

// LDL' of one nb x nb diagonal block, pivot test / inertia / TOL(2) as
// SPRF17 (sprfc1.f:1272-1294), and X = L11^-1 (unit lower) for the panel TRSM
// and the solves.  One CTA per block, so a chain of kNB dependent pivots
// bounds it: reciprocal, scaling, update, next pivot.  The block goes in eight
// groups of 8 columns.  A group's columns are eliminated by up to three
// warps without a CTA barrier: a lane holds one row's 8 entries in registers,
// lanes 0-7 the group's own rows (every warp repeats them) and lanes 8-31 24
// rows below; the pivot and the unscaled column (a_ij -= a_ik * a_jk / d_k) go
// round by shuffles, the column's ahead of the reciprocal.  The columns after the
// group are updated with DMMA tiles (K = 8), up to four at a time per warp: a
// DMMA takes some 130 clocks to its result, a multiply-add of one warp 8.
// The next pivot comes from the values before the step, in every lane, so that
// no shuffle is on the pivots' chain.
// The inverse goes by doubling (X21 = -X22 (L21 X11)) with DMMA; the idle warps
// form what is final of it, and write finished columns of L, beside the next
// groups' eliminations: after the last group 3 us are left of 5.
// Every entry takes its multiply-adds in ascending k (DMMA chains them in that
// order), so the factors do not depend on the grouping.  All blocks of a 32^3
// box by themselves: one barrier a column 15.0 ms, groups of 16 with the column
// through shared memory 10.5 ms, this 8.
constexpr int kD8 = 8;                               // columns of a group
constexpr int kDPanLd = kD8 + 1;

// one group's elimination by one warp: rows below in set w (rows
// c0 + 8 + 24 w ..), kmax columns; returns the failing column for the rule that
// stops at once (kPivotChol4), or -1
template <int PR>
__device__ __forceinline__ int diag_group(const PV& P, int js, int k0, int c0, int kmax, int w, int sets, int lane, int nb,
                                          double (*A)[kNB + 1], double (*Wp)[kDPanLd], double* dd, double* rdv,
                                          const double* adv) {
    const int fst = P.fst[js];
    const bool own = lane < kD8;
    const int row = own ? c0 + lane : c0 + 24 * w + lane;        // c0 + 8 + 24 w + (lane - 8)
    double a[kD8];
#pragma unroll
    for (int j = 0; j < kD8; ++j) a[j] = (row < nb && row >= c0 + j) ? A[row][c0 + j] : 0.0;
    if (sets > 1) sync_warps(sets);                    // all have read the own rows, which set 0 writes
    double dmine = 1.0, rmine = 1.0;                   // lane k keeps pivot k
    const bool keep = row < nb && (!own || w == 0);
    double* ap = &A[keep ? row : 0][c0];
    const bool below = !own && row < nb;
    double* wp = &Wp[below ? row : kD8][0];
    const int k_row = !keep ? -1 : own ? lane : kD8;   // columns k < k_row of this lane's row are L
    int k = 0;
    bool go = true;
    double d_next = __shfl_sync(0xffffffffu, a[0], 0);
    // the registers move down by one each step (a[0] is always the current
    // column): one copy of the step in the instruction stream
#pragma unroll 1
    for (; k < kmax && go; ++k) {
        const double a0 = a[0];
        double d = d_next;
        double c[kD8 - 1];                             // the column below the pivot
#pragma unroll
        for (int j = 0; j < kD8 - 1; ++j) c[j] = __shfl_sync(0xffffffffu, a0, k + 1 + j);
        const double ann = __shfl_sync(0xffffffffu, a[1], k + 1);      // the next pivot before this step
        if (PR == kPivotReplace) {
            const double d0 = d;
            d = fc3_pivot(P, d0, adv[c0 + k]);
            if (w == 0 && lane == 0) fc3_record(P, fst + k0 + c0 + k, d0, d);
        }
        if (PR == kPivotChol4) {
            // records replacements while it goes, so it stops at a failing pivot
            const int col = c0 + k;
            if (pivot_fails(PR, d, adv[col], P.tol1)) {
                if (w == 0 && lane == 0) {
                    record_fail(P, js, k0 + col, d, adv[col]);
                    chol4_fail_record(P, fst + k0 + col, d);
                }
                go = false;
                continue;
            }
            d = chol4_pivot(P, fst + k0 + col, d, adv[col], w == 0 && lane == 0);
        }
        const double rd = recip_nr_uniform(d);
        const double l = a0 * rd;
        d_next = fma(-(c[0] * rd), c[0], ann);         // as lane k + 1 does below, without its shuffle
#pragma unroll
        for (int j = 0; j < kD8 - 1; ++j) a[j] = fma(-l, c[j], a[j + 1]);
        dmine = lane == k ? d : dmine;
        rmine = lane == k ? rd : rmine;
        if (k < k_row) ap[k] = l;
        if (below) wp[k] = a0;
    }
    if (w == 0 && lane < kmax) {
        dd[c0 + lane] = dmine;
        rdv[c0 + lane] = rmine;
    }
    return go ? -1 : c0 + k - 1;
}

// one doubling pass of the inverse inside a group, by one warp: the pairs of
// blocks of order B; T = L21 X11 through t
template <int B>
__device__ __forceinline__ void diag_invert_pass(double (*A)[kNB + 1], double* t, int c0, int nb, int lane) {
    constexpr int BB = B * B, TOT = kD8 / 2 * B;
    static_assert(TOT <= 32, "one element a lane");
    const int bs = c0 + lane / BB * 2 * B, i = lane % BB / B, j = lane % B;
    if (lane < TOT) {
        double v = 0.0;
        if (bs + B + i < nb) {
            v = A[bs + B + i][bs + j];                                     // X11[j][j] = 1
#pragma unroll
            for (int m = 1; m < B; ++m) {
                const double f = fma(A[bs + B + i][bs + m], A[bs + j][bs + m], v);
                v = m > j ? f : v;
            }
        }
        t[lane] = v;
    }
    __syncwarp();
    if (lane < TOT) {
        double v = t[lane];                                                // X22[i][i] = 1
#pragma unroll
        for (int m = 0; m + 1 < B; ++m) {
            const double f = fma(A[bs + B + m][bs + B + i], t[lane / BB * BB + m * B + j], v);
            v = m < i ? f : v;
        }
        A[bs + j][bs + B + i] = -v;
    }
    __syncwarp();
}

// inverse of the unit-lower kD8 x kD8 block at c0 by one warp: doubling from
// order 1 (X21 = -X22 (L21 X11)); X[i][j] goes to A[c0 + j][c0 + i] (the free
// upper triangle)
__device__ __forceinline__ void diag_group_inverse(double (*A)[kNB + 1], double* t, int c0, int nb, int lane) {
    diag_invert_pass<1>(A, t, c0, nb, lane);
    diag_invert_pass<2>(A, t, c0, nb, lane);
    diag_invert_pass<4>(A, t, c0, nb, lane);
}

// A doubling step of the inverse with DMMA, X21 = -X22 (L21 X11) for the pair of
// blocks of order B at bs, in its two products: T = L21 X11, then X21.  A warp
// takes the 8 x 8 tiles w, w + NW, .., up to NQ of them side by side.
template <int B, int NW, int NQ>
__device__ __forceinline__ void diag_pair_t(double (*A)[kNB + 1], double* T, int bs, int nb, int w, int lane) {
    constexpr int TB = B / 8, LDT = B + 4;
    static_assert(NW * NQ == TB * TB, "every tile once");
    const int fr = lane >> 2, fk = lane & 3;
    double c[NQ][2];
#pragma unroll
    for (int q = 0; q < NQ; ++q) c[q][0] = c[q][1] = 0.0;
#pragma unroll
    for (int m0 = 0; m0 < B; m0 += 4)                      // X11[m][j] = 0 for m < j, 1 for m = j
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const int t = w + NW * q, i0 = t / TB * 8, j0 = t % TB * 8;
            const int gi = bs + B + i0 + fr, j = j0 + fr, m = m0 + fk;
            const double xv = A[bs + j][bs + m], lv = A[gi][bs + m];
            gemm::dmma(c[q][0], c[q][1], gi < nb ? lv : 0.0, m > j ? xv : m == j ? 1.0 : 0.0);
        }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const int t = w + NW * q, i0 = t / TB * 8, j0 = t % TB * 8;
        double* to = T + (i0 + fr) * LDT + j0 + 2 * fk;
        to[0] = c[q][0];
        to[1] = c[q][1];
    }
}

template <int B, int NW, int NQ>
__device__ __forceinline__ void diag_pair_x(double (*A)[kNB + 1], const double* T, int bs, int w, int lane) {
    constexpr int TB = B / 8, LDT = B + 4;
    const int fr = lane >> 2, fk = lane & 3;
    double c[NQ][2];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {                         // X22[i][i] = 1
        const int t = w + NW * q, i0 = t / TB * 8, j0 = t % TB * 8;
        const double* to = T + (i0 + fr) * LDT + j0 + 2 * fk;
        c[q][0] = to[0];
        c[q][1] = to[1];
    }
#pragma unroll
    for (int m0 = 0; m0 < B; m0 += 4)                      // X22[i][m] = 0 for m > i
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const int t = w + NW * q, i0 = t / TB * 8, j0 = t % TB * 8;
            const int i = i0 + fr, gb = bs + B, m = m0 + fk;
            const double xv = A[gb + m][gb + i];
            gemm::dmma(c[q][0], c[q][1], m < i ? xv : 0.0, T[m * LDT + j0 + fr]);
        }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const int t = w + NW * q, i0 = t / TB * 8, j0 = t % TB * 8;
        const int jc = bs + j0 + 2 * fk, gi = bs + B + i0 + fr;
        A[jc][gi] = -c[q][0];
        A[jc + 1][gi] = -c[q][1];
    }
}

// both products by one warp
template <int B>
__device__ __forceinline__ void diag_pair(double (*A)[kNB + 1], double* T, int bs, int nb, int lane) {
    diag_pair_t<B, 1, B * B / 64>(A, T, bs, nb, 0, lane);
    __syncwarp();
    diag_pair_x<B, 1, B * B / 64>(A, T, bs, 0, lane);
    __syncwarp();
}

// what a diagonal block's elimination keeps in shared memory beside A and pan
struct DiagShared {
    double w[(kNB - kD8) * kDPanLd];        // W of a group's rows below
    double t8[2][8 * 12], t16[16 * 20], t32[32 * 36], tinv[kD8 * kD8 / 4];
    double rdv[kNB], dd[kNB], adv[kNB];
    int fail;
};

// columns c0 .. c0 + n - 1 of L and D to the front, by nw warps; block: where the block starts
__device__ __forceinline__ void diag_store(double* block, int ld, int c0, int n, int nb, double (*A)[kNB + 1],
                                           const double* dd, int w, int nw, int lane) {
    for (int j = c0 + w; j < c0 + n; j += nw) {
        if (j + lane < nb) block[j + lane + (int64_t)j * ld] = lane == 0 ? dd[j] : A[j + lane][j];
        if (j + lane + 32 < nb) block[j + lane + 32 + (int64_t)j * ld] = A[j + lane + 32][j];
    }
}

// 32 x 32 of the inverse to lv at (i0, j0), by nw warps
__device__ __forceinline__ void diag_store_x(double* lv, int i0, int j0, int nb, double (*A)[kNB + 1], int w, int nw,
                                             int lane) {
    const int i = i0 + lane;
#pragma unroll 8
    for (int j = j0 + w; j < j0 + 32; j += nw)
        lv[i + j * kNB] = (i < nb && j < nb) ? (i > j ? A[j][i] : (i == j ? 1.0 : 0.0)) : 0.0;
}

// The rows [k0 + 64, next_end) of panel k0 transposed into the front's free upper
// triangle, for k_chain; by 96 threads
__device__ __forceinline__ void diag_copy_next(double* front, int ld, int k0, int nb, int next_end, int t) {
    const int n = next_end - (k0 + kNB);
    const double* from = front + k0 + kNB + (int64_t)k0 * ld;
    double* to = front + k0 + (int64_t)(k0 + kNB) * ld;
    for (int e0 = t; e0 < kNB * kNB && n > 0; e0 += 8 * 96) {
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int e = e0 + 96 * u, j = e & (kNB - 1), m = e >> 6;
            v[u] = j < n && m < nb ? __ldcg(from + j + (int64_t)m * ld) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int e = e0 + 96 * u, j = e & (kNB - 1), m = e >> 6;
            if (j < n && m < nb) to[m + (int64_t)j * ld] = v[u];
        }
    }
}

// The block in A (lower, zero elsewhere), its a_jj in S.adv, S.fail = kNB; all
// synchronised.  next_end: with Copy, the end of the next panel's rows.
template <int PR, bool Copy>
__device__ __forceinline__ void diag_block(const PV& P, int js, int k0, int nb, double* front, int ld, int next_end,
                                           double (*A)[kNB + 1], DiagShared& S) {
    const int fst = P.fst[js];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // W's rows are 8 .. 63: a group's own rows are not among them
    double(*Wp)[kDPanLd] = reinterpret_cast<double(*)[kDPanLd]>(S.w) - kD8;
    double* block = front + k0 + (int64_t)k0 * ld;
    double* lv = P.linv + P.linv_off[js] + (int64_t)(k0 / kNB) * kNB * kNB;
    const bool full = nb == kNB;
    int failed = -1;
#pragma unroll 1
    for (int c0 = 0; c0 < nb; c0 += kD8) {
        const int kmax = min(kD8, nb - c0), rest = nb - c0 - kD8;         // rest: rows below the group
        const int sets = rest > 0 ? (rest + 23) / 24 : 1;
        if (warp < sets) {
            const int f = diag_group<PR>(P, js, k0, c0, kmax, warp, sets, lane, nb, A, Wp, S.dd, S.rdv, S.adv);
            if (PR == kPivotChol4 && f >= 0 && lane == 0) S.fail = f;     // every warp finds the same column
        } else if (c0 > 0) {
            // beside the group, what is final of the ones before: their inverses (of a
            // full block as far as they go, as the schedule below), L to the front
            const int g = c0 / kD8;
            if (warp == 4) {
                diag_group_inverse(A, S.tinv, c0 - kD8, nb, lane);
                if (full && g == 7) diag_pair_t<8, 1, 1>(A, S.t8[0], 48, nb, 0, lane);
            } else if (warp == 5) {
                if (full && g == 3) diag_pair<8>(A, S.t8[1], 0, nb, lane);
                if (full && g == 5) diag_pair<8>(A, S.t8[1], 16, nb, lane);
                if (full && g == 6) diag_pair<16>(A, S.t16, 0, nb, lane);
                if (full && g == 7) {
                    diag_pair<8>(A, S.t8[1], 32, nb, lane);
                    diag_pair_t<16, 1, 4>(A, S.t16, 32, nb, 0, lane);
                }
            } else if (warp >= 6) {
                diag_store(block, ld, c0 - kD8, kD8, nb, A, S.dd, warp - 6, 2, lane);
            } else if (full && g == 7) {
                if (warp == 3) diag_store_x(lv, 0, 0, nb, A, 0, 1, lane);
            } else if (full && g == 4 && warp == 3) {
                for (int j = 32; j < kNB; ++j) lv[lane + j * kNB] = 0.0;
            }
            if (full && g == 7 && (warp & 2)) diag_pair_t<32, 4, 4>(A, S.t32, 0, nb, (warp >> 2) * 2 + (warp & 1), lane);
        }
        if (Copy && c0 == 0 && warp >= 5) diag_copy_next(front, ld, k0, nb, next_end, tid - 160);
        __syncthreads();
        if (PR == kPivotChol4 && S.fail < kNB) {
            failed = S.fail;
            break;
        }
        if (rest <= 0) continue;
        // A[i][j] -= sum_k L[i][k] W[j][k] on the lower 8x8 tiles of what follows:
        // up to 28, tiles warp, warp + 8, .. side by side
        const int nt = (rest + 7) >> 3, ntile = nt * (nt + 1) / 2, r0 = c0 + kD8;
        const int fr = lane >> 2, fk = lane & 3;
        double c[4][2], fa[4][2], fb[4][2];
        int ci[4], cj[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int t = warp + 8 * q;
            const int ti = (t >= 1) + (t >= 3) + (t >= 6) + (t >= 10) + (t >= 15) + (t >= 21) + (t >= 28);
            const int tj = t - ti * (ti + 1) / 2;
            const int i = r0 + 8 * ti + fr, j = r0 + 8 * tj + fr;
            const bool on = t < ntile;
            ci[q] = on && i < nb ? i : -1;
            cj[q] = r0 + 8 * tj + 2 * fk;
            const bool vj = on && j < nb;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                c[q][h] = ci[q] >= cj[q] + h ? A[ci[q]][cj[q] + h] : 0.0;
                fa[q][h] = ci[q] >= 0 ? -A[ci[q]][c0 + 4 * h + fk] : 0.0;
                fb[q][h] = vj ? Wp[j][4 * h + fk] : 0.0;
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (warp + 8 * q < ntile) gemm::dmma(c[q][0], c[q][1], fa[q][h], fb[q][h]);
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (ci[q] >= cj[q] + h) A[ci[q]][cj[q] + h] = c[q][h];
        __syncthreads();
    }
    // the first failing pivot (sprfc1.f:1274-1279), for the rules tested here (the
    // steps after a failure only computed values that are thrown away)
    if (PR == kPivotLDL || PR == kPivotChol) {
        if (tid < 32) {
            int f = nb;
            for (int k = tid; k < nb; k += 32)
                if (pivot_fails(PR, S.dd[k], S.adv[k], P.tol1)) f = min(f, k);
            for (int o = 16; o > 0; o >>= 1) f = min(f, __shfl_xor_sync(0xffffffffu, f, o));
            if (tid == 0) {
                if (f < nb) record_fail(P, js, k0 + f, S.dd[f], S.adv[f]);
                S.fail = f;
            }
        }
        __syncthreads();
        failed = S.fail < nb ? S.fail : -1;
    }
    if (warp == 0) {
        // inertia and TOL(2) of the processed columns (sprfc1.f:1280-1290)
        const int kend = failed < 0 ? nb : failed;
        int neg = 0, near = 0;
        double tmax = 0.0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int k = lane + 32 * h;
            const double d = k < kend ? S.dd[k] : 1.0, ad = k < kend ? S.adv[k] : 0.0;
            neg += __popc(__ballot_sync(0xffffffffu, d < 0.0));
            near += __popc(__ballot_sync(0xffffffffu, k < kend && near_zero_pivot(P, d, ad)));
            tmax = fmax(tmax, ad / d);
        }
        for (int o = 16; o > 0; o >>= 1) tmax = fmax(tmax, __shfl_xor_sync(0xffffffffu, tmax, o));
        if (lane == 0) {
            P.sn_neg[js] += neg;
            if (neg) atomicAdd(&P.st->numneg, (unsigned long long)neg);
            if (near) atomicAdd(&P.st->near_piv, (unsigned long long)near);
            if (failed < 0) atomic_max_double(&P.st->tol2, tmax);
        }
    }
    if (failed >= 0) return;
    // the last group's inverse and the pairs that wait for it, the pivots, and the
    // last group of L and D, by different warps
    const int cl = (nb - 1) / kD8 * kD8;
    if (warp == 4) {
        diag_group_inverse(A, S.tinv, cl, nb, lane);
        if (full) {
            diag_pair_x<8, 1, 1>(A, S.t8[0], 48, 0, lane);
            __syncwarp();
            diag_pair_x<16, 1, 4>(A, S.t16, 32, 0, lane);
        } else {
            for (int bs = 0; bs + 8 < nb; bs += 16) diag_pair<8>(A, S.t8[0], bs, nb, lane);
            for (int bs = 0; bs + 16 < nb; bs += 32) diag_pair<16>(A, S.t16, bs, nb, lane);
        }
    } else if (warp == 5) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int e = lane + 32 * h;
            if (e < nb) {
                const double d = S.dd[e];
                P.dvec[fst + k0 + e] = d;
                if (P.sqd) {
                    const double s = sqrt(fabs(d)), er = s > 0.0 ? fma(-s, s, fabs(d)) / (2.0 * s) : 0.0;
                    P.sqd[2 * (int64_t)(fst + k0 + e)] = copysign(s, d);
                    P.sqd[2 * (int64_t)(fst + k0 + e) + 1] = copysign(1.0, d) * er;
                }
            }
        }
    } else if (warp >= 6) {
        diag_store(block, ld, cl, nb - cl, nb, A, S.dd, warp - 6, 2, lane);
    }
    __syncthreads();
    if (nb > 32) {
        if (!full) {
            diag_pair_t<32, 8, 2>(A, S.t32, 0, nb, warp, lane);
            __syncthreads();
        }
        diag_pair_x<32, 8, 2>(A, S.t32, 0, warp, lane);
        __syncthreads();
    }
    if (!full) {
        diag_store_x(lv, 0, 0, nb, A, warp, 8, lane);
        diag_store_x(lv, 0, 32, nb, A, warp, 8, lane);
    }
    diag_store_x(lv, 32, 0, nb, A, warp, 8, lane);
    diag_store_x(lv, 32, 32, nb, A, warp, 8, lane);
}

constexpr size_t kDiagSmem = sizeof(double) * kNB * (kNB + 1) + sizeof(DiagShared);

// next: with it, k_chain follows, and takes the next panel's rows of this one
// from the upper triangle
template <int PR>
__global__ void __launch_bounds__(256) k_diag(const Job* jobs, PV P, int next) {
    extern __shared__ __align__(16) double dsh[];
    double(*A)[kNB + 1] = reinterpret_cast<double(*)[kNB + 1]>(dsh);    // L (lower, d on the diagonal), X transposed above
    DiagShared& S = *reinterpret_cast<DiagShared*>(dsh + kNB * (kNB + 1));
    if (P.st->any_fail) return;
    const Job& jb = jobs[blockIdx.x];
    const int js = jb.node, k0 = jb.k_lo, nb = jb.k_hi - jb.k_lo;
    if (P.sn_bad[js] || node_off(P, js)) return;
    const int ld = P.buf_ld[js], fst = P.fst[js];
    double* front = P.arena + P.buf_off[js];
    const int tid = threadIdx.x;
    {
        double v[kNB * kNB / 256];
#pragma unroll
        for (int q = 0; q < kNB * kNB / 256; ++q) {
            const int i = tid & (kNB - 1), j = (tid >> 6) + 4 * q;
            v[q] = (i >= j && i < nb) ? __ldcg(front + (int64_t)(k0 + i) + (int64_t)(k0 + j) * ld) : 0.0;
        }
        if (tid < nb) S.adv[tid] = __ldcg(P.adiag + fst + k0 + tid);
        if (tid == 0) S.fail = kNB;
#pragma unroll
        for (int q = 0; q < kNB * kNB / 256; ++q) A[tid & (kNB - 1)][(tid >> 6) + 4 * q] = v[q];
    }
    __syncthreads();
    const int next_end = next ? min(k0 + 2 * kNB, P.S[js]) : 0;
    diag_block<PR, true>(P, js, k0, nb, front, ld, next_end, A, S);
}

// Panel TRSM as a product with the stored inverse: for a 64-row block of the
// rows below the diagonal block, W = A21 X' (X = L11^-1), L21 = W D^-1.
// 128 threads = 2x2 warps of 32x32 DMMA tiles; the block is read completely
// into shared memory before it is overwritten, so the update is in place.
constexpr int kTrsmLds = kNB + 4;
constexpr size_t kTrsmSmem = sizeof(double) * (2 * (size_t)kNB * kTrsmLds + kNB);

__global__ void __launch_bounds__(128) k_trsm(const Job* jobs, int64_t njobs, const int32_t* tmap, PV P) {
    extern __shared__ double tsh[];
    double(*As)[kTrsmLds] = reinterpret_cast<double(*)[kTrsmLds]>(tsh);              // As[m][i]
    double(*Xs)[kTrsmLds] = reinterpret_cast<double(*)[kTrsmLds]>(tsh + kNB * kTrsmLds);  // Xs[m][c] = X[c][m]
    double* rd = tsh + 2 * kNB * kTrsmLds;
    if (P.st->any_fail) return;
    const int64_t task = blockIdx.x;
    const Job& jb = job_of(jobs, njobs, tmap, task);
    const int js = jb.node, k0 = jb.k_lo, nb = jb.k_hi - jb.k_lo;
    if (P.sn_bad[js] || node_off(P, js)) return;
    const int F = P.F[js], ld = P.buf_ld[js];
    const int r0 = jb.c0 + (int)(task - jb.task0) * kTRSMRows;
    double* front = P.arena + P.buf_off[js];
    const double* lv = P.linv + P.linv_off[js] + (int64_t)(k0 / kNB) * kNB * kNB;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // loads in groups of 8 per thread before their shared-memory stores
    for (int e0 = 0; e0 < kNB * kNB; e0 += 8 * 128) {
        double av[8], xv[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int e = e0 + u * 128 + tid;
            const int i = e % kNB, m = e / kNB;
            av[u] = (m < nb && r0 + i < F) ? __ldcg(front + (int64_t)(r0 + i) + (int64_t)(k0 + m) * ld) : 0.0;
            xv[u] = __ldcg(lv + i + m * kNB);          // X[i][m]: row i (output column), col m
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int e = e0 + u * 128 + tid;
            As[e / kNB][e % kNB] = av[u];
            Xs[e / kNB][e % kNB] = xv[u];
        }
    }
    for (int c = tid; c < kNB; c += blockDim.x)
        rd[c] = (c < nb) ? 1.0 / front[(int64_t)(k0 + c) * (ld + 1)] : 0.0;
    __syncthreads();
    const int wm = (warp & 1) * 32, wn = (warp >> 1) * 32;
    double acc[4][4][2];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
#pragma unroll 4
    for (int k4 = 0; k4 < kNB; k4 += 4) {
        const int kk = k4 + (lane & 3);
        double av[4], bv[4];
#pragma unroll
        for (int mi = 0; mi < 4; ++mi) av[mi] = As[kk][wm + mi * 8 + (lane >> 2)];
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) bv[ni] = Xs[kk][wn + ni * 8 + (lane >> 2)];
#pragma unroll
        for (int mi = 0; mi < 4; ++mi)
#pragma unroll
            for (int ni = 0; ni < 4; ++ni) gemm::dmma(acc[mi][ni][0], acc[mi][ni][1], av[mi], bv[ni]);
    }
#pragma unroll
    for (int mi = 0; mi < 4; ++mi) {
        const int r = r0 + wm + mi * 8 + (lane >> 2);
        if (r >= F) continue;
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c = wn + ni * 8 + 2 * (lane & 3) + h;
                if (c < nb) front[(int64_t)r + (int64_t)(k0 + c) * ld] = acc[mi][ni][h] * rd[c];
            }
    }
}

// A step of the panel chain inside a super-panel, panel p = [k0, k0 + 64) whose
// diagonal block is done: the panel's TRSM, the update of the next panel's
// columns by panels p - 1 and p (the columns after them get panel p beside the
// next step, k_gemm), and the next diagonal block.  Separate launches of the
// three before put two launches and two reads of the next panel on the chain, which
// bounds fronts of a few thousand rows.
// A CTA has 64 rows (the first CTA the next diagonal block's), and each
// forms the next panel's rows of L itself, from the copy of them that the step
// before left in the front's upper triangle (in place they are being replaced by
// the first CTA): one product of 64 x 64 x 64 more instead of a grid-wide wait.
// Products of 64 columns at a time and in the separate kernels' order: the same
// bits.  Fronts that end with panel p only take the TRSM.  The diagonal block's CTA
// takes its products' lower tiles and X's lower triangle alone; the block's own
// elimination is two thirds of its time.  Separate launches before: 20^3 factor 10.6
// -> 9.7 ms, 32^3 33.6 -> 30.8 ms, 48^3 250 -> 245 ms.
constexpr size_t kChainSmem = sizeof(double) * (3 * (size_t)kNB * kTrsmLds + 4 * kNB);
static_assert(sizeof(DiagShared) <= sizeof(double) * kNB * kTrsmLds, "in the inverse's buffer");

namespace gemm {
__device__ __forceinline__ void cp_async16(double* dst, const double* src, int bytes) {
    const unsigned saddr = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(saddr), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void cp_async8(double* dst, const double* src, bool valid) {
    const unsigned saddr = (unsigned)__cvta_generic_to_shared(dst);
    const int sz = valid ? 8 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(saddr), "l"(src), "r"(sz));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }
}  // namespace gemm

// 64 x 64 doubles, rows contiguous in memory, to buf[col][row]; rows x cols of them
// are there.  even: src is 16-byte aligned (ld is a multiple of four)
__device__ __forceinline__ void chain_load(double (*buf)[kTrsmLds], const double* src, int ld, int rows, int cols, bool even) {
    if (even) {
#pragma unroll
        for (int u = 0; u < kNB * kNB / 512; ++u) {
            const int e = threadIdx.x + 256 * u, i = 2 * (e & 31), m = e >> 5;
            const int n = m < cols ? max(0, min(2, rows - i)) : 0;
            gemm::cp_async16(&buf[m][i], n > 0 ? src + i + (int64_t)m * ld : src, 8 * n);
        }
    } else {
#pragma unroll 4
        for (int u = 0; u < kNB * kNB / 256; ++u) {
            const int e = threadIdx.x + 256 * u, i = e & 63, m = e >> 6;
            const bool in = m < cols && i < rows;
            gemm::cp_async8(&buf[m][i], in ? src + i + (int64_t)m * ld : src, in);
        }
    }
}

// the same from the transpose: element (i, m) at src[m + i * ld]
__device__ __forceinline__ void chain_load_t(double (*buf)[kTrsmLds], const double* src, int ld, int rows) {
#pragma unroll
    for (int u = 0; u < kNB * kNB / 256; ++u) {
        const int e = threadIdx.x + 256 * u;
        const int m = (e & 3) + 4 * (e >> 5 & 15), i = (e >> 2 & 7) + 8 * (e >> 9);
        gemm::cp_async8(&buf[m][i], i < rows ? src + m + (int64_t)i * ld : src, i < rows);
    }
}

// acc = sum_k (a[k][i] d[k]) b[k][j] (without D: a[k][i] b[k][j]) by DMMA, a warp 32 x 16
template <bool D>
__device__ __forceinline__ void chain_product(double (&acc)[4][2][2], const double (*a)[kTrsmLds], const double (*b)[kTrsmLds],
                                              const double* d, int wm, int wn, int lane, int kend) {
#pragma unroll
    for (int mi = 0; mi < 4; ++mi)
#pragma unroll
        for (int ni = 0; ni < 2; ++ni) acc[mi][ni][0] = acc[mi][ni][1] = 0.0;
#pragma unroll 4
    for (int k4 = 0; k4 < kend; k4 += 4) {
        const int kk = k4 + (lane & 3);
        double av[4], bv[2];
#pragma unroll
        for (int mi = 0; mi < 4; ++mi) av[mi] = D ? a[kk][wm + mi * 8 + (lane >> 2)] * d[kk] : a[kk][wm + mi * 8 + (lane >> 2)];
#pragma unroll
        for (int ni = 0; ni < 2; ++ni) bv[ni] = b[kk][wn + ni * 8 + (lane >> 2)];
#pragma unroll
        for (int mi = 0; mi < 4; ++mi)
#pragma unroll
            for (int ni = 0; ni < 2; ++ni) gemm::dmma(acc[mi][ni][0], acc[mi][ni][1], av[mi], bv[ni]);
    }
}

// The 36 lower 8 x 8 tiles of 64 x 64: row tiles p and 7 - p have nine, and go to
// warps p and p + 4, five and four of them (one scheduler's two warps: nine)
struct ChainTiles {
    int i[5], j[5], n;
    __device__ __forceinline__ explicit ChainTiles(int warp) {
        const int p = warp & 3, h = warp >> 2;
        n = 5 - h;
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            const int t = min(2 * q + h, 8);
            i[q] = t <= p ? p : 7 - p;
            j[q] = t <= p ? t : t - p - 1;
        }
    }
    __device__ __forceinline__ bool on(int q) const { return q < n; }
};

// c -= sum_k (a[k][i] d[k]) a[k][j] on them
__device__ __forceinline__ void chain_lower(double (&c)[5][2], const double (*a)[kTrsmLds], const double* d,
                                            const ChainTiles& tl, int lane) {
    double acc[5][2];
#pragma unroll
    for (int q = 0; q < 5; ++q) acc[q][0] = acc[q][1] = 0.0;
#pragma unroll 4
    for (int k4 = 0; k4 < kNB; k4 += 4) {
        const int kk = k4 + (lane & 3);
        const double dv = d[kk];
        double av[5], bv[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            av[q] = a[kk][8 * tl.i[q] + (lane >> 2)] * dv;
            bv[q] = a[kk][8 * tl.j[q] + (lane >> 2)];
        }
#pragma unroll
        for (int q = 0; q < 5; ++q)
            if (q < 4 || tl.on(q)) gemm::dmma(acc[q][0], acc[q][1], av[q], bv[q]);
    }
#pragma unroll
    for (int q = 0; q < 5; ++q)
#pragma unroll
        for (int h = 0; h < 2; ++h) c[q][h] -= acc[q][h];
}

template <int PR>
__global__ void __launch_bounds__(256, 2) k_chain(const Job* jobs, int64_t njobs, const int32_t* tmap, PV P) {
    extern __shared__ __align__(16) double csh[];
    using Buf = double(*)[kTrsmLds];
    const Buf B0 = reinterpret_cast<Buf>(csh), B1 = B0 + kNB, B2 = B1 + kNB;
    double* dp = csh + 3 * kNB * kTrsmLds;                  // D of panel p - 1
    double* dk = dp + kNB;                                  // and of p
    double* rd = dk + kNB;                                  // 1 / D of p
    double* adv = rd + kNB;
    DiagShared& S = *reinterpret_cast<DiagShared*>(&B2[0][0]);             // once X is read
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int any_fail = P.st->any_fail;
    const int64_t task = blockIdx.x;
    const Job& jb = job_of(jobs, njobs, tmap, task);
    const int js = jb.node, k0 = jb.k_lo, nb = jb.k_hi - jb.k_lo, c0 = jb.c0;
    const int F = P.F[js], ld = P.buf_ld[js], sn_s = P.S[js];
    const int64_t buf = P.buf_off[js], linv = P.linv_off[js];
    // the first CTA may mark the front as failed while others start: one thread asks
    if (__syncthreads_or(tid == 0 && (any_fail || P.sn_bad[js] || node_off(P, js)))) return;
    const int sp1 = min((k0 / kSuperPanel + 1) * kSuperPanel, sn_s);
    const bool chain = c0 < sp1, prev = chain && k0 % kSuperPanel != 0;
    const int c1 = min(c0 + kNB, sp1);                      // the next panel's columns end
    const int blk = (int)(task - jb.task0), r0 = c0 + blk * kNB;
    double* front = P.arena + buf;
    const double* pcol = front + (int64_t)k0 * ld;
    const bool first = blk == 0;
    const Buf own = first ? B1 : B0;                        // A, later L, of the CTA's rows
    // a warp's 32 x 16 of the products; X is lower triangular, so columns wn .. of
    // L21 take wn + 16 terms: the two warps of a scheduler have 80 together
    const int wm = (warp & 1) * 32, wn = (warp & 2 ? 16 : 0) ^ (warp & 4 ? 48 : 0);
    double cv[4][2][2], acc[4][2][2];
    if (prev) {
        const double* q = front + (int64_t)(k0 - kNB) * ld;
        chain_load(B0, q + r0, ld, F - r0, kNB, true);
        if (!first) chain_load(B1, q + c0, ld, c1 - c0, kNB, true);
        gemm::cp_async_commit();
    }
    chain_load(B2, P.linv + linv + (int64_t)(k0 / kNB) * kNB * kNB, kNB, kNB, kNB, true);
    if (first || !prev) {
        chain_load(own, pcol + r0, ld, F - r0, nb, (c0 & 1) == 0);      // (odd: S is, chain is off)
        if (!first && chain) chain_load_t(B1, front + k0 + (int64_t)c0 * ld, ld, c1 - c0);
    }
    gemm::cp_async_commit();
    if (tid < kNB) {
        const double d = tid < nb ? __ldcg(pcol + k0 + tid + (int64_t)tid * ld) : 0.0;
        dk[tid] = d;
        rd[tid] = tid < nb ? 1.0 / d : 0.0;
        if (prev) dp[tid] = __ldcg(front + (int64_t)(k0 - kNB + tid) * (ld + 1));
        if (first && chain && c0 + tid < c1) adv[tid] = __ldcg(P.adiag + P.fst[js] + c0 + tid);
    }
    const ChainTiles tl(warp);
    double (&ct)[5][2] = *reinterpret_cast<double (*)[5][2]>(&cv[0][0][0]);
    if (chain && first) {
#pragma unroll
        for (int q = 0; q < 5; ++q)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = c0 + 8 * tl.i[q] + (lane >> 2), c = c0 + 8 * tl.j[q] + 2 * (lane & 3) + h;
                ct[q][h] = (r < F && c < c1 && r >= c) ? __ldcg(front + r + (int64_t)c * ld) : 0.0;
            }
    } else if (chain) {
#pragma unroll
        for (int mi = 0; mi < 4; ++mi)
#pragma unroll
            for (int ni = 0; ni < 2; ++ni)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int r = r0 + wm + mi * 8 + (lane >> 2), c = c0 + wn + ni * 8 + 2 * (lane & 3) + h;
                    cv[mi][ni][h] = (r < F && c < c1 && r >= c) ? __ldcg(front + r + (int64_t)c * ld) : 0.0;
                }
    }
    if (prev) {
        gemm::cp_async_wait<1>();
        __syncthreads();
        if (first) chain_lower(ct, B0, dp, tl, lane);
        else chain_product<true>(acc, B0, B1, dp, wm, wn, lane, kNB);
        if (!first) {
#pragma unroll
            for (int mi = 0; mi < 4; ++mi)
#pragma unroll
                for (int ni = 0; ni < 2; ++ni)
#pragma unroll
                    for (int h = 0; h < 2; ++h) cv[mi][ni][h] -= acc[mi][ni][h];
            __syncthreads();
            chain_load(own, pcol + r0, ld, F - r0, nb, true);
            chain_load_t(B1, front + k0 + (int64_t)c0 * ld, ld, c1 - c0);
            gemm::cp_async_commit();
        }
    }
    gemm::cp_async_wait<0>();
    __syncthreads();
    // L21 = (A21 X') D^-1
    chain_product<false>(acc, own, B2, nullptr, wm, wn, lane, wn + 16);
    __syncthreads();
#pragma unroll
    for (int mi = 0; mi < 4; ++mi)
#pragma unroll
        for (int ni = 0; ni < 2; ++ni)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = wm + mi * 8 + (lane >> 2), c = wn + ni * 8 + 2 * (lane & 3) + h;
                const double l = acc[mi][ni][h] * rd[c];
                own[c][i] = l;
                if (r0 + i < F && c < nb) front[r0 + i + (int64_t)(k0 + c) * ld] = l;
            }
    if (!chain) return;
    if (first) {
        __syncthreads();
        chain_lower(ct, own, dk, tl, lane);
        double(*A)[kNB + 1] = reinterpret_cast<double(*)[kNB + 1]>(csh);     // in B0
        for (int e = tid; e < kNB * kNB; e += 256)
            if ((e & 63) < (e >> 6)) A[e & 63][e >> 6] = 0.0;
#pragma unroll
        for (int q = 0; q < 5; ++q)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = 8 * tl.i[q] + (lane >> 2), j = 8 * tl.j[q] + 2 * (lane & 3) + h, r = c0 + i, c = c0 + j;
                if (!tl.on(q) || i < j) continue;
                A[i][j] = r < c1 ? ct[q][h] : 0.0;                             // (c <= r)
                if (r >= c1 && r < F && c < c1) front[r + (int64_t)c * ld] = ct[q][h];
            }
        if (c0 + tid < c1) S.adv[tid & (kNB - 1)] = adv[tid & (kNB - 1)];
        if (tid == 0) S.fail = kNB;
        __syncthreads();
        diag_block<PR, false>(P, js, c0, c1 - c0, front, ld, 0, A, S);
        return;
    }
    chain_product<false>(acc, B1, B2, nullptr, wm, wn, lane, wn + 16);
    __syncthreads();
#pragma unroll
    for (int mi = 0; mi < 4; ++mi)
#pragma unroll
        for (int ni = 0; ni < 2; ++ni)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = wm + mi * 8 + (lane >> 2), c = wn + ni * 8 + 2 * (lane & 3) + h;
                B1[c][i] = acc[mi][ni][h] * rd[c];
            }
    __syncthreads();
    chain_product<true>(acc, own, B1, dk, wm, wn, lane, kNB);
    const bool copy = blk == 1 && c1 < sp1;                 // these are the panel after the next's rows
#pragma unroll
    for (int mi = 0; mi < 4; ++mi)
#pragma unroll
        for (int ni = 0; ni < 2; ++ni)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = r0 + wm + mi * 8 + (lane >> 2), c = c0 + wn + ni * 8 + 2 * (lane & 3) + h;
                if (r >= F || c >= c1) continue;
                const double v = cv[mi][ni][h] - acc[mi][ni][h];
                front[r + (int64_t)c * ld] = v;
                if (copy && r < sp1) front[c + (int64_t)r * ld] = v;
            }
}

// Inverse of the unit-lower diagonal blocks straight from LNZ (used when the
// factor in SM was not produced by this engine, e.g. a solve-only call).
__global__ void __launch_bounds__(64) k_linv(const Job* jobs, PV P) {
    __shared__ double L[kNB][kNB + 1];      // L strictly lower, X = L^-1 transposed above
    const Job& jb = jobs[blockIdx.x];
    const int js = jb.node, k0 = jb.k_lo, nb = jb.k_hi - jb.k_lo;
    const int F = P.F[js];
    const double* base = P.lnz + P.lnz_off[js];
    const int tid = threadIdx.x;
    for (int e = tid; e < nb * nb; e += blockDim.x) {
        const int i = e % nb, j = e / nb;
        if (i > j) L[i][j] = base[lnz_col(k0 + j, F) - (k0 + j) + (k0 + i)];
    }
    __syncthreads();
    if (tid < nb) {
        const int j = tid;
        for (int i = j + 1; i < nb; ++i) {
            double acc = -L[i][j];
            for (int m = j + 1; m < i; ++m) acc -= L[i][m] * L[j][m];
            L[j][i] = acc;
        }
    }
    __syncthreads();
    double* lv = P.linv + P.linv_off[js] + (int64_t)(k0 / kNB) * kNB * kNB;
    for (int e = tid; e < kNB * kNB; e += blockDim.x) {
        const int i = e % kNB, j = e / kNB;
        lv[e] = (i < nb && j < nb) ? (i > j ? L[j][i] : (i == j ? 1.0 : 0.0)) : 0.0;
    }
}

// Schur update C -= L D L' on T x T lower-triangle tiles with FP64 DMMA
// (mma.sync m8n8k4 f64).  A = rows i of L scaled by D (the scaling is applied
// to the A fragments), B = rows j of L, both read from the front buffer.
// Warps of WM x WN; K is staged through shared memory in 16-wide slices with
// a STAGES-deep cp.async pipeline (16-byte copies of row pairs).
namespace gemm {
constexpr int BK = 16;

template <int T, int WM, int WN, int STAGES>
struct Cfg {
    static constexpr int NWM = T / WM, NWN = T / WN, NT = NWM * NWN * 32;
    static constexpr int LDS = T + 4;                       // bank-conflict-free fragment reads
    static constexpr int MI = WM / 8, NI = WN / 8;
    static constexpr size_t smem = sizeof(double) * ((size_t)2 * STAGES * BK * LDS + (size_t)STAGES * BK);
};
}  // namespace gemm

template <int T, int WM, int WN, int STAGES>
__global__ void __launch_bounds__(gemm::Cfg<T, WM, WN, STAGES>::NT)
k_gemm(const Job* jobs, int64_t njobs, const int32_t* tmap, PV P) {
    using namespace gemm;
    using C = Cfg<T, WM, WN, STAGES>;
    extern __shared__ __align__(16) double gsh[];
    double* As = gsh;                                // [STAGES][BK][LDS]
    double* Bs = As + STAGES * BK * C::LDS;
    double* Ds = Bs + STAGES * BK * C::LDS;         // [STAGES][BK]
    if (P.st->any_fail) return;
    const int64_t task = blockIdx.x;
    const Job& jb = job_of(jobs, njobs, tmap, task);
    const int js = jb.node;
    if (P.sn_bad[js] || node_off(P, js)) return;
    const int ld = P.buf_ld[js];
    // decode the lower-triangle tile (column tile jt, row tile it >= jt)
    const int64_t u = task - jb.task0;
    const int nct = (jb.c_end - jb.c0 + T - 1) / T;
    const int nr = (jb.r_end - jb.c0 + T - 1) / T;
    int lo = 0, hi = nct - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        const int64_t pre = (int64_t)mid * nr - ((int64_t)mid * (mid - 1)) / 2;
        if (pre <= u) lo = mid;
        else hi = mid - 1;
    }
    const int jt = lo;
    const int it = jt + (int)(u - ((int64_t)jt * nr - ((int64_t)jt * (jt - 1)) / 2));
    const int i0 = jb.c0 + it * T, j0 = jb.c0 + jt * T;
    const int r_end = jb.r_end, c_end = jb.c_end;
    const double* front = P.arena + P.buf_off[js];
    double* frontw = P.arena + P.buf_off[js];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = (warp % C::NWM) * WM, wn = (warp / C::NWM) * WN;

    double acc[C::MI][C::NI][2];
#pragma unroll
    for (int a = 0; a < C::MI; ++a)
#pragma unroll
        for (int b = 0; b < C::NI; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;

    const int k_lo = jb.k_lo, k_hi = jb.k_hi;
    const int nk = (k_hi - k_lo + BK - 1) / BK;
    // 16-byte copies need an even first row (the buffer base and ld are
    // 32-byte multiples); tiles of jobs starting on an odd column use 8 bytes
    const bool even = ((i0 | j0) & 1) == 0;
    auto load_stage = [&](int stage, int kt) {
        const int kb = k_lo + kt * BK;
        double* as = As + stage * BK * C::LDS;
        double* bs = Bs + stage * BK * C::LDS;
#pragma unroll
        for (int e = 0; e < (T / 2 * BK + C::NT - 1) / C::NT; ++e) {
            const int idx = tid + e * C::NT;
            if (idx < T / 2 * BK) {
                const int pr = idx % (T / 2), k = idx / (T / 2);
                const int r = 2 * pr, kk = kb + k;
                const bool kv = kk < k_hi;
                const int64_t col = (int64_t)(kv ? kk : k_lo) * ld;
                const int ra = i0 + r, rb = j0 + r;
                const int na = kv ? max(0, min(2, r_end - ra)) : 0;
                const int nbb = kv ? max(0, min(2, r_end - rb)) : 0;
                if (even) {
                    cp_async16(as + k * C::LDS + r, front + col + (na > 0 ? ra : i0), 8 * na);
                    cp_async16(bs + k * C::LDS + r, front + col + (nbb > 0 ? rb : j0), 8 * nbb);
                } else {
                    cp_async8(as + k * C::LDS + r, front + col + (na > 0 ? ra : i0), na > 0);
                    cp_async8(as + k * C::LDS + r + 1, front + col + (na > 1 ? ra + 1 : i0), na > 1);
                    cp_async8(bs + k * C::LDS + r, front + col + (nbb > 0 ? rb : j0), nbb > 0);
                    cp_async8(bs + k * C::LDS + r + 1, front + col + (nbb > 1 ? rb + 1 : j0), nbb > 1);
                }
            }
        }
        if (tid < BK) {
            const int kk = kb + tid;
            cp_async8(Ds + stage * BK + tid, front + (int64_t)(kk < k_hi ? kk : k_lo) * (ld + 1), kk < k_hi);
        }
    };

#pragma unroll
    for (int st = 0; st < STAGES - 1; ++st) {
        if (st < nk) load_stage(st, st);
        cp_async_commit();
    }
    for (int kt = 0; kt < nk; ++kt) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();
        const int nxt = kt + STAGES - 1;
        if (nxt < nk) load_stage(nxt % STAGES, nxt);
        cp_async_commit();
        const int cur = kt % STAGES;
        const double* as = As + cur * BK * C::LDS;
        const double* bs = Bs + cur * BK * C::LDS;
        const double* ds = Ds + cur * BK;
#pragma unroll
        for (int k4 = 0; k4 < BK; k4 += 4) {
            const int kk = k4 + (lane & 3);
            const double dk = ds[kk];
            double a[C::MI], b[C::NI];
#pragma unroll
            for (int mi = 0; mi < C::MI; ++mi) a[mi] = as[kk * C::LDS + wm + mi * 8 + (lane >> 2)] * dk;
#pragma unroll
            for (int ni = 0; ni < C::NI; ++ni) b[ni] = bs[kk * C::LDS + wn + ni * 8 + (lane >> 2)];
#pragma unroll
            for (int mi = 0; mi < C::MI; ++mi)
#pragma unroll
                for (int ni = 0; ni < C::NI; ++ni) dmma(acc[mi][ni][0], acc[mi][ni][1], a[mi], b[ni]);
        }
    }
    cp_async_wait<0>();
    // epilogue: C -= acc on the lower part, inside [.., r_end) x [.., c_end);
    // in two halves of the warp tile, each with its loads ahead of its
    // stores, so that the loads overlap instead of waiting one latency each
    constexpr int MH = C::MI > 1 ? C::MI / 2 : 1;
#pragma unroll
    for (int m0 = 0; m0 < C::MI; m0 += MH) {
        double cv[MH][C::NI][2];
#pragma unroll
        for (int q = 0; q < MH; ++q) {
            const int r = i0 + wm + (m0 + q) * 8 + (lane >> 2);
#pragma unroll
            for (int ni = 0; ni < C::NI; ++ni)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int c = j0 + wn + ni * 8 + 2 * (lane & 3) + h;
                    cv[q][ni][h] =
                        (r < r_end && c < c_end && r >= c) ? __ldcg(front + (int64_t)r + (int64_t)c * ld) : 0.0;
                }
        }
#pragma unroll
        for (int q = 0; q < MH; ++q) {
            const int r = i0 + wm + (m0 + q) * 8 + (lane >> 2);
            if (r >= r_end) continue;
#pragma unroll
            for (int ni = 0; ni < C::NI; ++ni)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int c = j0 + wn + ni * 8 + 2 * (lane & 3) + h;
                    if (c < c_end && r >= c)
                        frontw[(int64_t)r + (int64_t)c * ld] = cv[q][ni][h] - acc[m0 + q][ni][h];
                }
        }
    }
}

#ifndef SPR_GEMM_BIG_WM
#define SPR_GEMM_BIG_WM 32
#endif
#ifndef SPR_GEMM_BIG_WN
#define SPR_GEMM_BIG_WN 32
#endif
#ifndef SPR_GEMM_STAGES
#define SPR_GEMM_STAGES 3
#endif
using GemmBig = gemm::Cfg<kTileBig, SPR_GEMM_BIG_WM, SPR_GEMM_BIG_WN, SPR_GEMM_STAGES>;
using GemmSmall = gemm::Cfg<kTile, 32, 32, SPR_GEMM_STAGES>;
using GemmTiny = gemm::Cfg<kTileTiny, 16, 16, SPR_GEMM_STAGES>;
#define K_GEMM_BIG k_gemm<kTileBig, SPR_GEMM_BIG_WM, SPR_GEMM_BIG_WN, SPR_GEMM_STAGES>
#define K_GEMM_SMALL k_gemm<kTile, 32, 32, SPR_GEMM_STAGES>
#define K_GEMM_TINY k_gemm<kTileTiny, 16, 16, SPR_GEMM_STAGES>

// Mixed-precision Schur update: C -= L D L' with 3xTF32 split products on
// the tensor cores (mma.sync m16n8k8 tf32, FP32 accumulation inside each
// 64-wide slice of K, FP64 accumulation across slices and in C).  Each FP64
// operand a is rounded to FP32, then split a = hi + lo with hi = tf32(a),
// lo = tf32(a - hi); the product uses hi*hi + hi*lo + lo*hi.
namespace x3 {
__device__ __forceinline__ uint32_t tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;\n" : "=r"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ void split(double v, uint32_t& hi, uint32_t& lo) {
    const float f = (float)v;
    hi = tf32(f);
    lo = tf32(f - __uint_as_float(hi));
}
__device__ __forceinline__ void mma(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
}  // namespace x3

#include "tc_gemm.cuh"
#include "i8_gemm.cuh"

__global__ void __launch_bounds__(128) k_gemm_x3(const Job* jobs, int64_t njobs, const int32_t* tmap, PV P) {
    using namespace gemm;
    constexpr int T = kTile, STAGES = 3, LDS = T + 4;
    extern __shared__ __align__(16) double gsh[];
    double* As = gsh;
    double* Bs = As + STAGES * BK * LDS;
    double* Ds = Bs + STAGES * BK * LDS;
    if (P.st->any_fail) return;
    const int64_t task = blockIdx.x;
    const Job& jb = job_of(jobs, njobs, tmap, task);
    const int js = jb.node;
    if (P.sn_bad[js] || node_off(P, js)) return;
    const int ld = P.buf_ld[js];
    const int64_t u = task - jb.task0;
    const int nct = (jb.c_end - jb.c0 + T - 1) / T;
    const int nr = (jb.r_end - jb.c0 + T - 1) / T;
    int lo = 0, hi = nct - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        const int64_t pre = (int64_t)mid * nr - ((int64_t)mid * (mid - 1)) / 2;
        if (pre <= u) lo = mid;
        else hi = mid - 1;
    }
    const int jt = lo;
    const int it = jt + (int)(u - ((int64_t)jt * nr - ((int64_t)jt * (jt - 1)) / 2));
    const int i0 = jb.c0 + it * T, j0 = jb.c0 + jt * T;
    const int r_end = jb.r_end, c_end = jb.c_end;
    const double* front = P.arena + P.buf_off[js];
    double* frontw = P.arena + P.buf_off[js];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int wm = (warp & 1) * 32, wn = (warp >> 1) * 32;
    float acc[2][4][4];
    double acc64[2][4][4];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                acc[a][b][c] = 0.f;
                acc64[a][b][c] = 0.0;
            }
    const int k_lo = jb.k_lo, k_hi = jb.k_hi;
    const int nk = (k_hi - k_lo + BK - 1) / BK;
    const bool even = ((i0 | j0) & 1) == 0;
    auto load_stage = [&](int stage, int kt) {
        const int kb = k_lo + kt * BK;
        double* as = As + stage * BK * LDS;
        double* bs = Bs + stage * BK * LDS;
#pragma unroll
        for (int e = 0; e < (T / 2 * BK + 127) / 128; ++e) {
            const int idx = tid + e * 128;
            if (idx < T / 2 * BK) {
                const int pr = idx % (T / 2), k = idx / (T / 2);
                const int r = 2 * pr, kk = kb + k;
                const bool kv = kk < k_hi;
                const int64_t col = (int64_t)(kv ? kk : k_lo) * ld;
                const int ra = i0 + r, rb = j0 + r;
                const int na = kv ? max(0, min(2, r_end - ra)) : 0;
                const int nbb = kv ? max(0, min(2, r_end - rb)) : 0;
                if (even) {
                    cp_async16(as + k * LDS + r, front + col + (na > 0 ? ra : i0), 8 * na);
                    cp_async16(bs + k * LDS + r, front + col + (nbb > 0 ? rb : j0), 8 * nbb);
                } else {
                    cp_async8(as + k * LDS + r, front + col + (na > 0 ? ra : i0), na > 0);
                    cp_async8(as + k * LDS + r + 1, front + col + (na > 1 ? ra + 1 : i0), na > 1);
                    cp_async8(bs + k * LDS + r, front + col + (nbb > 0 ? rb : j0), nbb > 0);
                    cp_async8(bs + k * LDS + r + 1, front + col + (nbb > 1 ? rb + 1 : j0), nbb > 1);
                }
            }
        }
        if (tid < BK) {
            const int kk = kb + tid;
            cp_async8(Ds + stage * BK + tid, front + (int64_t)(kk < k_hi ? kk : k_lo) * (ld + 1), kk < k_hi);
        }
    };
#pragma unroll
    for (int st = 0; st < STAGES - 1; ++st) {
        if (st < nk) load_stage(st, st);
        cp_async_commit();
    }
    for (int kt = 0; kt < nk; ++kt) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();
        const int nxt = kt + STAGES - 1;
        if (nxt < nk) load_stage(nxt % STAGES, nxt);
        cp_async_commit();
        const int cur = kt % STAGES;
        const double* as = As + cur * BK * LDS;
        const double* bs = Bs + cur * BK * LDS;
        const double* ds = Ds + cur * BK;
#pragma unroll
        for (int k8 = 0; k8 < BK; k8 += 8) {
            const double d0 = ds[k8 + t], d1 = ds[k8 + t + 4];
            uint32_t ah[2][4], al[2][4], bh[4][2], bl[4][2];
#pragma unroll
            for (int mi = 0; mi < 2; ++mi) {
                const int r0 = wm + mi * 16 + g;
                x3::split(as[(k8 + t) * LDS + r0] * d0, ah[mi][0], al[mi][0]);
                x3::split(as[(k8 + t) * LDS + r0 + 8] * d0, ah[mi][1], al[mi][1]);
                x3::split(as[(k8 + t + 4) * LDS + r0] * d1, ah[mi][2], al[mi][2]);
                x3::split(as[(k8 + t + 4) * LDS + r0 + 8] * d1, ah[mi][3], al[mi][3]);
            }
#pragma unroll
            for (int ni = 0; ni < 4; ++ni) {
                const int c = wn + ni * 8 + g;
                x3::split(bs[(k8 + t) * LDS + c], bh[ni][0], bl[ni][0]);
                x3::split(bs[(k8 + t + 4) * LDS + c], bh[ni][1], bl[ni][1]);
            }
#pragma unroll
            for (int mi = 0; mi < 2; ++mi)
#pragma unroll
                for (int ni = 0; ni < 4; ++ni) {
                    x3::mma(acc[mi][ni], al[mi], bh[ni][0], bh[ni][1]);
                    x3::mma(acc[mi][ni], ah[mi], bl[ni][0], bl[ni][1]);
                    x3::mma(acc[mi][ni], ah[mi], bh[ni][0], bh[ni][1]);
                }
        }
        if ((kt & 3) == 3 || kt == nk - 1) {           // FP64 accumulation across 64-wide K slices
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b)
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        acc64[a][b][c] += (double)acc[a][b][c];
                        acc[a][b][c] = 0.f;
                    }
        }
    }
    cp_async_wait<0>();
#pragma unroll
    for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = i0 + wm + mi * 16 + g + 8 * h;
            if (r >= r_end) continue;
#pragma unroll
            for (int ni = 0; ni < 4; ++ni)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int c = j0 + wn + ni * 8 + 2 * t + q;
                    if (c < c_end && r >= c) frontw[(int64_t)r + (int64_t)c * ld] -= acc64[mi][ni][2 * h + q];
                }
        }
}

// Store the S factored columns of a dense front into LNZ (sprfc1.f:630-637).
__global__ void k_writeback(const Job* jobs, int64_t njobs, const int32_t* tmap, int64_t ntasks, PV P) {
    if (P.st->any_fail) return;
    const int lane = threadIdx.x & 31;
    const int64_t task = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    if (task >= ntasks) return;
    const Job& jb = job_of(jobs, njobs, tmap, task);
    const int js = jb.node;
    if (P.sn_bad[js] || node_off(P, js)) return;
    const int j = jb.c0 + (int)(task - jb.task0);
    const int F = P.F[js], ld = P.buf_ld[js];
    const double* col = P.arena + P.buf_off[js] + (int64_t)j * ld;
    double* dst = P.lnz + P.lnz_off[js] + lnz_col(j, F) - j;
    int i = j + lane;
    for (; i + 96 < F; i += 128) {
        const double a0 = __ldcg(col + i), a1 = __ldcg(col + i + 32), a2 = __ldcg(col + i + 64),
                     a3 = __ldcg(col + i + 96);
        dst[i] = a0;
        dst[i + 32] = a1;
        dst[i + 64] = a2;
        dst[i + 96] = a3;
    }
    for (; i < F; i += 32) dst[i] = col[i];
}

// ---------------------------------------------------------------------------
// Solves (multi-RHS), one CTA per front, level by level.
// Front vectors live in vbuf: front p uses F_p x nrhs doubles at rbase[p]*nrhs
// (column r at offset r*F_p).  After the forward sweep, rows S..F of a front
// vector are its update vector for the parent.
// ---------------------------------------------------------------------------
constexpr int kSolveThreads = 256;
// threads of a one-CTA-per-front launch (factor or solve) of a size class:
// the smallest fronts take 128, so that twice as many fronts are in flight
// per SM (their shared memory allows it)
inline int small_threads(int maxF) { return maxF <= 64 ? 128 : 256; }

// Small fronts (F <= kSmallMaxF), one CTA each: the latency of the dependent
// loads (tables, children's vectors, L) and of the triangles' chain bounds
// them.  The whole trapezoid of L is copied to shared memory while the vectors
// are gathered.  Per 32 columns a warp solves the triangle for NG right-hand
// sides at a time, y_c going round by shuffles, and the rectangle takes one row
// (forward) or one column (back, rows dealt to the warps) a thread, NG
// right-hand sides at a time, so that an entry of L is read once for them.
// Before (L by blocks of 32 columns after the gather, one right-hand side a
// thread): 512 boxes of 3^3 to 12^3, 16 right-hand sides, 3.8 ms forward and
// 2.2 ms back, now 2.4 and 2.0; both sweeps of a 4^3 box 0.16 ms, now 0.11 ms.
constexpr int kSmallBlk = 32;
// shared memory: the front vector (F x the right-hand sides rounded up to whole
// groups), the warps' partial sums of the back sweep, L and its alignment
inline int small_group_of(int nrhs) { return nrhs == 1 ? 1 : nrhs == 2 ? 2 : 4; }
inline size_t small_solve_smem(int maxF, int maxL, int nrhs) {
    const int ng = small_group_of(nrhs), nrp = (nrhs + ng - 1) / ng * ng;
    return sizeof(double) * ((size_t)maxF * nrp + 8 * kSmallBlk * ng + maxL + 4);
}
constexpr size_t kSmallSolveSmem = sizeof(double) * ((size_t)kSmallMaxF * kMaxRHS + 8 * kSmallBlk * 4 +
                                                     (size_t)kSmallMaxF * (kSmallMaxF + 1) / 2 + 4);

// n doubles to shared memory without waiting; returns where they are (room, 16-byte
// aligned, has one more: the copy keeps the source's alignment)
__device__ __forceinline__ const double* small_copy(double* room, const double* src, int n) {
    const int head = min(n, (int)((uintptr_t)src >> 3 & 1)), pairs = (n - head) >> 1;
    double* to = room + ((uintptr_t)src >> 3 & 1);
    for (int e = threadIdx.x; e < pairs; e += blockDim.x) gemm::cp_async16(to + head + 2 * e, src + head + 2 * e, 16);
    if (threadIdx.x == 0 && head) gemm::cp_async8(to, src, true);
    if (threadIdx.x == 0 && (n - head & 1)) gemm::cp_async8(to + n - 1, src + n - 1, true);
    gemm::cp_async_commit();
    return to;
}

template <int NG>
__device__ __forceinline__ void small_get(const double* p, double (&v)[NG]) {
    if (NG == 1) {
        v[0] = p[0];
    } else {
#pragma unroll
        for (int r = 0; r < NG; r += 2) {
            const double2 d = *reinterpret_cast<const double2*>(p + r);
            v[r] = d.x;
            v[r + 1 < NG ? r + 1 : r] = d.y;
        }
    }
}

template <int NG>
__global__ void __launch_bounds__(kSolveThreads)
k_forward(const int32_t* nodes, PV P, double* vbuf, double* b, int64_t ldb, int nrhs_all) {
    extern __shared__ __align__(16) double wsm[];      // w[i * nrp + r], then L packed by columns
    const int js = nodes[blockIdx.x];
    if (node_off(P, js)) return;
    const int F = P.F[js], S = P.S[js], fst = P.fst[js];
    const int64_t rbase = P.rbase[js];
    // a retained front only passes its sums on (own rows to B, the rest to the parent)
    const bool ret = is_retained(P, js);
    // this CTA's right-hand sides: kMaxRHS from rg on
    const int rg = blockIdx.y * kMaxRHS, nrhs = min(kMaxRHS, nrhs_all - rg), ng = (nrhs + NG - 1) / NG, nrp = ng * NG;
    b += (int64_t)rg * ldb;
    double* room = wsm + (((size_t)F * nrp + 1) & ~(size_t)1);
    const double* L = small_copy(room, P.lnz + P.lnz_off[js], ret ? 0 : F * S - S * (S - 1) / 2);
    double* wg = vbuf + rbase * nrhs_all + (int64_t)rg * F;   // update rows for the parent (r*F + i)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5;
    for (int e = tid; e < F * ng; e += blockDim.x) {
        const int i = e % F, r0 = e / F * NG;
        double v[NG];
#pragma unroll
        for (int r = 0; r < NG; ++r) v[r] = (i < S && r0 + r < nrhs) ? b[(int64_t)(fst + i) + (r0 + r) * ldb] : 0.0;
        const int64_t e0 = P.cptr[rbase + i], e1 = P.cptr[rbase + i + 1];
        for (int64_t q = e0; q < e1; ++q) {
            const int c = P.cchild[q], t = P.ct[q], fc = P.F[c];
            const double* u = vbuf + P.rbase[c] * nrhs_all + (int64_t)(rg + r0) * fc + P.S[c] + t;
#pragma unroll
            for (int r = 0; r < NG; ++r)
                if (r0 + r < nrhs) v[r] += u[(int64_t)r * fc];
        }
#pragma unroll
        for (int r = 0; r < NG; ++r) wsm[i * nrp + r0 + r] = v[r];
    }
    gemm::cp_async_wait<0>();
    for (int j0 = 0; j0 < (ret ? 0 : S); j0 += kSmallBlk) {
        const int nb = min(kSmallBlk, S - j0);
        __syncthreads();
        // triangle of the block (SPRFS5 :600-608)
        for (int g = warp; g < ng; g += nwarp) {
            double y[NG];
            double* wp = wsm + (j0 + min(lane, nb - 1)) * nrp + g * NG;
            small_get<NG>(wp, y);
            const double* lp = L + pk(j0 + lane, j0, F);               // column c of this lane's row: c (F - j0 - 1) - c (c - 1) / 2 on
            const bool in = lane < nb;
#pragma unroll 8
            for (int c = 0; c < nb - 1; ++c) {
                const double l = lane > c && in ? *lp : 0.0;
#pragma unroll
                for (int r = 0; r < NG; ++r) {
                    const double yc = __shfl_sync(0xffffffffu, y[r], c);
                    if (lane > c) y[r] = fma(-yc, l, y[r]);
                }
                lp += F - (j0 + c) - 1;
            }
            if (in)
#pragma unroll
                for (int r = 0; r < NG; ++r) wp[r] = y[r];
        }
        __syncthreads();
        const int below = F - j0 - nb;
        for (int e = tid; e < below * ng; e += blockDim.x) {           // rectangle (SPRFS6)
            const int g = e / below, i = j0 + nb + e - g * below;
            double v[NG];
            small_get<NG>(wsm + i * nrp + g * NG, v);
            const double* lp = L + pk(i, j0, F);
            const double* wp = wsm + j0 * nrp + g * NG;
#pragma unroll 8
            for (int c = 0; c < nb; ++c) {
                double w[NG];
                small_get<NG>(wp, w);
                const double l = *lp;
#pragma unroll
                for (int r = 0; r < NG; ++r) v[r] = fma(-l, w[r], v[r]);
                lp += F - (j0 + c) - 1;
                wp += nrp;
            }
#pragma unroll
            for (int r = 0; r < NG; ++r) wsm[i * nrp + g * NG + r] = v[r];
        }
    }
    __syncthreads();
    for (int e = tid; e < F * nrhs; e += blockDim.x) {
        const int r = e / F, i = e - r * F;
        const double v = wsm[i * nrp + r];
        if (i < S) b[(int64_t)(fst + i) + r * ldb] = ret ? v : v / L[pk(i, i, F)];
        else wg[(int64_t)r * F + i] = v;
    }
}

template <int NG>
__global__ void __launch_bounds__(kSolveThreads)
k_backward(const int32_t* nodes, PV P, double* b, int64_t ldb, int nrhs_all) {
    extern __shared__ __align__(16) double wsm[];
    const int js = nodes[blockIdx.x];
    if (node_off(P, js)) return;
    if (is_retained(P, js)) return;
    const int F = P.F[js], S = P.S[js], fst = P.fst[js];
    const int64_t rbase = P.rbase[js];
    // this CTA's right-hand sides: kMaxRHS from rg on
    const int rg = blockIdx.y * kMaxRHS, nrhs = min(kMaxRHS, nrhs_all - rg), ng = (nrhs + NG - 1) / NG, nrp = ng * NG;
    b += (int64_t)rg * ldb;
    double* red = wsm + (((size_t)F * nrp + 1) & ~(size_t)1);          // [warp][column][NG]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5;
    const double* L = small_copy(red + nwarp * kSmallBlk * NG, P.lnz + P.lnz_off[js], F * S - S * (S - 1) / 2);
    // own rows (forward result) and the ancestors' solved rows; the row list
    // of front js starts at rbase[js] (LINDX concatenates the row lists)
    for (int e = tid; e < F * ng; e += blockDim.x) {
        const int i = e % F, r0 = e / F * NG;
        const int row = (i < S) ? (fst + i) : P.rows[rbase + i];
#pragma unroll
        for (int r = 0; r < NG; ++r) wsm[i * nrp + r0 + r] = r0 + r < nrhs ? b[(int64_t)row + (r0 + r) * ldb] : 0.0;
    }
    gemm::cp_async_wait<0>();
    // the rows below a block are dealt to `slices` warps per group of right-hand sides
    const int slices = nwarp / ng, g = warp / slices, slice = warp % slices;
    const int nblk = (S + kSmallBlk - 1) / kSmallBlk;
    for (int bi = nblk - 1; bi >= 0; --bi) {
        const int j0 = bi * kSmallBlk, nb = min(kSmallBlk, S - j0);
        __syncthreads();
        if (g < ng) {                                                  // rows below the block (SPRBS6)
            double v[NG];
#pragma unroll
            for (int r = 0; r < NG; ++r) v[r] = 0.0;
            const int c = j0 + min(lane, nb - 1);
            const double* lp = L + pk(0, c, F);
#pragma unroll 4
            for (int i = j0 + nb + slice; i < F; i += slices) {
                double w[NG];
                small_get<NG>(wsm + i * nrp + g * NG, w);
                const double l = lp[i];
#pragma unroll
                for (int r = 0; r < NG; ++r) v[r] = fma(l, w[r], v[r]);
            }
#pragma unroll
            for (int r = 0; r < NG; ++r) red[(warp * kSmallBlk + lane) * NG + r] = v[r];
        }
        __syncthreads();
        // triangle of the block, bottom-up: lane c holds x_c; each finished x_i is
        // shuffled to the lanes above it
        if (g < ng && slice == 0) {
            double x[NG];
            double* wp = wsm + (j0 + min(lane, nb - 1)) * nrp + g * NG;
            small_get<NG>(wp, x);
            double sum[NG];
#pragma unroll
            for (int r = 0; r < NG; ++r) sum[r] = 0.0;
            for (int q = 0; q < slices; ++q) {
                double v[NG];
                small_get<NG>(red + ((warp + q) * kSmallBlk + lane) * NG, v);
#pragma unroll
                for (int r = 0; r < NG; ++r) sum[r] += v[r];
            }
#pragma unroll
            for (int r = 0; r < NG; ++r) x[r] -= sum[r];
            const double* lp = L + pk(j0, j0 + min(lane, nb - 1), F);
#pragma unroll 8
            for (int i = nb - 1; i > 0; --i) {
                const double l = lane < i ? lp[i] : 0.0;
#pragma unroll
                for (int r = 0; r < NG; ++r) {
                    const double xi = __shfl_sync(0xffffffffu, x[r], i);
                    if (lane < i) x[r] = fma(-l, xi, x[r]);
                }
            }
            if (lane < nb)
#pragma unroll
                for (int r = 0; r < NG; ++r) wp[r] = x[r];
        }
    }
    __syncthreads();
    for (int e = tid; e < S * nrhs; e += blockDim.x) {
        const int r = e / S, i = e - r * S;
        b[(int64_t)(fst + i) + r * ldb] = wsm[i * nrp + r];
    }
}

// ---------------------------------------------------------------------------
// Solves of the large fronts, per tree level: forward k_fwd_tri (rows [0, S))
// and k_fwd_rect (rows [S, F)), back k_bwd_rect and k_bwd_tri.  L is read
// from LNZ (packed).  Right-hand sides go in groups of NG = 1, 2 or 4 (nrp in
// all, with the last group's padding): a group's values of an equation lie
// together, y[(group * NEQ + equation) * NG + r], so that the groups are
// independent tasks which share L through L2.
// ---------------------------------------------------------------------------
// row i of front js in the forward sweep: own row of B (i < S) plus the
// children's update vectors, in SPRF12's order
__device__ __forceinline__ double gather_row(const PV& P, const double* vbuf, const double* b, int64_t ldb, int nrhs,
                                             int js, int i, int r) {
    double v = i < P.S[js] ? b[(int64_t)(P.fst[js] + i) + r * ldb] : 0.0;
    const int64_t e0 = P.cptr[P.rbase[js] + i], e1 = P.cptr[P.rbase[js] + i + 1];
    for (int64_t e = e0; e < e1; ++e) {
        const int c = P.cchild[e], t = P.ct[e];
        v += vbuf[P.rbase[c] * nrhs + (int64_t)r * P.F[c] + P.S[c] + t];
    }
    return v;
}

// A retained front passes its gathered sums on: own rows to B, the rest to
// its parent (thread per row).
__global__ void k_fwd_retained(const Job* jobs, int64_t njobs, const int32_t* tmap, int64_t ntasks, PV P, double* vbuf,
                               double* b, int64_t ldb, int nrhs) {
    const int64_t task = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (task >= ntasks) return;
    const Job& jb = job_of(jobs, njobs, tmap, task);
    const int js = jb.node;
    if (node_off(P, js) || !is_retained(P, js)) return;
    const int i = (int)(task - jb.task0);
    for (int r = 0; r < nrhs; ++r) {
        const double v = gather_row(P, vbuf, b, ldb, nrhs, js, i, r);
        if (i < P.S[js]) b[(int64_t)(P.fst[js] + i) + r * ldb] = v;
        else vbuf[P.rbase[js] * nrhs + (int64_t)r * P.F[js] + i] = v;
    }
}

// Reduce-scatter of NR per-lane partial sums over a warp: halving exchanges
// (NR/2 + NR/4 + ... shuffles) then full sums over the remaining lane bits.
// Returns the total of partial index `rhs`; the lanes whose remaining bits
// are zero (lane & (first_rem * 2 - 1)) == 0 hold distinct totals.
template <int NR>
__device__ __forceinline__ double warp_reduce_scatter(double (&v)[NR], int lane, int& rhs, int& owner_mask) {
    int base = 0, o = 16;
#pragma unroll
    for (int h = NR / 2; h >= 1; h >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int j = 0; j < h; ++j) {
            const double send = up ? v[j] : v[j + h];
            const double keep = up ? v[j + h] : v[j];
            v[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
        if (up) base += h;
    }
    owner_mask = 2 * o - 1;
#pragma unroll
    for (; o >= 1; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    rhs = base;
    return v[0];
}

// Forward sweep, rows [S, F): w[i] = gathered[i] - sum_{c < S} L[i][c] y[c].
// One CTA per tile and M groups of right-hand sides.  Fronts of at most
// kFwdNarrow columns (most of them): 256 rows, a thread per row, all columns.
// Wider ones: kFwdRows rows x kFwdCols columns, a thread per row and quarter of the
// columns, the quarters added in shared memory; a front of one column tile is
// finished here, with several each tile writes its partial sums and
// k_fwd_rect_sum adds them in a fixed order.  Latency bounds it in all but the
// largest levels (loads of L go in unpredicated batches: 48^3, 4 right-hand
// sides 2.0 ms, 3.4 ms with a test per load).  Every front with 64-column tiles and
// partials, a launch to add them and launches to gather before and to finish
// after took 3.5 ms there, and on 512 boxes of 3^3 to 12^3 with 16 right-hand
// sides 4.5 ms (now 1.9 ms).
template <int NG, int M>
__global__ void __launch_bounds__(256, M > 1 ? 3 : 4) k_fwd_rect(const Job* jobs, int64_t njobs, const int32_t* tmap, PV P,
                                                  const double* y, double* vbuf, double* pbuf, int nrhs, int nrp,
                                                  int64_t neq) {
    constexpr int NR = NG * M;
    constexpr int LB = NR >= 4 ? 8 : 16;                       // loads of L in flight per thread
    __shared__ __align__(16) double ys[kFwdCols * NR];
    __shared__ double part[M == 1 ? 4 : 3][NR][kFwdRows];
    const int64_t task = blockIdx.x;
    const Job& jb = job_of(jobs, njobs, tmap, task);
    const int js = jb.node;
    if (node_off(P, js)) return;
    const int F = P.F[js], S = P.S[js], fst = P.fst[js];
    const int ncc = jb.k_hi, g0 = blockIdx.y * M;                 // first group
    const int64_t u = task - jb.task0;
    const int cc = (int)(u % ncc), rc = (int)(u / ncc);
    const int tid = threadIdx.x;
    const bool narrow = S <= kFwdNarrow;
    const int row = narrow ? tid : tid & (kFwdRows - 1), q = narrow ? 0 : tid >> 6;
    const int i = S + rc * (narrow ? 256 : kFwdRows) + row;
    const int cbeg = cc * kFwdCols, ncol = min(kFwdCols, S - cbeg);
    const int r0 = g0 * NG, nr = min(NR, nrhs - r0);             // this CTA's right-hand sides
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const double* yg = y + ((int64_t)(g0 + m) * neq + fst + cbeg) * NG;
        for (int e = tid; e < ncol * NG; e += 256)
            ys[(e / NG) * NR + m * NG + e % NG] = (g0 + m) * NG < nrhs ? yg[e] : 0.0;
    }
    // the gathered entries (a chain of dependent loads): a narrow tile's thread
    // takes all of its row's, a wide one's r = q, q + 4, ..; ahead of L with few
    // right-hand sides, after it where the registers would cost occupancy
    double w[NR];
    if constexpr (M == 1) {
#pragma unroll
    for (int r = 0; r < NR; ++r) w[r] = 0.0;
    if (i < F && ncc == 1) {
        const int64_t e0 = P.cptr[P.rbase[js] + i], e1 = P.cptr[P.rbase[js] + i + 1];
        for (int64_t e = e0; e < e1; ++e) {
            const int c = P.cchild[e], fc = P.F[c];
            const double* v = vbuf + P.rbase[c] * nrhs + (int64_t)r0 * fc + P.S[c] + P.ct[e];
            if (narrow) {
#pragma unroll
                for (int r = 0; r < NR; ++r)
                    if (r < nr) w[r] += v[(int64_t)r * fc];
            } else {
#pragma unroll
                for (int k = 0; k < (NR + 3) / 4; ++k)
                    if (q + 4 * k < nr) w[k] += v[(int64_t)(q + 4 * k) * fc];
            }
        }
    }
    }
    __syncthreads();
    double acc[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) acc[r] = 0.0;
    if (i < F) {
        const int c0 = 64 * q, c1 = min(c0 + 64, ncol);
        const double* p = P.lnz + P.lnz_off[js] + lnz_col(cbeg + c0, F) - (cbeg + c0) + i;
        int64_t step = F - (cbeg + c0) - 1;                     // to the next column, same row
        int c = c0;
        for (; c + LB <= c1; c += LB) {
            double l[LB];
#pragma unroll
            for (int k = 0; k < LB; ++k) {
                l[k] = __ldg(p);
                p += step--;
            }
#pragma unroll
            for (int k = 0; k < LB; ++k)
#pragma unroll
                for (int r = 0; r < NR; ++r) acc[r] += l[k] * ys[(c + k) * NR + r];
        }
        if (c < c1) {
            double l[LB];
#pragma unroll
            for (int k = 0; k < LB; ++k) {
                l[k] = c + k < c1 ? __ldg(p) : 0.0;
                p += step--;
            }
#pragma unroll
            for (int k = 0; k < LB; ++k)
                if (c + k < c1)
#pragma unroll
                    for (int r = 0; r < NR; ++r) acc[r] += l[k] * ys[(c + k) * NR + r];
        }
    }
    if constexpr (M > 1) {
#pragma unroll
    for (int r = 0; r < NR; ++r) w[r] = 0.0;
    if (i < F && ncc == 1) {
        const int64_t e0 = P.cptr[P.rbase[js] + i], e1 = P.cptr[P.rbase[js] + i + 1];
        for (int64_t e = e0; e < e1; ++e) {
            const int c = P.cchild[e], fc = P.F[c];
            const double* v = vbuf + P.rbase[c] * nrhs + (int64_t)r0 * fc + P.S[c] + P.ct[e];
            if (narrow) {
#pragma unroll
                for (int r = 0; r < NR; ++r)
                    if (r < nr) w[r] += v[(int64_t)r * fc];
            } else {
#pragma unroll
                for (int k = 0; k < (NR + 3) / 4; ++k)
                    if (q + 4 * k < nr) w[k] += v[(int64_t)(q + 4 * k) * fc];
            }
        }
    }
    }
    if (narrow) {
        if (i >= F) return;
        double* out = vbuf + P.rbase[js] * nrhs + (int64_t)r0 * F + i;
#pragma unroll
        for (int r = 0; r < NR; ++r)
            if (r < nr) out[(int64_t)r * F] = w[r] - acc[r];
        return;
    }
    // quarters 1 .. 3 through shared memory (all four when a thread finishes
    // one right-hand side), then thread (row, q) takes r = q, q + 4, ..
    if constexpr (M == 1) {
#pragma unroll
        for (int r = 0; r < NR; ++r) part[q][r][row] = acc[r];
        __syncthreads();
        if (i >= F || q >= nr) return;
        const double s = (part[0][q][row] + part[1][q][row]) + (part[2][q][row] + part[3][q][row]);
        if (ncc == 1)
            vbuf[P.rbase[js] * nrhs + (int64_t)(r0 + q) * F + i] = w[0] - s;
        else
            pbuf[(P.fwd_off[js] + (int64_t)cc * (F - S) + (i - S)) * nrp + r0 + q] = s;
    } else {
        if (q)
#pragma unroll
            for (int r = 0; r < NR; ++r) part[q - 1][r][row] = acc[r];
        __syncthreads();
        if (q == 0)
#pragma unroll
            for (int r = 0; r < NR; ++r)
                part[0][r][row] = (acc[r] + part[0][r][row]) + (part[1][r][row] + part[2][r][row]);
        __syncthreads();
        if (i >= F) return;
#pragma unroll
        for (int k = 0; k < NR / 4; ++k) {
            const int r = q + 4 * k;
            if (r >= nr) break;
            const double s = part[0][r][row];
            if (ncc == 1)
                vbuf[P.rbase[js] * nrhs + (int64_t)(r0 + r) * F + i] = w[k] - s;
            else
                pbuf[(P.fwd_off[js] + (int64_t)cc * (F - S) + (i - S)) * nrp + r0 + r] = s;
        }
    }
}

// thread per (row, right-hand side) of the fronts with several column tiles
__global__ void k_fwd_rect_sum(const Job* jobs, int64_t njobs, const int32_t* tmap, int64_t ntasks, PV P, double* vbuf,
                               const double* pbuf, const double* b, int64_t ldb, int nrhs, int nrp) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t task = t / nrhs;
    const int r = (int)(t % nrhs);
    if (task >= ntasks) return;
    const Job& jb = job_of(jobs, njobs, tmap, task);
    const int js = jb.node;
    if (node_off(P, js)) return;
    const int F = P.F[js], S = P.S[js];
    const int row = S + (int)(task - jb.task0);
    const int ncc = (S + kFwdCols - 1) / kFwdCols;
    const double* part = pbuf + (P.fwd_off[js] + (row - S)) * nrp + r;
    const double w = gather_row(P, vbuf, b, ldb, nrhs, js, row, r);
    double v = 0.0;
#pragma unroll 8
    for (int k = 0; k < ncc; ++k) v += __ldcg(part + (int64_t)k * (F - S) * nrp);
    vbuf[P.rbase[js] * nrhs + (int64_t)r * F + row] = w - v;
}

// Back sweep, update rows [S, F): partial sums of L[S:F, c]' x[S:F].  One CTA
// per (kRectCols columns, kRectRows rows) and group stages the ancestors'
// solution rows in shared memory once and writes one partial dot product per
// column (a warp per CG columns at a time, lanes along the rows); k_bwd_tri adds
// a column's partials in a fixed order.
// kOnce: one group, so L is read once
template <int NG, bool kOnce>
__global__ void __launch_bounds__(256) k_bwd_rect(const Job* jobs, int64_t njobs, const int32_t* tmap, PV P,
                                                  double* pbuf, const double* b, int64_t ldb, int nrhs, int nrp) {
    __shared__ double ws[NG][kRectRows];
    __shared__ double segs[8][4][NG];
    const int64_t task = blockIdx.x;
    const Job& jb = job_of(jobs, njobs, tmap, task);
    const int js = jb.node;
    if (node_off(P, js)) return;
    const int F = P.F[js], S = P.S[js];
    const int ncc = jb.k_hi, g = blockIdx.y;
    const int64_t u = task - jb.task0;
    const int cc = (int)(u % ncc), rc = (int)(u / ncc);
    const double* base = P.lnz + P.lnz_off[js];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rbeg = S + rc * kRectRows, nr = min(kRectRows, F - rbeg);
    if (tid < nr) {
        const int64_t row = P.rows[P.rbase[js] + rbeg + tid];
#pragma unroll
        for (int r = 0; r < NG; ++r) ws[r][tid] = g * NG + r < nrhs ? b[row + (g * NG + r) * ldb] : 0.0;
    }
    __syncthreads();
    double* part = pbuf + (P.rect_off[js] + (int64_t)rc * S) * nrp + g * NG;
    constexpr int cw = kRectCols / 8;
    constexpr int CG = 4, UR = 4;                      // columns and row steps with loads in flight
    // a front of few columns has fewer column groups than warps: the warps then
    // split the rows as well and the segments are added in shared memory
    const int ncg = (min(S, kRectCols) + CG - 1) / CG, nseg = ncg <= 1 ? 8 : ncg <= 2 ? 4 : ncg <= 4 ? 2 : 1;
    const int seg = nseg > 1 ? warp % nseg : 0, rows = kRectRows / nseg;
    const int a1 = nseg > 1 ? CG : cw;
    for (int a = 0; a < a1; a += CG) {
        const int c0 = cc * kRectCols + (nseg > 1 ? warp / nseg * CG : warp * cw + a);
        const bool any = c0 < S;
        if (!any && nseg == 1) break;
        const double* col[CG];
        bool cv[CG];
#pragma unroll
        for (int q = 0; q < CG; ++q) {
            cv[q] = c0 + q < S;
            const int c = cv[q] ? c0 + q : min(c0, S - 1);
            col[q] = base + lnz_col(c, F) - c + rbeg;
        }
        double acc[CG][NG];
#pragma unroll
        for (int q = 0; q < CG; ++q)
#pragma unroll
            for (int r = 0; r < NG; ++r) acc[q][r] = 0.0;
        const int i1 = any ? min(nr, (seg + 1) * rows) : 0;
#pragma unroll(UR)
        for (int i = seg * rows + lane; i < i1; i += 32) {
            double l[CG];
#pragma unroll
            for (int q = 0; q < CG; ++q) l[q] = kOnce ? __ldcs(col[q] + i) : __ldg(col[q] + i);
#pragma unroll
            for (int r = 0; r < NG; ++r) {
                const double x = ws[r][i];
#pragma unroll
                for (int q = 0; q < CG; ++q) acc[q][r] += l[q] * x;
            }
        }
#pragma unroll
        for (int q = 0; q < CG; ++q) {
            int r, om;
            const double v = warp_reduce_scatter<NG>(acc[q], lane, r, om);
            if ((lane & om) == 0) {
                if (nseg > 1) segs[warp][q][r] = v;
                else if (cv[q]) part[(int64_t)(c0 + q) * nrp + r] = v;
            }
        }
    }
    if (nseg > 1) {
        __syncthreads();
        const int e = tid;                                        // (column, right-hand side)
        if (e < ncg * CG * NG) {
            const int c = e / NG, r = e % NG;
            double v = 0.0;
            for (int k = 0; k < nseg; ++k) v += segs[c / CG * nseg + k][c % CG][r];
            if (c < S) part[(int64_t)c * nrp + r] = v;
        }
    }
}

// ---------------------------------------------------------------------------
// Triangles of the solves as one dataflow launch per level.  Task (js, rb,
// group) is the 64-row block rb of front js (rows [64 rb, 64 rb + 64) of [0, S))
// for one group of right-hand sides.  Forward: y_rb = X_rb (w_rb - sum_{b < rb}
// L[rb, b] y_b), X_rb = L_rb,rb^-1 (the stored 64x64 inverse), w_rb gathered
// here, B = D^-1 y; backward: x_cb = X_cb' (w_cb - sum_{r > cb} L[r, cb]' x_r).
// Persistent CTAs take tasks in order from a counter (forward block-major
// ascending, backward descending), so a task only waits for tasks taken before
// it, by CTAs that are running: the waits always end.
// The chain of a front's blocks bounds it, one hand-over per block, so the
// values themselves say that they are there: the y array is filled with
// kNoValue (a NaN no computation produces; a NaN result is stored as
// another), a consumer thread takes its value with one load, prefetched a block
// ahead, and repeats it while it is missing.  48^3, 4 right-hand sides: 2.0 and
// 2.45 ms a sweep; with a flag per block (store, fence, flag; poll, barrier, load)
// 2.7 and 3.1 ms.  The groups keep one task at 4 right-hand sides: 24^3, 40 of
// them, both sweeps 1.6 ms in one pass, 10.7 ms in three passes of 16.
// Each wait is bounded (PV::wait_ns); one that gives up sets
// Stats::solve_timeout and an abort word every waiting thread checks, and the
// host turns it into an error.  Per tile, a thread owns one row (forward) or
// one column (backward) and a quarter of the 64 columns (rows).
// ---------------------------------------------------------------------------
constexpr unsigned long long kNoValue = 0xffffffffffffffffull;

__device__ __forceinline__ double ld_value(const double* p) {
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_value(double* p, double v) {
    if (v != v) v = __longlong_as_double(0x7ff8000000000000ll);
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
__device__ __forceinline__ bool no_value(double v) { return (unsigned long long)__double_as_longlong(v) == kNoValue; }
__device__ __forceinline__ unsigned long long tri_now() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// waits (bounded) for the value at p; ok = false when the launch aborts
__device__ __forceinline__ double tri_wait(const double* p, int* abort_word, const PV& P, bool& ok) {
    const unsigned long long t0 = tri_now();
    for (int spin = 1;; ++spin) {
        const double v = ld_value(p);
        if (!no_value(v)) return v;
        if ((spin & 15) == 0) {
            if (*(volatile int*)abort_word) break;
            if (tri_now() - t0 > P.wait_ns) {
                atomicExch(&P.st->solve_timeout, 1);
                atomicExch(abort_word, 1);
                break;
            }
        }
    }
    ok = false;
    return 0.0;
}

template <int NG>
__global__ void __launch_bounds__(256) k_fwd_tri(const int32_t* tasks, int ntasks, int ng, int32_t* counter, PV P,
                                                 const double* vbuf, double* y, double* b, int64_t ldb, int nrhs,
                                                 int64_t neq) {
    __shared__ __align__(16) double ys[2][kNB * NG];
    __shared__ double part[4][NG][kNB];
    __shared__ int task_sh;
    int* abort_word = counter + 1;
    const int tid = threadIdx.x, row = tid & (kNB - 1), q = tid >> 6;
    for (;;) {
        if (tid == 0) task_sh = atomicAdd(counter, 1);
        __syncthreads();
        const int t = task_sh;
        if (t >= ntasks * ng) break;
        const int js = tasks[2 * (t / ng)], rb = tasks[2 * (t / ng) + 1], g = t % ng;
        if (node_off(P, js)) {
            __syncthreads();                                          // all have read task_sh
            continue;
        }
        const int F = P.F[js], S = P.S[js];
        const int r0 = rb * kNB, nrow = min(kNB, S - r0);
        const double* base = P.lnz + P.lnz_off[js];
        double* yf = y + ((int64_t)g * neq + P.fst[js]) * NG;              // the front's y
        // what needs no other task: this row's X entries (the product with the
        // block inverse at the end), the gathered right-hand side and the pivot
        const double* lv = P.linv + P.linv_off[js] + (int64_t)rb * kNB * kNB;
        double xr[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const int m = 16 * q + k;
            xr[k] = (m <= row) ? __ldg(lv + row + m * kNB) : 0.0;         // X[row][m], unit lower
        }
        const int rr = g * NG + q;                                        // thread (row, q < NG) finishes entry (row, q)
        const bool fin = q < NG && row < nrow;
        double w = 0.0, d = 1.0;
        if (fin && rr < nrhs) {
            w = gather_row(P, vbuf, b, ldb, nrhs, js, r0 + row, rr);
            d = base[lnz_col(r0 + row, F)];
        }
        double acc[NG];
#pragma unroll
        for (int r = 0; r < NG; ++r) acc[r] = 0.0;
        bool ok = true;
        double next = (tid < kNB * NG && rb > 0) ? ld_value(yf + tid) : 0.0;
        for (int blk = 0; blk < rb; ++blk) {
            // this thread's 16 entries of the tile L[rb, blk], ahead of the wait
            double lr[16];
            {
                const int c0 = kNB * blk + 16 * q;
                int64_t p = lnz_col(c0, F) - c0 + r0 + row;               // L[r0 + row][c0]
#pragma unroll
                for (int k = 0; k < 16; ++k) {
                    lr[k] = (row < nrow) ? __ldg(base + p) : 0.0;
                    p += F - (c0 + k) - 1;                                // next column, same row
                }
            }
            double* yb = ys[blk & 1];
            if (tid < kNB * NG) {
                const double* at = yf + (int64_t)kNB * NG * blk + tid;
                double v = next;
                if (no_value(v)) v = tri_wait(at, abort_word, P, ok);
                yb[tid] = v;
                if (blk + 1 < rb) next = ld_value(at + kNB * NG);
            }
            if (!__syncthreads_and(ok)) {
                ok = false;
                break;
            }
#pragma unroll
            for (int k = 0; k < 16; ++k)
#pragma unroll
                for (int r = 0; r < NG; ++r) acc[r] += lr[k] * yb[(16 * q + k) * NG + r];
        }
        if (!ok) break;
        // v = w - sum of the four quarters, then y = X v
#pragma unroll
        for (int r = 0; r < NG; ++r) part[q][r][row] = acc[r];
        __syncthreads();
        if (q < NG) ys[0][row * NG + q] = w - ((part[0][q][row] + part[1][q][row]) + (part[2][q][row] + part[3][q][row]));
        __syncthreads();
#pragma unroll
        for (int r = 0; r < NG; ++r) acc[r] = 0.0;
#pragma unroll
        for (int k = 0; k < 16; ++k)
#pragma unroll
            for (int r = 0; r < NG; ++r) acc[r] += xr[k] * ys[0][(16 * q + k) * NG + r];
#pragma unroll
        for (int r = 0; r < NG; ++r) part[q][r][row] = acc[r];
        __syncthreads();
        if (fin) {
            const double v = (part[0][q][row] + part[1][q][row]) + (part[2][q][row] + part[3][q][row]);
            // (watchdog test switch: the first task of the launch never reports)
            if (!(P.tc_drop && t == 0)) st_value(yf + (int64_t)(r0 + row) * NG + q, v);
            if (rr < nrhs) b[(int64_t)(P.fst[js] + r0 + row) + rr * ldb] = v / d;
        }
    }
}

template <int NG>
__global__ void __launch_bounds__(256) k_bwd_tri(const int32_t* tasks, int ntasks, int ng, int32_t* counter, PV P,
                                                 const double* pbuf, double* x, double* b, int64_t ldb, int nrhs,
                                                 int nrp, int64_t neq) {
    __shared__ __align__(16) double xs[2][kNB * NG];
    __shared__ double part[4][NG][kNB];
    __shared__ int task_sh;
    int* abort_word = counter + 1;
    const int tid = threadIdx.x, col = tid & (kNB - 1), q = tid >> 6;
    for (;;) {
        if (tid == 0) task_sh = atomicAdd(counter, 1);
        __syncthreads();
        if (task_sh >= ntasks * ng) break;
        const int t = ntasks * ng - 1 - task_sh;                         // descending blocks
        const int js = tasks[2 * (t / ng)], cb = tasks[2 * (t / ng) + 1], g = t % ng;
        if (node_off(P, js)) {
            __syncthreads();
            continue;
        }
        const int F = P.F[js], S = P.S[js];
        const int c0 = cb * kNB, ncol = min(kNB, S - c0);
        const int nblk = (S + kNB - 1) / kNB;
        const double* base = P.lnz + P.lnz_off[js];
        double* xf = x + ((int64_t)g * neq + P.fst[js]) * NG;
        const int64_t pc = (col < ncol) ? lnz_col(c0 + col, F) - (c0 + col) : 0;   // column c0 + col, row 0
        const double* lv = P.linv + P.linv_off[js] + (int64_t)cb * kNB * kNB;
        double xr[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const int m = 16 * q + k;
            xr[k] = (m >= col) ? __ldg(lv + m + col * kNB) : 0.0;         // X[m][col]
        }
        // own row less the partial sums of the rows below the triangle
        const int rr = g * NG + q;
        const bool fin = q < NG && col < ncol;
        double w = 0.0;
        if (fin && rr < nrhs) {
            const int nrc = (F - S + kRectRows - 1) / kRectRows;
            const double* pp = pbuf + (P.rect_off[js] + c0 + col) * nrp + rr;
            double s = 0.0;
#pragma unroll 8
            for (int k = 0; k < nrc; ++k) s += __ldcg(pp + (int64_t)k * S * nrp);
            w = b[(int64_t)(P.fst[js] + c0 + col) + rr * ldb] - s;
        }
        double acc[NG];
#pragma unroll
        for (int r = 0; r < NG; ++r) acc[r] = 0.0;
        bool ok = true;
        // the blocks below finish from the bottom up: taken in that order, so
        // that only the nearest one (cb + 1, the last to finish) is waited for;
        // the last block may be short: its missing rows count as zero
        const int nlast = S - (nblk - 1) * kNB;
        double next = 0.0;
        if (tid < kNB * NG && cb + 1 < nblk && tid < nlast * NG) next = ld_value(xf + (int64_t)kNB * NG * (nblk - 1) + tid);
        for (int rb = nblk - 1; rb > cb; --rb) {
            const int nr = rb == nblk - 1 ? nlast : kNB;
            double lr[16];                                   // L[64 rb + 16 q + k][c0 + col], ahead of the wait
            {
                const int i0 = kNB * rb + 16 * q;
#pragma unroll
                for (int k = 0; k < 16; ++k) lr[k] = (col < ncol && 16 * q + k < nr) ? __ldg(base + pc + i0 + k) : 0.0;
            }
            double* xb = xs[rb & 1];
            if (tid < kNB * NG) {
                const double* at = xf + (int64_t)kNB * NG * rb + tid;
                double v = next;
                if (tid < nr * NG && no_value(v)) v = tri_wait(at, abort_word, P, ok);
                xb[tid] = v;
                if (rb - 1 > cb) next = ld_value(at - kNB * NG);
            }
            if (!__syncthreads_and(ok)) {
                ok = false;
                break;
            }
#pragma unroll
            for (int k = 0; k < 16; ++k)
#pragma unroll
                for (int r = 0; r < NG; ++r) acc[r] += lr[k] * xb[(16 * q + k) * NG + r];
        }
        if (!ok) break;
#pragma unroll
        for (int r = 0; r < NG; ++r) part[q][r][col] = acc[r];
        __syncthreads();
        if (q < NG) xs[0][col * NG + q] = w - ((part[0][q][col] + part[1][q][col]) + (part[2][q][col] + part[3][q][col]));
        __syncthreads();
        // x = X' v: x[col] = sum_{m >= col} X[m][col] v[m]
#pragma unroll
        for (int r = 0; r < NG; ++r) acc[r] = 0.0;
#pragma unroll
        for (int k = 0; k < 16; ++k)
#pragma unroll
            for (int r = 0; r < NG; ++r) acc[r] += xr[k] * xs[0][(16 * q + k) * NG + r];
#pragma unroll
        for (int r = 0; r < NG; ++r) part[q][r][col] = acc[r];
        __syncthreads();
        if (fin) {
            const double v = (part[0][q][col] + part[1][q][col]) + (part[2][q][col] + part[3][q][col]);
            if (!(P.tc_drop && t == ntasks * ng - 1)) st_value(xf + (int64_t)(c0 + col) * NG + q, v);
            if (rr < nrhs) b[(int64_t)(P.fst[js] + c0 + col) + rr * ldb] = v;
        }
    }
}

// ---------------------------------------------------------------------------
// Cholesky form (SPRFC2, src/SPR/sprfc2.f:1013-1032): column j of C is
// L(:, j) sqrt(d_j) with sqrt(d_j) on the diagonal and in D; back again, d_j =
// c_jj^2 and L(:, j) = C(:, j) / c_jj.  Retained fronts are left as assembled.
// One CTA per supernode, one warp per column of the packed trapezoid.
// ---------------------------------------------------------------------------
template <bool TO_CHOL>
__global__ void k_chol_convert(PV P, int64_t nsuper) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    for (int64_t js = blockIdx.x; js < nsuper; js += gridDim.x) {
        if (is_retained(P, (int)js)) continue;
        const int S = P.S[js], F = P.F[js], fst = P.fst[js];
        double* base = P.lnz + P.lnz_off[js];
        for (int j = warp; j < S; j += nwarp) {
            double* col = base + lnz_col(j, F);          // col[0] is the diagonal
            const double x = col[0];
            const double diag = TO_CHOL ? sqrt(x) : x * x;
            const double sc = TO_CHOL ? diag : 1.0 / x;
            for (int i = 1 + lane; i < F - j; i += 32) col[i] *= sc;
            __syncwarp();
            if (lane == 0) {
                col[0] = diag;
                P.dvec[fst + j] = diag;
            }
        }
    }
}

// b(i, r) times sqrt(d_i) (divide = 0) or divided by it, where d_i > 0:
// C^-1 b = D^1/2 (D^-1 L^-1 b) after the L D L' forward sweep, and
// C^-T y = L^-T (D^-1/2 y) before the back sweep (SPRFS9/SPRBS9,
// sprfs2.f:575-610, sprbs2.f:500-540, with C = L D^1/2).
__global__ void k_scale_sqrt_d(const double* dvec, double* b, int64_t ldb, int64_t n, int64_t nrhs, int divide) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n * nrhs;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = e % n, r = e / n;
        const double d = dvec[i];
        if (d > 0.0) {
            const double sq = sqrt(d);
            double* x = b + i + r * ldb;
            *x = divide ? *x / sq : *x * sq;
        }
    }
}

// ---------------------------------------------------------------------------
// Residual of the FP64 matrix for iterative refinement (the product SPRPRQ
// forms from the packed pattern, src/SPR/sprprm.f:243-325): the nonzeros of
// the assembled LNZ are compacted once into a full symmetric CSR with rows
// sorted by column, so r = b - K x is a deterministic warp-per-row SpMV.
// ---------------------------------------------------------------------------
//
// The build is bound by two reads of LNZ (8 bytes per entry each), so a warp
// takes one column at a time and the columns of all supernodes run at once:
// a 32^3 pass with it 42 ms against 770 ms with a warp per supernode (whose root, 6,867
// columns, one warp scanned alone) and a serial insertion sort per row.
// Rows come out of the atomics in any order; k_csr_rank puts each entry at the
// number of smaller columns in its row, so the result does not depend on it.

// supernode of an equation (P.fst increases)
__device__ __forceinline__ int supernode_of(const PV& P, int64_t nsuper, int64_t eq) {
    int64_t lo = 0, hi = nsuper - 1;
    while (lo < hi) {
        const int64_t mid = (lo + hi + 1) >> 1;
        if (P.fst[mid] <= eq) lo = mid;
        else hi = mid - 1;
    }
    return (int)lo;
}

__global__ void k_csr_count(PV P, int64_t nsuper, int64_t neq, int* rowcnt) {
    const int lane = threadIdx.x & 31;
    for (int64_t c = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; c < neq;
         c += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        const int js = supernode_of(P, nsuper, c);
        const int F = P.F[js], j = (int)(c - P.fst[js]);
        const int32_t* rows = P.rows + P.rbase[js];
        const double* cj = P.lnz + P.lnz_off[js] + lnz_col(j, F) - j;
        int upper = 0;                                   // nonzeros of row c right of the diagonal
        for (int i0 = j + lane; i0 < F; i0 += 128) {
            double a[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) a[u] = i0 + 32 * u < F ? __ldcs(cj + i0 + 32 * u) : 0.0;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (a[u] != 0.0) {
                    atomicAdd(&rowcnt[rows[i0 + 32 * u]], 1);
                    upper += i0 + 32 * u != j;
                }
        }
        for (int o = 16; o > 0; o >>= 1) upper += __shfl_xor_sync(0xffffffffu, upper, o);
        if (lane == 0 && upper) atomicAdd(&rowcnt[c], upper);
    }
}

// rowptr = exclusive prefix sums of cnt, fill = the same (the fill's cursors);
// one CTA, 1024 counts a step
__global__ void __launch_bounds__(1024) k_csr_scan(const int* cnt, int64_t n, int64_t* rowptr, int64_t* fill) {
    __shared__ int64_t warp_sum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t base = 0;
    for (int64_t i0 = 0; i0 < n; i0 += blockDim.x) {
        const int64_t i = i0 + threadIdx.x;
        const int64_t v = i < n ? cnt[i] : 0;
        int64_t s = v;
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t t = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += t;
        }
        if (lane == 31) warp_sum[warp] = s;
        __syncthreads();
        if (warp == 0) {
            int64_t w = warp_sum[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const int64_t t = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += t;
            }
            warp_sum[lane] = w;
        }
        __syncthreads();
        const int64_t at = base + s - v + (warp ? warp_sum[warp - 1] : 0);
        if (i < n) rowptr[i] = fill[i] = at;
        base += warp_sum[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) rowptr[n] = base;
}

__global__ void k_csr_fill(PV P, int64_t nsuper, int64_t neq, int64_t* fill, int32_t* ci, double* cv) {
    const int lane = threadIdx.x & 31;
    unsigned long long* cur = reinterpret_cast<unsigned long long*>(fill);
    for (int64_t c = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; c < neq;
         c += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        const int js = supernode_of(P, nsuper, c);
        const int F = P.F[js], j = (int)(c - P.fst[js]);
        const int32_t* rows = P.rows + P.rbase[js];
        const double* cj = P.lnz + P.lnz_off[js] + lnz_col(j, F) - j;
        for (int i0 = j + lane; i0 < F; i0 += 128) {
            double a[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) a[u] = i0 + 32 * u < F ? __ldcs(cj + i0 + 32 * u) : 0.0;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (a[u] == 0.0) continue;
                const int i = i0 + 32 * u, row = rows[i];
                int64_t p = (int64_t)atomicAdd(&cur[row], 1ull);
                ci[p] = (int32_t)c;
                cv[p] = a[u];
                if (i != j) {
                    p = (int64_t)atomicAdd(&cur[c], 1ull);
                    ci[p] = row;
                    cv[p] = a[u];
                }
            }
        }
    }
}

// a warp per row: sorts it by column (an entry's place is the number of
// smaller columns in the row) and forms the row's sum of |a|, whose maximum
// over the rows is the matrix norm (sums that are NaN are left out)
__global__ void k_csr_rank(const int64_t* rowptr, int64_t neq, const int32_t* ci, const double* cv, int32_t* co,
                           double* vo, unsigned long long* norm) {
    const int lane = threadIdx.x & 31;
    for (int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; r < neq;
         r += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        const int64_t p0 = rowptr[r], p1 = rowptr[r + 1];
        double sabs = 0.0;
        for (int64_t p = p0 + lane; p < p1; p += 32) {
            const int32_t c = ci[p];
            int64_t at = p0;
            for (int64_t q = p0; q < p1; ++q) at += ci[q] < c;
            co[at] = c;
            vo[at] = cv[p];
        }
        __syncwarp();                                        // the sum in the columns' order
        for (int64_t p = p0 + lane; p < p1; p += 32) sabs += fabs(vo[p]);
        for (int o = 16; o > 0; o >>= 1) sabs += __shfl_xor_sync(0xffffffffu, sabs, o);
        if (lane == 0 && sabs == sabs) atomicMax(norm, (unsigned long long)__double_as_longlong(sabs));
    }
}

__device__ __forceinline__ void atomic_max_nonneg(double* addr, double v) {
    atomicMax(reinterpret_cast<unsigned long long*>(addr), (unsigned long long)__double_as_longlong(v));
}

// r = b - K x for up to NR right-hand sides in one pass over each row (a warp
// per row, rows taken grid-stride).  Per right-hand side the products of a
// row are added in the same order as a pass per right-hand side would add
// them (lane-strided, then the xor tree).  norms[3q..3q+2] = max|r|, max|x|,
// max|b|: kept per warp in shared memory and reduced per CTA before one
// atomic each; the maxima compare bit patterns, so a NaN ranks above every
// number, as in the atomic.
constexpr int kResThreads = 256;
__device__ __forceinline__ double max_nonneg(double a, double v) {
    return __double_as_longlong(v) > __double_as_longlong(a) ? v : a;
}
template <int NR>
__global__ void __launch_bounds__(kResThreads) k_residual(const int64_t* rowptr, const int32_t* ci, const double* cv,
                                                          int64_t neq, const double* b, const double* x, double* r,
                                                          int64_t ld, int nrhs, double* norms) {
    constexpr int kW = kResThreads / 32;
    __shared__ double red[kW][3 * NR];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0)
        for (int e = 0; e < 3 * NR; ++e) red[warp][e] = 0.0;
    const int64_t stride = (int64_t)gridDim.x * kW;
    for (int64_t row = (int64_t)blockIdx.x * kW + warp; row < neq; row += stride) {
        const int64_t p0 = rowptr[row], p1 = rowptr[row + 1];
        double acc[NR];
#pragma unroll
        for (int q = 0; q < NR; ++q) acc[q] = 0.0;
        for (int64_t p = p0 + lane; p < p1; p += 32) {
            const double v = cv[p];
            const int64_t c = ci[p];
#pragma unroll
            for (int q = 0; q < NR; ++q)
                if (q < nrhs) acc[q] += v * x[c + q * ld];
        }
#pragma unroll
        for (int q = 0; q < NR; ++q)
            if (q < nrhs)
                for (int o = 16; o > 0; o >>= 1) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
        if (lane == 0)
#pragma unroll
            for (int q = 0; q < NR; ++q)
                if (q < nrhs) {
                    const double bi = b[row + q * ld], ri = bi - acc[q];
                    r[row + q * ld] = ri;
                    red[warp][3 * q] = max_nonneg(red[warp][3 * q], fabs(ri));
                    red[warp][3 * q + 1] = max_nonneg(red[warp][3 * q + 1], fabs(x[row + q * ld]));
                    red[warp][3 * q + 2] = max_nonneg(red[warp][3 * q + 2], fabs(bi));
                }
    }
    __syncthreads();
    if (threadIdx.x < 3 * nrhs && threadIdx.x < 3 * NR) {
        double m = 0.0;
        for (int w = 0; w < kW; ++w) m = max_nonneg(m, red[w][threadIdx.x]);
        atomic_max_nonneg(&norms[threadIdx.x], m);
    }
}

__global__ void k_axpy(double* x, const double* d, int64_t n) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) x[i] += d[i];
}

// ---------------------------------------------------------------------------
// Engine
// ---------------------------------------------------------------------------
#define TMAP(l) ((l).map_begin >= 0 ? d_->task_map + (l).map_begin : nullptr)
// Copy plan of the streamed factorisation.  Levels below L1 form group 0; each
// level L >= L1 is group L - L1 + 1 (L1 is the lowest level with at most
// kMaxTopNodes supernodes at or above it, so the copies stay few).  A group's
// LNZ ranges are its supernodes' blocks, adjacent blocks merged; group 0 is
// the gaps between the others.
struct Engine::Transfer {
    static constexpr int64_t kMaxTopNodes = 1024;
    int L1 = 0;
    std::vector<std::vector<std::pair<int64_t, int64_t>>> ranges;   // per group: (LNZ offset, doubles)
    std::vector<cudaEvent_t> up, done;                             // per group
    cudaStream_t ups = nullptr;                                    // uploads (the caller's copy stream: downloads)
    // the last level's super-panels come back as they become final: per panel
    // step, the LNZ ranges of the super-panels ending there and their event
    int32_t early_level = -1;
    std::vector<std::vector<std::pair<int64_t, int64_t>>> spranges;
    std::vector<cudaEvent_t> spev;
    // per group, the download ranges: the upload ranges without the early
    // fronts' LNZ
    std::vector<std::vector<std::pair<int64_t, int64_t>>> dranges;
    // the early fronts and a device copy of their uploaded LNZ: a front whose
    // pivot fails later gets its original columns back, in the device LNZ and
    // on the host, as a factorisation without early writes leaves them
    std::vector<int32_t> early_nodes;
    std::vector<std::pair<int64_t, int64_t>> early_ranges;      // LNZ offset, doubles (backup offsets: running sum)
    double* d_backup = nullptr;
    cudaEvent_t start = nullptr, fin = nullptr;
    cudaEvent_t ts = nullptr, tu = nullptr, tf = nullptr, te = nullptr;   // timing: start, group 0 up, factor end, last download
    cudaEvent_t tf0 = nullptr;                                            // timing: factorisation start
    std::vector<int64_t> diag_pos;                                 // LNZ offset of each equation's diagonal
    double* h_diag = nullptr;                                      // pinned
    double* d_diag = nullptr;
    ~Transfer() {
        if (ups) cudaStreamDestroy(ups);
        for (cudaEvent_t e : spev) cudaEventDestroy(e);
        if (d_backup) cudaFree(d_backup);
        for (cudaEvent_t e : up) cudaEventDestroy(e);
        for (cudaEvent_t e : done) cudaEventDestroy(e);
        if (start) cudaEventDestroy(start);
        if (fin) cudaEventDestroy(fin);
        if (ts) cudaEventDestroy(ts);
        if (tu) cudaEventDestroy(tu);
        if (te) cudaEventDestroy(te);
        if (tf) cudaEventDestroy(tf);
        if (tf0) cudaEventDestroy(tf0);
        if (h_diag) cudaFreeHost(h_diag);
        if (d_diag) cudaFree(d_diag);
    }
    int group(int32_t level) const { return level < L1 ? 0 : level - L1 + 1; }
};

Engine::Engine() : d_(new Dev()) {
    const char* e = getenv("SPR_B200_GRAPHS");
    use_graphs_ = !(e && e[0] == '0');
}

cudaGraphExec_t Engine::find_graph(const GraphKey& k) {
    for (auto& g : graphs_)
        if (g.key == k) return g.exec;
    return nullptr;
}

int64_t Engine::graph_launches(const GraphKey& k) {
    for (auto& g : graphs_)
        if (g.key == k) return g.launches;
    return 0;
}

void Engine::store_graph(const GraphKey& k, cudaGraphExec_t exec, int64_t launches) {
    if (graphs_.size() >= 16) {
        cudaGraphExecDestroy(graphs_.front().exec);
        graphs_.erase(graphs_.begin());
    }
    graphs_.push_back(GraphEntry{k, exec, launches});
}
// The solves' graphs (the factorisation's have no B in their key).
void Engine::drop_solve_graphs() {
    for (auto& g : graphs_)
        if (g.key.b) cudaGraphExecDestroy(g.exec);
    graphs_.erase(std::remove_if(graphs_.begin(), graphs_.end(), [](const GraphEntry& g) { return g.key.b != nullptr; }),
                  graphs_.end());
}

Engine::~Engine() {
    for (auto& g : graphs_) cudaGraphExecDestroy(g.exec);
    for (cudaEvent_t e : d_->evpool) cudaEventDestroy(e);
    if (d_->side) cudaStreamDestroy(d_->side);
    if (d_->ahead) cudaStreamDestroy(d_->ahead);
    if (d_->wbs) cudaStreamDestroy(d_->wbs);
    if (d_->mbox) cudaFreeHost(d_->mbox);
    if (d_->slab) cudaFree(d_->slab);
    if (d_->slab_far) cudaFree(d_->slab_far);
    if (d_->tc_off) cudaFree(d_->tc_off);
    if (d_->i8_slab) cudaFree(d_->i8_slab);
    if (d_->i8_scales) cudaFree(d_->i8_scales);
    if (d_->sqd) cudaFree(d_->sqd);
    for (void* p : {(void*)csr_.rowptr, (void*)csr_.fill, (void*)csr_.cnt, (void*)csr_.ci, (void*)csr_.cv,
                    (void*)csr_.ci2, (void*)csr_.cv2})
        cudaFree(p);
    if (rbuf_) cudaFree(rbuf_);
    if (nbuf_) cudaFree(nbuf_);
    if (guard_copy_) cudaFree(guard_copy_);
    xfer_.reset();
    if (!d_) return;
    for (void* p : d_->owned) cudaFree(p);
    if (d_->arena) cudaFree(d_->arena);
    if (d_->vbuf) cudaFree(d_->vbuf);
    if (d_->ybuf) cudaFree(d_->ybuf);
    if (d_->pbuf) cudaFree(d_->pbuf);
    if (d_->ev0) cudaEventDestroy(d_->ev0);
    if (d_->ev1) cudaEventDestroy(d_->ev1);
}

int Engine::open(const int64_t* mspar, const int64_t* mtrees, const int64_t* msifa) {
    int rc = build_plan(mspar, mtrees, msifa, P_);
    if (rc != 0) return rc;
    Dev& D = *d_;
    auto& o = D.owned;
    int dev = 0;
    CK(cudaGetDevice(&dev));
    CK(cudaDeviceGetAttribute(&sm_count_, cudaDevAttrMultiProcessorCount, dev));
    {
        // side and look-ahead streams and the fork/join events of one
        // factorisation (two per step that forks a far or look-ahead update)
        size_t nev = 0;
        for (const LevelPlan& lp : P_.levels)
            for (size_t st = 0; st < lp.far.size(); ++st) {
                if (!lp.far[st].empty() || !lp.far_tc[st].empty()) nev += 2;
                if (!lp.ahead[st].empty()) nev += 2;
                if (st < lp.wb_sp.size() && lp.wb_sp[st].ntasks > 0) nev += 1;
            }
        // two each for two streams of a level's small fronts and for its write-back beside its large ones
        // (the solves use the same events again)
        nev += 6 * P_.levels.size();
        for (const LevelPlan& lp : P_.levels)           // the join after a level's early writes
            for (const Launch& w : lp.wb_sp)
                if (w.ntasks > 0) {
                    nev += 1;
                    break;
                }
        CK(cudaStreamCreateWithFlags(&D.side, cudaStreamNonBlocking));
        CK(cudaStreamCreateWithFlags(&D.ahead, cudaStreamNonBlocking));
        CK(cudaStreamCreateWithFlags(&D.wbs, cudaStreamNonBlocking));
        D.evpool.resize(nev);
        for (cudaEvent_t& e : D.evpool) CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
    if (dev_upload(o, &D.fst, P_.fst) || dev_upload(o, &D.S, P_.S) || dev_upload(o, &D.F, P_.F) ||
        dev_upload(o, &D.child_ptr, P_.child_ptr) || dev_upload(o, &D.child, P_.child) ||
        dev_upload(o, &D.rows, P_.rows) || dev_upload(o, &D.rel, P_.rel) ||
        dev_upload(o, &D.cchild, P_.cchild) || dev_upload(o, &D.ct, P_.ct) ||
        dev_upload(o, &D.buf_ld, P_.buf_ld) || dev_upload(o, &D.lnz_off, P_.lnz_off) ||
        dev_upload(o, &D.rel_off, P_.rel_off) || dev_upload(o, &D.rbase, P_.rbase) ||
        dev_upload(o, &D.cptr, P_.cptr) || dev_upload(o, &D.buf_off, P_.buf_off) ||
        dev_upload(o, &D.upd_off, P_.upd_off) || dev_upload(o, &D.jobs, P_.jobs) ||
        dev_upload(o, &D.linv_off, P_.linv_off) ||
        dev_upload(o, &D.rect_off, P_.rect_off) || dev_upload(o, &D.fwd_off, P_.fwd_off) ||
        dev_upload(o, &D.task_map, P_.task_map))
        return -4;
    CK(cudaMalloc((void**)&D.linv, std::max<int64_t>(P_.linv_doubles, 1) * sizeof(double)));
    o.push_back(D.linv);
    std::vector<int32_t> small;
    D.small_begin.clear();
    for (const LevelPlan& lp : P_.levels) {
        D.small_begin.push_back((int64_t)small.size());
        small.insert(small.end(), lp.small_nodes.begin(), lp.small_nodes.end());
    }
    if (dev_upload(o, &D.level_nodes, small)) return -4;
    D.ret = nullptr;
    if (P_.any_retained && dev_upload(o, &D.ret, P_.retained)) return -4;
    CK(cudaMalloc((void**)&D.arena, std::max<int64_t>(P_.arena_doubles, 32) * sizeof(double)));
    CK(cudaMalloc((void**)&D.adiag, P_.neq * sizeof(double)));
    o.push_back(D.adiag);
    CK(cudaMalloc((void**)&D.sn_neg, P_.nsuper * sizeof(int32_t)));
    o.push_back(D.sn_neg);
    CK(cudaMalloc((void**)&D.sn_fail, P_.nsuper * sizeof(int32_t)));
    o.push_back(D.sn_fail);
    CK(cudaMalloc((void**)&D.sn_bad, P_.nsuper * sizeof(int32_t)));
    o.push_back(D.sn_bad);
    CK(cudaMalloc((void**)&D.sn_faild, P_.nsuper * sizeof(double)));
    o.push_back(D.sn_faild);
    CK(cudaMalloc((void**)&D.sn_faila, P_.nsuper * sizeof(double)));
    o.push_back(D.sn_faila);
    CK(cudaMalloc((void**)&D.st, sizeof(Stats)));
    o.push_back(D.st);
    CK(cudaMalloc((void**)&D.hbuf, sizeof(unsigned long long)));
    o.push_back(D.hbuf);
    if (dev_upload(o, &D.tri_tasks, P_.tri_tasks)) return -4;
    CK(cudaMalloc((void**)&D.tri_sync, sizeof(int32_t) * (size_t)(2 * P_.levels.size() + 2)));
    o.push_back(D.tri_sync);
    CK(cudaHostAlloc((void**)&D.mbox, 32 * sizeof(unsigned long long), cudaHostAllocMapped));
    CK(cudaHostGetDevicePointer((void**)&D.mbox_dev, D.mbox, 0));
    CK(cudaEventCreate(&D.ev0));
    CK(cudaEventCreate(&D.ev1));
    int smem_max = 0;
    CK(cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    const size_t need = ((size_t)kSmallMaxF * (kSmallMaxF + 1) / 2 + 2 * kSmallMaxF) * sizeof(double);
    if ((size_t)smem_max < need) return -4;
    CK(cudaFuncSetAttribute(k_small_front<kPivotLDL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)need));
    CK(cudaFuncSetAttribute(k_small_front<kPivotReplace>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)need));
    CK(cudaFuncSetAttribute(k_small_front<kPivotChol>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)need));
    CK(cudaFuncSetAttribute(k_small_front<kPivotChol4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)need));
    CK(cudaFuncSetAttribute(k_trsm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrsmSmem));
    for (const void* f : {(const void*)k_diag<kPivotLDL>, (const void*)k_diag<kPivotReplace>, (const void*)k_diag<kPivotChol>,
                          (const void*)k_diag<kPivotChol4>})
        CK(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDiagSmem));
    for (const void* f : {(const void*)k_chain<kPivotLDL>, (const void*)k_chain<kPivotReplace>, (const void*)k_chain<kPivotChol>,
                          (const void*)k_chain<kPivotChol4>})
        CK(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kChainSmem));
    for (const void* f : {(const void*)k_forward<1>, (const void*)k_forward<2>, (const void*)k_forward<4>,
                          (const void*)k_backward<1>, (const void*)k_backward<2>, (const void*)k_backward<4>})
        CK(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallSolveSmem));
    CK(cudaFuncSetAttribute(K_GEMM_BIG, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GemmBig::smem));
    CK(cudaFuncSetAttribute(K_GEMM_SMALL, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GemmSmall::smem));
    CK(cudaFuncSetAttribute(K_GEMM_TINY, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GemmTiny::smem));
    CK(cudaFuncSetAttribute(k_gemm_x3, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GemmSmall::smem));
    CK(cudaFuncSetAttribute(k_gemm_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tc::kSmem));
    CK(cudaFuncSetAttribute(k_gemm_i8, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)i8::kSmemI8));
    set_int_min(i8_min_flops_);
    return 0;
}

void Engine::set_int_min(double flops) {
    i8_min_flops_ = flops;
    any_i8_ = false;
    for (const LevelPlan& lp : P_.levels) {
        for (const I8Launch& t : lp.trail_i8) any_i8_ |= t.gemm.ntasks > 0 && t.flops >= flops;
        any_i8_ |= !lp.outer_i8.empty() && lp.outer_i8[0].flops >= flops;
    }
}

// Operand slabs of the tensor-core updates and the 2-D TMA map over them:
// [slab_rows][32] fp32, box 32 x 128 rows, 128-byte swizzle.
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static int make_slab(Engine& eng, int64_t rows_needed, float** slab, CUtensorMap* map) {
    const int64_t rows = std::max<int64_t>(rows_needed, tc::kTM);
    if (rows >= (int64_t(1) << 31)) return -3;                 // TMA row coordinates are 32-bit
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn)
        return -4;
    CK(eng.alloc((void**)slab, rows * tc::kBK * sizeof(float)));
    const cuuint64_t dims[2] = {(cuuint64_t)tc::kBK, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)tc::kBK * sizeof(float)};
    const cuuint32_t box[2] = {(cuuint32_t)tc::kBK, (cuuint32_t)tc::kTM};
    const cuuint32_t es[2] = {1, 1};
    const CUresult r = ((EncodeTiledFn)fn)(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, *slab, dims, strides, box, es,
                                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        cudaFree(*slab);
        *slab = nullptr;
        return -4;
    }
    return 0;
}

int Engine::ensure_slabs() {
    Dev& D = *d_;
    if (D.slab && D.slab_far && D.tc_off) return 0;
    if (!D.tc_off) CK(alloc((void**)&D.tc_off, 2 * P_.nsuper * sizeof(int32_t)));
    if (!D.slab) {
        const int rc = make_slab(*this, P_.slab_rows, &D.slab, &D.slab_map);
        if (rc != 0) return rc;
    }
    if (!D.slab_far) return make_slab(*this, P_.slab_rows_far, &D.slab_far, &D.slab_map_far);
    return 0;
}


// Digit slabs of the integer updates: [i8_rows][128] bytes, one map with boxes of
// 128 rows (row tiles) and one with 64 (column tiles), 128-byte swizzle.
// Returns nonzero when they cannot be had.
int Engine::ensure_i8() {
    Dev& D = *d_;
    if (D.i8_slab) return 0;
    const int64_t rows = std::max<int64_t>(P_.i8_rows, i8::kM);
    if (rows >= (int64_t(1) << 31)) return -3;                 // TMA row coordinates are 32-bit
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn)
        return -4;
    uint8_t* slab = nullptr;
    if ((!D.sqd && cudaMalloc((void**)&D.sqd, P_.neq * 2 * sizeof(double)) != cudaSuccess) ||
        (!D.i8_scales &&
         cudaMalloc((void**)&D.i8_scales, std::max<int64_t>(P_.i8_scales, 1) * sizeof(double)) != cudaSuccess) ||
        cudaMalloc((void**)&slab, rows * i8::kK) != cudaSuccess) {
        cudaGetLastError();
        return -4;
    }
    const cuuint64_t dims[2] = {(cuuint64_t)i8::kK, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)i8::kK};
    const cuuint32_t es[2] = {1, 1};
    for (int m = 0; m < 2; ++m) {
        const cuuint32_t box[2] = {(cuuint32_t)i8::kK, (cuuint32_t)(m == 0 ? i8::kM : i8::kN)};
        const CUresult r = ((EncodeTiledFn)fn)(m == 0 ? &D.i8_map_a : &D.i8_map_b, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2,
                                               slab, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) {
            cudaFree(slab);
            return -4;
        }
    }
    D.i8_slab = slab;
    return 0;
}

void Engine::release_i8() {
    Dev& D = *d_;
    for (auto& g : graphs_)
        if (!g.key.b) cudaGraphExecDestroy(g.exec);              // factorisations captured on the slab
    graphs_.erase(std::remove_if(graphs_.begin(), graphs_.end(), [](const GraphEntry& g) { return g.key.b == nullptr; }),
                  graphs_.end());
    cudaFree(D.i8_slab);
    D.i8_slab = nullptr;
}

cudaError_t Engine::alloc(void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaSuccess && d_->i8_slab) {
        cudaGetLastError();
        release_i8();
        e = cudaMalloc(p, bytes);
    }
    if (e != cudaSuccess) *p = nullptr;
    return e;
}

static cudaEvent_t record_event(cudaStream_t s) {
    cudaEvent_t e = nullptr;
    cudaEventCreate(&e);
    cudaEventRecord(e, s);
    return e;
}

static PV make_view(Engine::Dev& D, const Plan& P, double* d_sm, double tol1) {
    PV v;
    v.fst = D.fst;
    v.S = D.S;
    v.F = D.F;
    v.child_ptr = D.child_ptr;
    v.child = D.child;
    v.rows = D.rows;
    v.rel = D.rel;
    v.cchild = D.cchild;
    v.ct = D.ct;
    v.buf_ld = D.buf_ld;
    v.lnz_off = D.lnz_off;
    v.rel_off = D.rel_off;
    v.rbase = D.rbase;
    v.cptr = D.cptr;
    v.buf_off = D.buf_off;
    v.upd_off = D.upd_off;
    v.arena = D.arena;
    v.dvec = d_sm;
    v.lnz = d_sm + P.neq;
    v.adiag = D.adiag;
    v.sn_neg = D.sn_neg;
    v.sn_fail = D.sn_fail;
    v.sn_bad = D.sn_bad;
    v.sn_faild = D.sn_faild;
    v.sn_faila = D.sn_faila;
    v.st = D.st;
    v.linv_off = D.linv_off;
    v.linv = D.linv;
    v.rect_off = D.rect_off;
    v.fwd_off = D.fwd_off;
    v.tol1 = tol1;
    v.fc3 = 0;
    v.tol4 = 0.0;
    v.dcor = nullptr;
    v.ret = D.ret;
    v.near_tol = 0.0;
    v.wait_ns = 2000000000ull;
    v.tc_drop = 0;
    v.adiag_in = nullptr;
    v.skip = D.skip_on ? D.skip : nullptr;
    v.sqd = D.sqd;
    return v;
}

// The streams of a level's small fronts beside its large ones: its classes in
// turn on the side and the look-ahead stream, the first on s where it has no
// large front.
struct Engine::SmallStreams {
    cudaStream_t t[2];
    cudaStream_t of(const LevelPlan& lp, const LevelPlan::SmallClass& c) const {
        return t[(&c - lp.small_classes.data()) & 1];
    }
};

Engine::SmallStreams Engine::small_streams(const LevelPlan& lp, cudaStream_t s, size_t& evi) {
    Dev& D = *d_;
    SmallStreams r{lp.large_nodes.empty() ? s : D.side, lp.small_classes.size() > 1 ? D.ahead : s};
    cudaEvent_t e = D.evpool[evi];
    if (r.t[0] != s || r.t[1] != s) {
        ++evi;
        cudaEventRecord(e, s);
    }
    for (cudaStream_t t : r.t)
        if (t != s) cudaStreamWaitEvent(t, e, 0);
    return r;
}

void Engine::join_small(const SmallStreams& r, cudaStream_t s, size_t& evi) {
    for (cudaStream_t t : r.t)
        if (t != s) {
            cudaEvent_t e = d_->evpool[evi++];
            cudaEventRecord(e, t);
            cudaStreamWaitEvent(s, e, 0);
        }
}

void Engine::launch_diag(const Launch& pl, cudaStream_t s, const PV& pv) {
    const Job* jobs = d_->jobs + pl.job_begin;
    const int n = (int)pl.job_count;
    if (pv.fc3 == 2) k_diag<kPivotChol4><<<n, 256, kDiagSmem, s>>>(jobs, pv, 1);
    else if (pv.fc3) k_diag<kPivotReplace><<<n, 256, kDiagSmem, s>>>(jobs, pv, 1);
    else if (chol_) k_diag<kPivotChol><<<n, 256, kDiagSmem, s>>>(jobs, pv, 1);
    else k_diag<kPivotLDL><<<n, 256, kDiagSmem, s>>>(jobs, pv, 1);
    ++timing.launches;
}

void Engine::launch_chain(const Launch& pl, cudaStream_t s, const PV& pv) {
    const Job* jobs = d_->jobs + pl.job_begin;
    const int n = (int)pl.ntasks;
    if (pv.fc3 == 2) k_chain<kPivotChol4><<<n, 256, kChainSmem, s>>>(jobs, pl.job_count, TMAP(pl), pv);
    else if (pv.fc3) k_chain<kPivotReplace><<<n, 256, kChainSmem, s>>>(jobs, pl.job_count, TMAP(pl), pv);
    else if (chol_) k_chain<kPivotChol><<<n, 256, kChainSmem, s>>>(jobs, pl.job_count, TMAP(pl), pv);
    else k_chain<kPivotLDL><<<n, 256, kChainSmem, s>>>(jobs, pl.job_count, TMAP(pl), pv);
    ++timing.launches;
}

void Engine::launch_gemm(const Launch& l, cudaStream_t s, const PV& pv, std::vector<cudaEvent_t>& gev) {
    if (l.ntasks <= 0) return;
    if (profile_) gev.push_back(record_event(s));
    const Job* jobs = d_->jobs + l.job_begin;
    if (mixed_ == 2) {
        k_gemm_x3<<<(int)l.ntasks, 128, GemmSmall::smem, s>>>(jobs, l.job_count, TMAP(l), pv);
    } else if (l.tile == kTileBig) {
        K_GEMM_BIG<<<(int)l.ntasks, GemmBig::NT, GemmBig::smem, s>>>(jobs, l.job_count, TMAP(l), pv);
    } else if (small_tile_ == kTileTiny && l.alt >= 0) {
        const Launch& a = P_.alt[l.alt];
        K_GEMM_TINY<<<(int)a.ntasks, GemmTiny::NT, GemmTiny::smem, s>>>(d_->jobs + a.job_begin, a.job_count,
                                                                       TMAP(a), pv);
    } else {
        K_GEMM_SMALL<<<(int)l.ntasks, GemmSmall::NT, GemmSmall::smem, s>>>(jobs, l.job_count, TMAP(l), pv);
    }
    if (profile_) gev.push_back(record_event(s));
    ++timing.launches;
    ++timing.gemm_launches;
}

void Engine::launch_tc(const TcLaunch& t, cudaStream_t s, const PV& pv, std::vector<cudaEvent_t>& gev, bool far) {
    if (t.gemm.ntasks <= 0) return;
    Dev& D = *d_;
    if (profile_) {
        tc_pairs_.push_back(gev.size());
        gev.push_back(record_event(s));
    }
    int32_t* off = D.tc_off + (far ? P_.nsuper : 0);
    k_split_tc<<<(int)t.split.ntasks, 256, 0, s>>>(D.jobs + t.split.job_begin, t.split.job_count, TMAP(t.split), pv,
                                                   far ? D.slab_far : D.slab, off);
    // a side-stream launch leaves a quarter of the SMs to the panel chain
    // (a persistent tensor-core CTA holds most of an SM's shared memory)
    const int cap = (far && !profile_) ? std::max(1, sm_count_ * far_cap_q_ / 4) : sm_count_;
    const int grid = (int)std::min<int64_t>(t.gemm.ntasks, cap);
    k_gemm_tc<<<grid, tc::kThreads, tc::kSmem, s>>>(D.jobs + t.gemm.job_begin, t.gemm.job_count, TMAP(t.gemm),
                                                    t.gemm.ntasks, pv, off,
                                                    far ? D.slab_map_far : D.slab_map);
    if (profile_) gev.push_back(record_event(s));
    timing.launches += 2;
    ++timing.gemm_launches;
}

// The integer-digit form of an update: the panel's digits, then the products.
void Engine::launch_i8_split(const I8Launch& t, cudaStream_t s, const PV& pv, std::vector<cudaEvent_t>& gev) {
    if (profile_) {
        tc_pairs_.push_back(gev.size());
        gev.push_back(record_event(s));
    }
    k_split_i8<<<(int)t.split.ntasks, 256, 0, s>>>(d_->jobs + t.split.job_begin, t.split.job_count, TMAP(t.split), pv,
                                                   d_->i8_slab, d_->i8_scales);
    if (profile_) gev.push_back(record_event(s));
    ++timing.launches;
}

void Engine::launch_i8_gemm(const Launch& l, cudaStream_t s, const PV& pv, std::vector<cudaEvent_t>& gev, bool far) {
    if (l.ntasks <= 0) return;
    Dev& D = *d_;
    if (profile_) {
        tc_pairs_.push_back(gev.size());
        gev.push_back(record_event(s));
    }
    // a side-stream launch leaves SMs to the panel chain (one CTA holds an SM's shared memory)
    const int cap = (far && !profile_) ? std::max(1, sm_count_ * i8_far_q_ / 8) : sm_count_;
    const int grid = (int)std::min<int64_t>(l.ntasks, cap);
    k_gemm_i8<<<grid, i8::kThreadsI8, i8::kSmemI8, s>>>(D.jobs + l.job_begin, l.job_count, TMAP(l), l.ntasks, pv,
                                                        D.i8_scales, D.i8_map_a, D.i8_map_b);
    if (profile_) gev.push_back(record_event(s));
    ++timing.launches;
    ++timing.gemm_launches;
}

// ---------------------------------------------------------------------------
// Split across GPUs: node mask and the exchange of subtree roots' update
// blocks (factor) and update vectors (forward solve).
// ---------------------------------------------------------------------------
int Engine::set_skip(const uint8_t* host_mask) {
    Dev& D = *d_;
    if (!host_mask) {
        D.skip_on = false;
        split_ = !fout_.empty() || !fin_.empty() || !vout_.empty() || !vin_.empty();
        return 0;
    }
    if (!D.skip) {
        CK(cudaMalloc((void**)&D.skip, std::max<int64_t>(P_.nsuper, 1)));
        D.owned.push_back(D.skip);
    }
    CK(cudaMemcpy(D.skip, host_mask, P_.nsuper, cudaMemcpyHostToDevice));
    D.skip_on = true;
    split_ = true;
    return 0;
}

void Engine::set_exchange(std::vector<Xfer> fo, std::vector<Xfer> fi, std::vector<Xfer> vo, std::vector<Xfer> vi) {
    fout_ = std::move(fo);
    fin_ = std::move(fi);
    vout_ = std::move(vo);
    vin_ = std::move(vi);
    split_ = d_->skip_on || !fout_.empty() || !fin_.empty() || !vout_.empty() || !vin_.empty();
}

// node js's update block <-> buf ((F-S) x (F-S), leading dimension F-S)
void Engine::block_copy(int32_t js, double* buf, bool out, cudaStream_t s) {
    const int64_t q = P_.F[js] - P_.S[js];
    if (q <= 0) return;
    double* blk = d_->arena + P_.upd_off[js];
    const size_t ld = (size_t)P_.buf_ld[js] * sizeof(double), w = (size_t)q * sizeof(double);
    if (out)
        cudaMemcpy2DAsync(buf, w, blk, ld, w, q, cudaMemcpyDeviceToDevice, s);
    else
        cudaMemcpy2DAsync(blk, ld, buf, w, w, q, cudaMemcpyDeviceToDevice, s);
}

// node js's forward update vector (rows [S, F) of its front vector, per RHS) <-> buf ((F-S) x nrhs)
void Engine::vec_copy(int32_t js, double* buf, bool out, int64_t nrhs, cudaStream_t s) {
    const int64_t f = P_.F[js], q = f - P_.S[js];
    if (q <= 0) return;
    double* v = d_->vbuf + P_.rbase[js] * nrhs + P_.S[js];
    const size_t ld = (size_t)f * sizeof(double), w = (size_t)q * sizeof(double);
    if (out)
        cudaMemcpy2DAsync(buf, w, v, ld, w, nrhs, cudaMemcpyDeviceToDevice, s);
    else
        cudaMemcpy2DAsync(v, ld, buf, w, w, nrhs, cudaMemcpyDeviceToDevice, s);
}

namespace {
// The exchange lists as level hooks: "in" entries before their parent's
// level, "out" entries after their node's level.
struct ExchangeHooks : LevelHooks {
    const Plan* P = nullptr;
    const std::vector<Engine::Xfer>* out = nullptr;
    const std::vector<Engine::Xfer>* in = nullptr;
    std::function<void(int32_t, double*, bool, cudaStream_t)> copy;
    void before(size_t L, cudaStream_t s) const override {
        for (const Engine::Xfer& x : *in) {
            const int32_t p = P->parent[x.node];
            if (p >= 0 && (size_t)P->level[p] == L) copy(x.node, x.buf, false, s);
        }
    }
    void after(size_t L, cudaStream_t s) const override {
        for (const Engine::Xfer& x : *out)
            if ((size_t)P->level[x.node] == L) copy(x.node, x.buf, true, s);
    }
};
}  // namespace

// Copies n 8-byte words to the mailbox (one thread per word).
__global__ void k_mailbox(const unsigned long long* src, int n, unsigned long long* dst) {
    const int i = threadIdx.x;
    if (i < n) dst[i] = src[i];
}

void Engine::enqueue_factor(const PV& pv, cudaStream_t s, std::vector<cudaEvent_t>& gev) {
    Dev& D = *d_;
    timing.launches = 0;
    timing.tc_flops = 0.0;
    auto mark = [&](int phase) {
        if (profile_) marks_.emplace_back(phase, record_event(s));
    };
    constexpr size_t kSteps = kSuperPanel / kNB;
    // side stream for the trailing-update columns beyond the next super-panel,
    // look-ahead stream for the in-super-panel columns after the next two panels
    // (profile mode keeps everything on one stream so the events time it)
    cudaStream_t u = (profile_ || !D.side) ? s : D.side;
    cudaStream_t la = (profile_ || !D.ahead) ? s : D.ahead;
    size_t evi = 0;
    cudaEvent_t far_done = nullptr, ahead_done[2] = {nullptr, nullptr};      // ahead: of even and odd steps
    auto join_far = [&]() {
        if (far_done) {
            cudaStreamWaitEvent(s, far_done, 0);
            far_done = nullptr;
        }
    };
    auto join_ahead = [&](size_t st) {
        if (ahead_done[st & 1]) {
            cudaStreamWaitEvent(s, ahead_done[st & 1], 0);
            ahead_done[st & 1] = nullptr;
        }
    };
    // A level's small fronts run beside its large ones (side stream), and its
    // write-back beside its K = S update and the next level, until the arena is
    // reused: a front's buffer is free again from the second level after its own.
    // With hooks a level's work is all on s when they are called.
    // 12^3 factor 2.67 -> 2.10 ms, 20^3 9.6 -> 9.0 ms, 512 boxes 29.1 -> 28.2 ms.
    const bool beside = u != s && !hooks_;
    cudaEvent_t wb_done[2] = {nullptr, nullptr};
    auto fork_to = [&](cudaStream_t t) {
        cudaEvent_t e = D.evpool[evi++];
        cudaEventRecord(e, s);
        cudaStreamWaitEvent(t, e, 0);
    };
    auto join_wb = [&](size_t L) {
        if (wb_done[L & 1]) cudaStreamWaitEvent(s, wb_done[L & 1], 0);
        wb_done[L & 1] = nullptr;
    };
    mark(0);
    k_prepass<<<(int)std::min<int64_t>((P_.nsuper * 32 + 255) / 256, 4736), 256, 0, s>>>(pv, P_.nsuper);
    k_reduce<false><<<1, 1024, 0, s>>>(D.adiag, P_.neq, &D.st->trace);
    timing.launches += 2;
    char lname[48];
    for (size_t L = 0; L < P_.levels.size(); ++L) {
        const LevelPlan& lp = P_.levels[L];
        snprintf(lname, sizeof lname, "factor level %zu", L);
        NvtxRange level_range(lname);
        trace_point(lname);
        if (hooks_) hooks_->before(L, s);
        struct AfterLevel {                      // runs at every exit of this iteration
            const LevelHooks* h;
            size_t L;
            cudaStream_t s;
            ~AfterLevel() {
                if (h) h->after(L, s);
            }
        } after_level{hooks_, L, s};
        join_wb(L);                              // of level L - 2
        SmallStreams small{s, s};
        if (!lp.small_nodes.empty()) {
            mark(1);
            if (beside) small = small_streams(lp, s, evi);
            for (const LevelPlan::SmallClass& c : lp.small_classes) {
                const int F = c.maxF;
                const size_t smem = ((size_t)F * (F + 1) / 2 + 2 * F) * sizeof(double);
                const int thr = small_threads(F);
                const int32_t* nodes = D.level_nodes + D.small_begin[L] + c.begin;
                cudaStream_t ss = small.of(lp, c);
                if (pv.fc3 == 2)
                    k_small_front<kPivotChol4><<<c.count, thr, smem, ss>>>(nodes, pv);
                else if (pv.fc3)
                    k_small_front<kPivotReplace><<<c.count, thr, smem, ss>>>(nodes, pv);
                else if (chol_)
                    k_small_front<kPivotChol><<<c.count, thr, smem, ss>>>(nodes, pv);
                else
                    k_small_front<kPivotLDL><<<c.count, thr, smem, ss>>>(nodes, pv);
                ++timing.launches;
            }
        }
        if (lp.large_nodes.empty()) {
            join_small(small, s, evi);
            continue;
        }
        const Job* jobs = D.jobs;
        const bool early = hooks_ && hooks_->early_columns(L);
        bool wrote_early = false;
        {
            mark(2);
            const Launch& l = lp.assemble;
            k_poison<<<(int)((l.job_count + 127) / 128), 128, 0, s>>>(jobs + l.job_begin, l.job_count, TMAP(l), pv);
            const int64_t threads = l.ntasks * 32;
            k_assemble<<<(int)((threads + 255) / 256), 256, 0, s>>>(jobs + l.job_begin, l.job_count, TMAP(l), l.ntasks, pv);
            ++timing.launches;
        }
        for (size_t st = 0; st < lp.panel.size(); ++st) {
            const Launch& pl = lp.panel[st];
            // a super-panel's first diagonal block has a launch of its own, the others
            // come with the step before
            if (st % kSteps == 0) {
                mark(3);
                launch_diag(pl, s, pv);
            }
            const bool chain = (st + 1) % kSteps != 0;
            // the look-ahead update of two steps before wrote the columns that
            // this step is about to update (and the event's slot is free again)
            join_ahead(st);
            if (pl.ntasks > 0) {
                mark(chain ? 3 : 4);
                if (chain) {
                    launch_chain(pl, s, pv);
                } else {
                    k_trsm<<<(int)pl.ntasks, 128, kTrsmSmem, s>>>(jobs + pl.job_begin, pl.job_count, TMAP(pl), pv);
                    ++timing.launches;
                }
            }
            const bool has_far = !lp.far[st].empty() || !lp.far_tc[st].empty();
            const bool far_tc = mixed_ == 1 && lp.far_flops[st] >= tc_min_flops_;
            const bool trail_i8 = use_i8_ && lp.trail_i8[st].gemm.ntasks > 0 && lp.trail_i8[st].flops >= i8_min_flops_;
            if (has_far && u != s && !trail_i8) {
                // the super-panel is final: fork the far columns of its trailing update
                cudaEvent_t e = D.evpool[evi++];
                cudaEventRecord(e, s);
                cudaStreamWaitEvent(u, e, 0);
            }
            if (early && st < lp.wb_sp.size() && lp.wb_sp[st].ntasks > 0) {
                // super-panels that end here are final: write them to LNZ beside
                // the rest of the level, for the caller to copy early
                const Launch& w = lp.wb_sp[st];
                cudaEvent_t e = D.evpool[evi++];
                cudaEventRecord(e, s);
                cudaStreamWaitEvent(D.wbs, e, 0);
                k_writeback<<<(int)((w.ntasks * 32 + 255) / 256), 256, 0, D.wbs>>>(jobs + w.job_begin, w.job_count,
                                                                                 TMAP(w), w.ntasks, pv);
                ++timing.launches;
                hooks_->columns_written(L, st, D.wbs);
                wrote_early = true;
            }
            mark(5);
            // a trailing update's next-super-panel columns were also updated by
            // the previous super-panel's far launch: wait for it first
            if (!chain) join_far();
            cudaEvent_t fork_ahead = nullptr;
            if (!lp.ahead[st].empty() && la != s) {
                fork_ahead = D.evpool[evi++];
                cudaEventRecord(fork_ahead, s);
            }
            // the K = kSuperPanel update of the next super-panel's columns is on
            // the critical path; in mixed mode it takes the tensor cores when large
            // enough (the next panel's K = 64 updates stay FP64 in every mode)
            if (trail_i8) {
                // one split serves both column ranges; the slabs are free again
                // because the previous far update was joined above
                launch_i8_split(lp.trail_i8[st], s, pv, gev);
                timing.tc_flops += lp.trail_i8[st].flops;
                if (has_far && u != s) {
                    cudaEvent_t e = D.evpool[evi++];
                    cudaEventRecord(e, s);
                    cudaStreamWaitEvent(u, e, 0);
                }
                launch_i8_gemm(lp.trail_i8[st].gemm, s, pv, gev, false);
                for (const Launch& ul : lp.trail_i8[st].rest) launch_gemm(ul, s, pv, gev);
            } else if (mixed_ == 1 && !lp.next_tc[st].empty() && lp.next_flops[st] >= tc_min_flops_) {
                for (const TcLaunch& t : lp.next_tc[st]) launch_tc(t, s, pv, gev);
                timing.tc_flops += lp.next_flops[st];
            } else {
                for (const Launch& ul : lp.update[st]) launch_gemm(ul, s, pv, gev);
            }
            if (!lp.ahead[st].empty()) {
                if (fork_ahead) cudaStreamWaitEvent(la, fork_ahead, 0);
                for (const Launch& al : lp.ahead[st]) launch_gemm(al, la, pv, gev);
                if (la != s) {
                    ahead_done[st & 1] = D.evpool[evi++];
                    cudaEventRecord(ahead_done[st & 1], la);
                }
            }
            if (has_far) {
                if (trail_i8) {
                    launch_i8_gemm(lp.trail_i8[st].far, u, pv, gev, true);
                    for (const Launch& fl : lp.trail_i8[st].far_rest) launch_gemm(fl, u, pv, gev);
                } else if (far_tc) {
                    for (const TcLaunch& t : lp.far_tc[st]) launch_tc(t, u, pv, gev, true);
                    timing.tc_flops += lp.far_flops[st];
                }
                else {
                    for (const Launch& fl : lp.far[st]) launch_gemm(fl, u, pv, gev);
                }
                if (u != s) {
                    far_done = D.evpool[evi++];
                    cudaEventRecord(far_done, u);
                }
            }
        }
        join_ahead(0);
        join_ahead(1);
        join_far();
        auto writeback = [&](cudaStream_t ws) {
            mark(7);
            const Launch& l = lp.writeback;
            const int64_t threads = l.ntasks * 32;
            k_writeback<<<(int)((threads + 255) / 256), 256, 0, ws>>>(jobs + l.job_begin, l.job_count, TMAP(l), l.ntasks, pv);
            ++timing.launches;
        };
        if (beside) {
            fork_to(D.wbs);
            writeback(D.wbs);
            wb_done[L & 1] = D.evpool[evi++];
            cudaEventRecord(wb_done[L & 1], D.wbs);
        }
        mark(6);
        if (mixed_ == 1 && lp.outer_flops >= tc_min_flops_) {
            for (const TcLaunch& t : lp.outer_tc) launch_tc(t, s, pv, gev);
            timing.tc_flops += lp.outer_flops;
        } else if (use_i8_ && !lp.outer_i8.empty() && lp.outer_i8[0].flops >= i8_min_flops_) {
            for (const I8Launch& t : lp.outer_i8) {
                if (t.gemm.ntasks > 0) {
                    launch_i8_split(t, s, pv, gev);
                    launch_i8_gemm(t.gemm, s, pv, gev, false);
                    timing.tc_flops += t.flops;
                }
                for (const Launch& ol : t.rest) launch_gemm(ol, s, pv, gev);
            }
        } else
            for (const Launch& ol : lp.outer) launch_gemm(ol, s, pv, gev);
        if (wrote_early) {
            // the level's own write-back rewrites the same values: after the early ones
            cudaEvent_t e = D.evpool[evi++];
            cudaEventRecord(e, D.wbs);
            cudaStreamWaitEvent(s, e, 0);
        }
        if (!beside) writeback(s);
        join_small(small, s, evi);
    }
    join_wb(0);
    join_wb(1);
    mark(8);
    k_reduce<true><<<1, 1024, 0, s>>>(pv.dvec, P_.neq, &D.st->mindpos);
    ++timing.launches;
}

int Engine::factor(double* d_sm, double tol1, FactorResult& res, const Singular* fc3) {
    NvtxRange range("spr_b200 factor");
    Dev& D = *d_;
    cudaStream_t s = stream_;
    // without room for the slabs the updates stay on the FP64 kernel
    use_i8_ = mixed_ == 0 && any_i8_ && ensure_i8() == 0;
    PV pv = make_view(D, P_, d_sm, tol1);
    if (fc3) {
        if (!fc3->d_dcor) return -2;
        pv.fc3 = chol_ ? 2 : 1;               // SPRF47 (SPRFC4) or SPRF37 (SPRFC3)
        pv.tol4 = fc3->tol4;
        pv.dcor = fc3->d_dcor;
    }
    pv.wait_ns = wait_ns_;
    pv.tc_drop = tc_drop_ ? 1 : 0;
    pv.adiag_in = streamed_diag_;
    linv_valid_ = false;
    last_near_ = 0;
    last_refactor_ = false;
    if (mixed_ == 1) {
        const int rc = ensure_slabs();
        if (rc != 0) return rc;
    }
    // inertia guard: keep the assembled SM, so that the factorisation can be
    // redone in FP64 when a pivot's sign may depend on the TF32 rounding
    const bool guard = mixed_ != 0 && guard_tol_ > 0.0;
    const int64_t nsm = P_.neq + P_.nzerol;
    if (guard) {
        if (guard_cap_ < nsm) {
            if (guard_copy_) cudaFree(guard_copy_);
            guard_copy_ = nullptr;
            guard_cap_ = 0;
            CK(alloc((void**)&guard_copy_, nsm * sizeof(double)));
            guard_cap_ = nsm;
        }
        CK(cudaMemcpyAsync(guard_copy_, d_sm, nsm * sizeof(double), cudaMemcpyDeviceToDevice, s));
        pv.near_tol = guard_tol_;
    }
    Stats init{};
    init.first_zero = 0x7fffffff;
    CK(cudaMemcpyAsync(D.st, &init, sizeof(Stats), cudaMemcpyHostToDevice, s));
    CK(cudaMemsetAsync(D.sn_neg, 0, P_.nsuper * sizeof(int32_t), s));
    CK(cudaMemsetAsync(D.sn_fail, 0xff, P_.nsuper * sizeof(int32_t), s));
    CK(cudaMemsetAsync(D.sn_bad, 0, P_.nsuper * sizeof(int32_t), s));
    timing.gemm_ms = 0.f;
    timing.gemm_launches = 0;
    tc_pairs_.clear();
    CK(cudaEventRecord(D.ev0, s));
    std::vector<cudaEvent_t> gev;
    // the legacy default stream cannot be captured: graphs need a stream of our own;
    // the watchdog test launches kernel by kernel (its settings are not in the key)
    // a streamed factorisation enqueues its copies' waits between the levels;
    // a split run its exchanges
    ExchangeHooks xh;
    const LevelHooks* saved_hooks = hooks_;
    if (split_ && !hooks_) {
        xh.P = &P_;
        xh.out = &fout_;
        xh.in = &fin_;
        xh.copy = [this](int32_t js, double* b, bool o, cudaStream_t st) { block_copy(js, b, o, st); };
        hooks_ = &xh;
    }
    struct RestoreHooks {
        const LevelHooks** h;
        const LevelHooks* v;
        ~RestoreHooks() { *h = v; }
    } restore{&hooks_, saved_hooks};
    const bool graph = use_graphs_ && !profile_ && s != nullptr && !tc_drop_ && wait_ns_ == 2000000000ull && !hooks_;
    if (graph) {
        const GraphKey key{(const void*)d_sm, nullptr, tol1, far_cap_q_,
                           mixed_ | (chol_ ? 16 : 0) | (small_tile_ == kTileTiny ? 32 : 0) | (use_i8_ ? 64 : 0),
                           (int64_t)std::min(use_i8_ ? i8_min_flops_ : tc_min_flops_, 9.0e18), (const void*)pv.dcor, pv.tol4,
                           pv.near_tol};
        cudaGraphExec_t exec = find_graph(key);
        if (!exec) {
            CK(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
            enqueue_factor(pv, s, gev);
            cudaGraph_t g = nullptr;
            CK(cudaStreamEndCapture(s, &g));
            CK(cudaGraphInstantiate(&exec, g, 0));
            cudaGraphDestroy(g);
            store_graph(key, exec, timing.launches);
        } else {
            timing.launches = graph_launches(key);
        }
        CK(cudaGraphLaunch(exec, s));
    } else {
        enqueue_factor(pv, s, gev);
    }
    trace_point(graph ? "factor graph launched" : "factor launches enqueued");
    CK(cudaEventRecord(D.ev1, s));
    CK(cudaGetLastError());
    Stats hs;
    static_assert(sizeof(Stats) % 8 == 0 && sizeof(Stats) / 8 <= 32, "Stats fits the mailbox");
    k_mailbox<<<1, 32, 0, s>>>(reinterpret_cast<const unsigned long long*>(D.st), (int)(sizeof(Stats) / 8),
                               D.mbox_dev);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(s));
    std::memcpy(&hs, D.mbox, sizeof(Stats));
    trace_point("factor stream synchronised");
    CK(cudaEventElapsedTime(&timing.factor_ms, D.ev0, D.ev1));
    timing.tc_ms = 0.f;
    size_t tp = 0;
    for (size_t k = 0; k + 1 < gev.size(); k += 2) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, gev[k], gev[k + 1]);
        timing.gemm_ms += ms;
        if (tp < tc_pairs_.size() && tc_pairs_[tp] == k) {
            timing.tc_ms += ms;
            ++tp;
        }
    }
    tc_pairs_.clear();
    for (cudaEvent_t e : gev) cudaEventDestroy(e);
    for (int k = 0; k < 9; ++k) timing.phase_ms[k] = 0.f;
    for (size_t k = 0; k < marks_.size(); ++k) {
        float ms = 0.f;
        cudaEventElapsedTime(&ms, marks_[k].second, k + 1 < marks_.size() ? marks_[k + 1].second : D.ev1);
        timing.phase_ms[marks_[k].first] += ms;
        cudaEventDestroy(marks_[k].second);
    }
    marks_.clear();
    res = FactorResult();
    last_trace_ = hs.trace;
    if (hs.tc_timeout) {
        fprintf(stderr, "spr_b200: a tensor-core update gave up waiting for its operands\n");
        return -4;
    }
    if (guard && (hs.near_piv > 0 || (hs.pivot_fail && hs.zero_count == 0))) {
        // a pivot within guard_tol_ |a_jj| of zero, or a failed pivot test,
        // after TF32 updates: decide inertia and the pivot test in FP64
        const float first_ms = timing.factor_ms;
        const int64_t near = (int64_t)hs.near_piv;
        CK(cudaMemcpyAsync(d_sm, guard_copy_, nsm * sizeof(double), cudaMemcpyDeviceToDevice, s));
        const int mode = mixed_;
        mixed_ = 0;
        const int rc = factor(d_sm, tol1, res, fc3);
        mixed_ = mode;
        timing.factor_ms += first_ms;
        last_near_ = near;
        last_refactor_ = true;
        return rc;
    }
    last_near_ = (int64_t)hs.near_piv;
    if (hs.zero_count > 0) {                       // sprfc1.f:474-488
        // the reference's pre-pass has already replaced D by the original diagonal
        CK(cudaMemcpy(pv.dvec, D.adiag, P_.neq * sizeof(double), cudaMemcpyDeviceToDevice));
        res.lierr = -35;
        res.numneg = hs.zero_count;
        res.supeqt = (int64_t)hs.first_zero + 1;
        res.tol2 = 0.0;
        res.tol3 = hs.trace;
        return 0;
    }
    if (hs.pivot_fail) {                           // sprfc1.f:610-616
        std::vector<int32_t> fail(P_.nsuper), neg(P_.nsuper);
        CK(cudaMemcpy(fail.data(), D.sn_fail, P_.nsuper * sizeof(int32_t), cudaMemcpyDeviceToHost));
        CK(cudaMemcpy(neg.data(), D.sn_neg, P_.nsuper * sizeof(int32_t), cudaMemcpyDeviceToHost));
        int64_t jf = -1;
        for (int64_t js = 0; js < P_.nsuper; ++js)
            if (fail[js] >= 0) {
                jf = js;
                break;
            }
        int64_t nn = 0;
        for (int64_t js = 0; js <= jf; ++js) nn += neg[js];
        double fd = 0.0, fa = 0.0;
        CK(cudaMemcpy(&fd, D.sn_faild + jf, sizeof(double), cudaMemcpyDeviceToHost));
        CK(cudaMemcpy(&fa, D.sn_faila + jf, sizeof(double), cudaMemcpyDeviceToHost));
        res.lierr = -30;
        res.numneg = nn;
        res.supeqt = (int64_t)P_.fst[jf] + fail[jf] + 1;
        res.tol2 = fd;
        res.tol3 = fa;
        return 0;
    }
    linv_valid_ = true;
    if (fc3 && hs.nsing > 0) {                     // sprfc3.f:796-799, sprfc4.f:719-722
        res.lierr = chol_ ? -33 : -31;
        res.supeqt = (int64_t)hs.nsing;
    }
    res.numneg = hs.numneg;
    res.tol2 = (hs.tol2 != 0.0) ? 1.0 / hs.tol2 : 0.0;          // sprfc1.f:699-703
    res.tol3 = (hs.mindpos != 0.0) ? hs.trace / hs.mindpos : 0.0;  // sprfc1.f:704-708
    if (chol_) {                                                   // sprfc2.f:699-716
        const double m = std::sqrt(hs.mindpos);
        res.tol3 = (m != 0.0) ? hs.trace / (m * m) : 0.0;
    }
    return 0;
}

int Engine::hash(const double* d_a, int64_t n, uint64_t& h) {
    Dev& D = *d_;
    unsigned long long hv = 0ull;
    CK(cudaMemsetAsync(D.hbuf, 0, sizeof(unsigned long long), stream_));
    if (n > 0) {
        const int grid = (int)std::min<int64_t>((n + 255) / 256, 8 * (int64_t)std::max(sm_count_, 1));
        k_sm_hash<<<grid, 256, 0, stream_>>>(d_a, n, D.hbuf);
        CK(cudaGetLastError());
    }
    k_mailbox<<<1, 32, 0, stream_>>>(D.hbuf, 1, D.mbox_dev);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(stream_));
    hv = D.mbox[0];
    h = (uint64_t)hv;
    return 0;
}

// dst[0 .. n) = src[0 .. n) on the device (the early fronts' backup).
__global__ void k_copy_d(const double* __restrict__ src, double* __restrict__ dst, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = src[i];
}

namespace {
// Host-side pacing of the streamed copies.  Hundreds of queued copy
// operations make the next kernel launch wait until they drain, and copies
// in one direction share the copy engine whatever their stream, so neither
// all uploads nor all downloads are queued at once: one thread queues a
// group's uploads once the group two below it is up, another queues a
// group's downloads once its last level has finished on the device.  The
// enqueueing thread waits, before a level's first launch, until that level's
// upload event has been recorded, and marks each group's end event as
// recorded after its last level.
struct CopyScheduler {
    // a download: once ev has completed, copy these LNZ ranges to the host
    struct Item {
        cudaEvent_t ev;
        const std::vector<std::pair<int64_t, int64_t>>* ranges;
        bool last;
    };
    std::mutex mu;
    std::condition_variable cv;
    std::vector<char> up_recorded;
    std::deque<Item> downloads;                 // in the order the enqueueing thread recorded them
    bool abort = false;
    int status = 0;
    void push(const Item& it) {
        {
            std::lock_guard<std::mutex> lk(mu);
            downloads.push_back(it);
        }
        cv.notify_all();
    }
    bool pop(Item& it) {
        std::unique_lock<std::mutex> lk(mu);
        cv.wait(lk, [&] { return !downloads.empty() || abort; });
        if (downloads.empty()) return false;
        it = downloads.front();
        downloads.pop_front();
        return true;
    }
    void mark(std::vector<char>& v, size_t g) {
        {
            std::lock_guard<std::mutex> lk(mu);
            v[g] = 1;
        }
        cv.notify_all();
    }
    bool wait(std::vector<char>& v, size_t g) {
        std::unique_lock<std::mutex> lk(mu);
        cv.wait(lk, [&] { return v[g] != 0 || abort; });
        return v[g] != 0;
    }
    void stop() {
        {
            std::lock_guard<std::mutex> lk(mu);
            abort = true;
        }
        cv.notify_all();
    }
};

struct StreamHooks : LevelHooks {
    const Engine::Transfer* t = nullptr;
    CopyScheduler* cs_sched = nullptr;
    double* d_lnz = nullptr;
    int sm_count = 148;
    size_t nlev = 0;
    void before(size_t L, cudaStream_t s) const override {
        const int g = t->group((int32_t)L);
        if (L == 0 || (g > 0)) {
            if (!cs_sched->wait(cs_sched->up_recorded, (size_t)g)) return;
            cudaStreamWaitEvent(s, t->up[g], 0);
        }
        if ((int32_t)L == t->early_level) {
            // the early fronts' uploaded LNZ, kept in case a pivot of theirs fails
            int64_t b = 0;
            for (const auto& r : t->early_ranges) {
                k_copy_d<<<2 * sm_count, 256, 0, s>>>(d_lnz + r.first, t->d_backup + b, r.second);
                b += r.second;
            }
        }
    }
    void after(size_t L, cudaStream_t s) const override {
        const int g = t->group((int32_t)L);
        const bool last_of_group = (L + 1 == nlev) || t->group((int32_t)(L + 1)) != g;
        if (!last_of_group) return;
        cudaEventRecord(t->done[g], s);
        cs_sched->push({t->done[g], &t->dranges[g], (size_t)g + 1 == t->dranges.size()});
    }
    bool early_columns(size_t L) const override { return (int32_t)L == t->early_level; }
    void columns_written(size_t L, size_t st, cudaStream_t ws) const override {
        cudaEventRecord(t->spev[st], ws);
        cs_sched->push({t->spev[st], &t->spranges[st], false});
    }
};
}  // namespace

int Engine::factor_streamed(double* h_sm, double* d_sm, double tol1, FactorResult& res, cudaStream_t cs) {
    NvtxRange range("spr_b200 factor (streamed copies)");
    const int64_t neq = P_.neq;
    if (!xfer_) {
        std::unique_ptr<Transfer> t(new Transfer());
        const int32_t nlev = (int32_t)P_.levels.size();
        std::vector<int64_t> at_level(nlev + 1, 0);
        for (int64_t js = 0; js < P_.nsuper; ++js) ++at_level[P_.level[js]];
        int64_t above = 0;
        t->L1 = nlev;
        for (int32_t L = nlev - 1; L >= 1; --L) {
            above += at_level[L];
            if (above > Transfer::kMaxTopNodes) break;
            t->L1 = L;
        }
        const int ng = 1 + (nlev - t->L1);
        // the last level's eliminated large fronts: their columns come back
        // super-panel by super-panel, not with the level's group
        std::vector<char> early(P_.nsuper, 0);
        if (nlev > 0) {
            const LevelPlan& lp = P_.levels[nlev - 1];
            t->spranges.assign(lp.wb_sp.size(), {});
            for (size_t st = 0; st < lp.wb_sp.size(); ++st) {
                const Launch& w = lp.wb_sp[st];
                for (int64_t j = 0; j < w.job_count; ++j) {
                    const Job& jb = P_.jobs[w.job_begin + j];
                    const int64_t f = P_.F[jb.node];
                    const int64_t a = P_.lnz_off[jb.node] + lnz_col(jb.c0, f);
                    t->spranges[st].emplace_back(a, lnz_col(jb.c_end, f) - lnz_col(jb.c0, f));
                    early[jb.node] = 1;
                    t->early_level = nlev - 1;
                }
            }
            t->spev.resize(lp.wb_sp.size());
            for (cudaEvent_t& e : t->spev) CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        }
        t->ranges.assign(ng, {});
        t->dranges.assign(ng, {});
        auto append = [](std::vector<std::pair<int64_t, int64_t>>& rg, int64_t off, int64_t len) {
            if (!rg.empty() && rg.back().first + rg.back().second == off)
                rg.back().second += len;
            else
                rg.emplace_back(off, len);
        };
        int64_t nbackup = 0;
        for (int64_t js = 0; js < P_.nsuper; ++js) {
            const int64_t f = P_.F[js], sw = P_.S[js];
            const int64_t off = P_.lnz_off[js], len = f * sw - sw * (sw - 1) / 2;
            const int g = t->group(P_.level[js]);
            append(t->ranges[g], off, len);
            if (early[js]) {
                t->early_nodes.push_back((int32_t)js);
                t->early_ranges.emplace_back(off, len);
                nbackup += len;
            } else {
                append(t->dranges[g], off, len);
            }
        }
        if (nbackup > 0) CK(alloc((void**)&t->d_backup, nbackup * sizeof(double)));
        t->up.resize(ng);
        t->done.resize(ng);
        for (int g = 0; g < ng; ++g) {
            CK(cudaEventCreateWithFlags(&t->up[g], cudaEventDisableTiming));
            CK(cudaEventCreateWithFlags(&t->done[g], cudaEventDisableTiming));
        }
        CK(cudaStreamCreateWithFlags(&t->ups, cudaStreamNonBlocking));
        CK(cudaEventCreateWithFlags(&t->start, cudaEventDisableTiming));
        CK(cudaEventCreateWithFlags(&t->fin, cudaEventDisableTiming));
        CK(cudaEventCreate(&t->ts));
        CK(cudaEventCreate(&t->tu));
        CK(cudaEventCreate(&t->te));
        CK(cudaEventCreate(&t->tf));
        CK(cudaEventCreate(&t->tf0));
        t->diag_pos.resize(neq);
        for (int64_t js = 0; js < P_.nsuper; ++js)
            for (int64_t j = 0; j < P_.S[js]; ++j) t->diag_pos[P_.fst[js] + j] = P_.lnz_off[js] + lnz_col(j, P_.F[js]);
        CK(cudaMallocHost((void**)&t->h_diag, std::max<int64_t>(neq, 1) * sizeof(double)));
        CK(alloc((void**)&t->d_diag, std::max<int64_t>(neq, 1) * sizeof(double)));
        xfer_ = std::move(t);
    }
    Transfer& t = *xfer_;
    const size_t ng = t.ranges.size();
    cudaStream_t s = stream_;
    double* h_lnz = h_sm + neq;
    double* d_lnz = d_sm + neq;
    // the pre-pass needs every original diagonal before anything is factored
    // (the zero test of sprfc1.f:465-488): gathered first, so that D and the
    // diagonals are the first uploads in the copy engine's queue
    {
        const int nt = (int)std::min<int64_t>(8, std::max<int64_t>(1, neq / 65536));
        std::vector<std::thread> pool;
        for (int k = 0; k < nt; ++k)
            pool.emplace_back([&, k]() {
                for (int64_t j = neq * k / nt; j < neq * (k + 1) / nt; ++j) t.h_diag[j] = h_lnz[t.diag_pos[j]];
            });
        for (auto& th : pool) th.join();
    }
    CK(cudaEventRecord(t.ts, s));
    // D on the compute stream (the pre-pass writes D of retained supernodes)
    CK(cudaMemcpyAsync(d_sm, h_sm, neq * sizeof(double), cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(t.d_diag, t.h_diag, neq * sizeof(double), cudaMemcpyHostToDevice, s));
    // the copy streams start after the compute stream's earlier work
    CK(cudaEventRecord(t.start, s));
    CK(cudaStreamWaitEvent(cs, t.start, 0));
    CK(cudaStreamWaitEvent(t.ups, t.start, 0));
    CopyScheduler sched;
    sched.up_recorded.assign(ng, 0);
    std::thread uploader([&]() {
        for (size_t g = 0; g < ng; ++g) {
            if (g >= 2 && cudaEventSynchronize(t.up[g - 2]) != cudaSuccess) sched.status = -4;
            for (const auto& r : t.ranges[g])
                if (cudaMemcpyAsync(d_lnz + r.first, h_lnz + r.first, r.second * sizeof(double),
                                    cudaMemcpyHostToDevice, t.ups) != cudaSuccess)
                    sched.status = -4;
            if (cudaEventRecord(t.up[g], t.ups) != cudaSuccess) sched.status = -4;
            if (g == 0) cudaEventRecord(t.tu, t.ups);
            sched.mark(sched.up_recorded, g);
        }
    });
    std::thread downloader([&]() {
        CopyScheduler::Item it;
        while (sched.pop(it)) {
            if (cudaEventSynchronize(it.ev) != cudaSuccess) sched.status = -4;
            for (const auto& r : *it.ranges)
                if (cudaMemcpyAsync(h_lnz + r.first, d_lnz + r.first, r.second * sizeof(double),
                                    cudaMemcpyDeviceToHost, cs) != cudaSuccess)
                    sched.status = -4;
            if (it.last) return;
        }
    });
    if (trace_on()) {
        size_t nu = 0;
        for (const auto& u : t.ranges) nu += u.size();
        char b[96];
        snprintf(b, sizeof b, "diagonal gathered, copy threads started (%zu ranges each way)", nu);
        trace_point(b);
    }
    StreamHooks hk;
    hk.t = &t;
    hk.cs_sched = &sched;
    hk.d_lnz = d_lnz;
    hk.sm_count = std::max(sm_count_, 1);
    hk.nlev = P_.levels.size();
    hooks_ = &hk;
    streamed_diag_ = t.d_diag;
    cudaEventRecord(t.tf0, s);
    const int rc = factor(d_sm, tol1, res, nullptr);
    hooks_ = nullptr;
    streamed_diag_ = nullptr;
    if (rc != 0) sched.stop();                  // a level that was never enqueued records no end event
    uploader.join();
    downloader.join();
    trace_point("copy threads joined");
    if (rc != 0 || sched.status != 0) {
        cudaStreamSynchronize(t.ups);
        cudaStreamSynchronize(cs);
        return rc != 0 ? rc : -4;
    }
    if (res.lierr != 0 && !t.early_nodes.empty()) {
        // an early front that failed keeps its uploaded columns, on the device
        // and on the host (its early super-panels are undone)
        std::vector<int32_t> bad(t.early_nodes.size(), 0);
        for (size_t i = 0; i < t.early_nodes.size(); ++i)
            CK(cudaMemcpy(&bad[i], d_->sn_bad + t.early_nodes[i], sizeof(int32_t), cudaMemcpyDeviceToHost));
        int64_t b = 0;
        for (size_t i = 0; i < t.early_nodes.size(); ++i) {
            const auto& r = t.early_ranges[i];
            if (bad[i]) k_copy_d<<<2 * std::max(sm_count_, 1), 256, 0, s>>>(t.d_backup + b, d_lnz + r.first, r.second);
            b += r.second;
        }
        CK(cudaGetLastError());
        CK(cudaEventRecord(t.fin, s));
        CK(cudaStreamWaitEvent(cs, t.fin, 0));
        for (size_t i = 0; i < t.early_nodes.size(); ++i)
            if (bad[i]) {
                const auto& r = t.early_ranges[i];
                CK(cudaMemcpyAsync(h_lnz + r.first, d_lnz + r.first, r.second * sizeof(double),
                                   cudaMemcpyDeviceToHost, cs));
            }
    }
    // D is final only now (and on a zero diagonal it holds the original diagonal)
    CK(cudaEventRecord(t.fin, s));
    CK(cudaEventRecord(t.tf, s));
    CK(cudaStreamWaitEvent(cs, t.fin, 0));
    CK(cudaMemcpyAsync(h_sm, d_sm, neq * sizeof(double), cudaMemcpyDeviceToHost, cs));
    CK(cudaEventRecord(t.te, cs));
    return 0;
}

int Engine::streamed_times(double* out) {
    out[0] = out[1] = out[2] = 0.0;
    if (!xfer_) return 0;
    float a = 0.f, c = 0.f;
    // from the call's first copy to the factorisation's first launch, and from
    // its end to the end of the last download
    if (cudaEventElapsedTime(&a, xfer_->ts, xfer_->tf0) != cudaSuccess ||
        cudaEventElapsedTime(&c, xfer_->tf, xfer_->te) != cudaSuccess)
        return -4;
    out[0] = a;
    out[1] = timing.factor_ms;
    out[2] = c;
    return 0;
}

int Engine::factor_chol(double* d_sm, double tol1, FactorResult& res, const Singular* fc4) {
    chol_ = true;
    const int rc = factor(d_sm, tol1, res, fc4);
    chol_ = false;
    return rc;
}

int Engine::chol_convert(double* d_sm, bool to_chol) {
    Dev& D = *d_;
    PV pv = make_view(D, P_, d_sm, 0.0);
    const int grid = (int)std::min<int64_t>(P_.nsuper, 8 * (int64_t)std::max(sm_count_, 1));
    if (to_chol)
        k_chol_convert<true><<<grid, 256, 0, stream_>>>(pv, P_.nsuper);
    else
        k_chol_convert<false><<<grid, 256, 0, stream_>>>(pv, P_.nsuper);
    CK(cudaGetLastError());
    linv_valid_ = false;
    return 0;
}

int Engine::scale_sqrt_d(const double* d_sm, double* d_b, int64_t ldb, int64_t nrhs, bool divide) {
    const int64_t n = P_.neq * nrhs;
    if (n <= 0) return 0;
    const int grid = (int)std::min<int64_t>((n + 255) / 256, 8 * (int64_t)std::max(sm_count_, 1));
    k_scale_sqrt_d<<<grid, 256, 0, stream_>>>(d_sm, d_b, ldb, P_.neq, nrhs, divide ? 1 : 0);
    CK(cudaGetLastError());
    return 0;
}

int Engine::sn_stats(int32_t* neg, int32_t* fail) {
    Dev& D = *d_;
    CK(cudaMemcpy(neg, D.sn_neg, P_.nsuper * sizeof(int32_t), cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(fail, D.sn_fail, P_.nsuper * sizeof(int32_t), cudaMemcpyDeviceToHost));
    return 0;
}

// Buffers for up to nrhs right-hand sides in a pass; returns how many a pass
// may take (0: not even kMaxRHS fit).  Graphs captured on the old buffers go
// with them: the three move independently, and a new one may lie where another was.
int64_t Engine::ensure_vectors(int64_t nrhs) {
    Dev& D = *d_;
    if (nrhs <= 0) return D.vbuf ? 1 : 0;                // nothing to solve
    for (;;) {
        const int64_t want = std::min(nrhs, D.pass_rhs);
        if (D.vbuf && D.vbuf_rhs >= want) return want;
        drop_solve_graphs();
        for (double** p : {&D.vbuf, &D.ybuf, &D.pbuf}) {
            if (*p) cudaFree(*p);
            *p = nullptr;
        }
        D.vbuf_rhs = 0;
        const int64_t nrp = (want + 3) / 4 * 4;
        const size_t d = sizeof(double);
        // (a narrower pass comes before the integer updates' slabs are given up)
        auto get = [&](double** p, int64_t n) {
            return (want > kMaxRHS ? cudaMalloc((void**)p, n * d) : alloc((void**)p, n * d)) == cudaSuccess;
        };
        if (get(&D.vbuf, std::max<int64_t>(P_.rbase.back(), 1) * want) && get(&D.ybuf, P_.neq * nrp) &&
            get(&D.pbuf, std::max<int64_t>(std::max(P_.rect_entries, P_.fwd_entries), 1) * nrp)) {
            D.vbuf_rhs = want;
            return want;
        }
        cudaGetLastError();
        if (want <= kMaxRHS) return 0;
        D.pass_rhs = kMaxRHS;
    }
}

void Engine::enqueue_solve(const PV& pv, cudaStream_t s, double* d_b, int64_t ldb, int64_t nrhs, int64_t chunk,
                           int which, int64_t& nl) {
    Dev& D = *d_;
    auto mark = [&](int phase) {
        if (profile_) marks_.emplace_back(9 + phase, record_event(s));
    };
    const Job* jobs = D.jobs;
    const int64_t neq = P_.neq;
    auto blocks = [](int64_t threads) { return (int)((threads + 255) / 256); };
    const size_t ctr_bytes = sizeof(int32_t) * 2 * P_.levels.size();
    for (int64_t r0 = 0; r0 < nrhs; r0 += chunk) {
        const int nr = (int)std::min<int64_t>(chunk, nrhs - r0);
        // ng groups of gw right-hand sides; y and the partials are padded to whole groups
        const int gw = nr == 1 ? 1 : nr == 2 ? 2 : 4, ng = (nr + gw - 1) / gw, nrp = gw * ng;
        const int sg = (nr + kMaxRHS - 1) / kMaxRHS, sr = std::min(nr, kMaxRHS);
        double* b = d_b + r0 * ldb;
        if (which & 1) {
            cudaMemsetAsync(D.tri_sync, 0, ctr_bytes, s);
            if (P_.any_large) cudaMemsetAsync(D.ybuf, 0xff, neq * nrp * sizeof(double), s);
            // split run: the other ranks' subtree roots' update vectors come in
            // before their parent's level, this rank's go out after their level
            ExchangeHooks vx;
            vx.P = &P_;
            vx.out = &vout_;
            vx.in = &vin_;
            vx.copy = [this, nr](int32_t js, double* buf, bool o, cudaStream_t st) { vec_copy(js, buf, o, nr, st); };
            const bool vexch = !vout_.empty() || !vin_.empty();
            size_t evi = 0;
            for (size_t L = 0; L < P_.levels.size(); ++L) {
                const LevelPlan& lp = P_.levels[L];
                if (vexch) vx.before(L, s);
                struct AfterLevel {
                    const ExchangeHooks* h;
                    size_t L;
                    cudaStream_t s;
                    ~AfterLevel() {
                        if (h) h->after(L, s);
                    }
                } after_level{vexch ? &vx : nullptr, L, s};
                // the small fronts beside the large ones, as in the factorisation:
                // 12^3, 3 right-hand sides 0.91 -> 0.72 ms, 24^3, 40 of them 3.6 -> 3.2 ms
                SmallStreams small{s, s};
                struct JoinSmall {                       // at every exit of this iteration, before after_level
                    Engine* e;
                    const SmallStreams& r;
                    cudaStream_t s;
                    size_t& evi;
                    ~JoinSmall() { e->join_small(r, s, evi); }
                } join{this, small, s, evi};
                if (!lp.small_nodes.empty()) {
                    mark(0);
                    if (!profile_) small = small_streams(lp, s, evi);
                    for (const LevelPlan::SmallClass& c : lp.small_classes) {
                        const auto f = sr == 1 ? k_forward<1> : sr == 2 ? k_forward<2> : k_forward<4>;
                        f<<<dim3(c.count, sg), small_threads(c.maxF), small_solve_smem(c.maxF, c.maxL, sr), small.of(lp, c)>>>(
                            D.level_nodes + D.small_begin[L] + c.begin, pv, D.vbuf, b, ldb, nr);
                        ++nl;
                    }
                }
                if (lp.large_nodes.empty()) continue;
                if (lp.retained_large) {
                    mark(1);
                    const Launch& ga = lp.assemble;
                    k_fwd_retained<<<blocks(ga.ntasks), 256, 0, s>>>(jobs + ga.job_begin, ga.job_count, TMAP(ga),
                                                                     ga.ntasks, pv, D.vbuf, b, ldb, nr);
                    ++nl;
                }
                if (lp.tri_count > 0) {
                    mark(2);
                    const int nt = (int)lp.tri_count;
                    const int grid = (int)std::min<int64_t>((int64_t)nt * ng, 4 * (int64_t)std::max(sm_count_, 1));
                    const int32_t* tasks = D.tri_tasks + 2 * lp.tri_begin;
                    int32_t* ctr = D.tri_sync + 2 * L;
                    if (gw == 1)
                        k_fwd_tri<1><<<grid, 256, 0, s>>>(tasks, nt, ng, ctr, pv, D.vbuf, D.ybuf, b, ldb, nr, neq);
                    else if (gw == 2)
                        k_fwd_tri<2><<<grid, 256, 0, s>>>(tasks, nt, ng, ctr, pv, D.vbuf, D.ybuf, b, ldb, nr, neq);
                    else
                        k_fwd_tri<4><<<grid, 256, 0, s>>>(tasks, nt, ng, ctr, pv, D.vbuf, D.ybuf, b, ldb, nr, neq);
                    ++nl;
                }
                const Launch& rl = lp.rect;
                if (rl.ntasks > 0) {
                    mark(3);
                    const Job* j = jobs + rl.job_begin;
                    const unsigned nt = (unsigned)rl.ntasks;
                    // from two groups on a CTA takes two: L is read half as often from L2
                    if (gw == 1)
                        k_fwd_rect<1, 1><<<dim3(nt, ng), 256, 0, s>>>(j, rl.job_count, TMAP(rl), pv, D.ybuf, D.vbuf, D.pbuf,
                                                                      nr, nrp, neq);
                    else if (gw == 2)
                        k_fwd_rect<2, 1><<<dim3(nt, ng), 256, 0, s>>>(j, rl.job_count, TMAP(rl), pv, D.ybuf, D.vbuf, D.pbuf,
                                                                      nr, nrp, neq);
                    else if (ng == 1)
                        k_fwd_rect<4, 1><<<dim3(nt, ng), 256, 0, s>>>(j, rl.job_count, TMAP(rl), pv, D.ybuf, D.vbuf, D.pbuf,
                                                                      nr, nrp, neq);
                    else
                        k_fwd_rect<4, 2><<<dim3(nt, (ng + 1) / 2), 256, 0, s>>>(j, rl.job_count, TMAP(rl), pv, D.ybuf, D.vbuf,
                                                                                D.pbuf, nr, nrp, neq);
                    ++nl;
                    const Launch& rr = lp.rect_rows;
                    if (rr.ntasks > 0) {
                        k_fwd_rect_sum<<<blocks(rr.ntasks * nr), 256, 0, s>>>(jobs + rr.job_begin, rr.job_count, TMAP(rr),
                                                                              rr.ntasks, pv, D.vbuf, D.pbuf, b, ldb, nr,
                                                                              nrp);
                        ++nl;
                    }
                }
            }
        }
        if (which & 2) {
            cudaMemsetAsync(D.tri_sync, 0, ctr_bytes, s);
            if (P_.any_large) cudaMemsetAsync(D.ybuf, 0xff, neq * nrp * sizeof(double), s);
            size_t evi = 0;
            for (size_t L = P_.levels.size(); L-- > 0;) {
                const LevelPlan& lp = P_.levels[L];
                SmallStreams small{s, s};
                if (!lp.small_nodes.empty()) {
                    mark(5);
                    if (!profile_) small = small_streams(lp, s, evi);
                    for (const LevelPlan::SmallClass& c : lp.small_classes) {
                        const auto f = sr == 1 ? k_backward<1> : sr == 2 ? k_backward<2> : k_backward<4>;
                        f<<<dim3(c.count, sg), small_threads(c.maxF), small_solve_smem(c.maxF, c.maxL, sr), small.of(lp, c)>>>(
                            D.level_nodes + D.small_begin[L] + c.begin, pv, b, ldb, nr);
                        ++nl;
                    }
                }
                const Launch& rl = lp.rect_back;
                if (rl.ntasks > 0) {
                    mark(7);
                    const dim3 grid((unsigned)rl.ntasks, ng);
                    const Job* j = jobs + rl.job_begin;
                    if (gw == 1)
                        k_bwd_rect<1, true><<<grid, 256, 0, s>>>(j, rl.job_count, TMAP(rl), pv, D.pbuf, b, ldb, nr, nrp);
                    else if (gw == 2)
                        k_bwd_rect<2, true><<<grid, 256, 0, s>>>(j, rl.job_count, TMAP(rl), pv, D.pbuf, b, ldb, nr, nrp);
                    else if (ng == 1)
                        k_bwd_rect<4, true><<<grid, 256, 0, s>>>(j, rl.job_count, TMAP(rl), pv, D.pbuf, b, ldb, nr, nrp);
                    else
                        k_bwd_rect<4, false><<<grid, 256, 0, s>>>(j, rl.job_count, TMAP(rl), pv, D.pbuf, b, ldb, nr, nrp);
                    ++nl;
                }
                if (lp.tri_count > 0) {
                    mark(8);
                    const int nt = (int)lp.tri_count;
                    const int grid = (int)std::min<int64_t>((int64_t)nt * ng, 4 * (int64_t)std::max(sm_count_, 1));
                    const int32_t* tasks = D.tri_tasks + 2 * lp.tri_begin;
                    int32_t* ctr = D.tri_sync + 2 * L;
                    if (gw == 1)
                        k_bwd_tri<1><<<grid, 256, 0, s>>>(tasks, nt, ng, ctr, pv, D.pbuf, D.ybuf, b, ldb, nr, nrp, neq);
                    else if (gw == 2)
                        k_bwd_tri<2><<<grid, 256, 0, s>>>(tasks, nt, ng, ctr, pv, D.pbuf, D.ybuf, b, ldb, nr, nrp, neq);
                    else
                        k_bwd_tri<4><<<grid, 256, 0, s>>>(tasks, nt, ng, ctr, pv, D.pbuf, D.ybuf, b, ldb, nr, nrp, neq);
                    ++nl;
                }
                join_small(small, s, evi);
            }
        }
    }
}

int Engine::solve(const double* d_sm, double* d_b, int64_t ldb, int64_t nrhs, int which) {
    NvtxRange range("spr_b200 solve");
    Dev& D = *d_;
    cudaStream_t s = stream_;
    PV pv = make_view(D, P_, const_cast<double*>(d_sm), 0.0);
    pv.wait_ns = wait_ns_;
    pv.tc_drop = tc_drop_ ? 1 : 0;
    const int64_t chunk = ensure_vectors(nrhs);
    if (chunk <= 0) return -4;
    CK(cudaEventRecord(D.ev0, s));
    int64_t nl = 0;
    CK(cudaMemsetAsync(&D.st->solve_timeout, 0, sizeof(int), s));
    if (!linv_valid_) {
        for (const LevelPlan& lp : P_.levels)
            for (const Launch& pl : lp.panel)
                if (pl.job_count > 0) {
                    k_linv<<<(int)pl.job_count, 64, 0, s>>>(D.jobs + pl.job_begin, pv);
                    ++nl;
                }
        linv_valid_ = true;
    }
    if (use_graphs_ && !profile_ && s != nullptr && !tc_drop_ && wait_ns_ == 2000000000ull && !split_) {
        const GraphKey key{(const void*)d_sm, (const void*)d_b, (double)ldb, nrhs, which, chunk};
        cudaGraphExec_t exec = find_graph(key);
        if (!exec) {
            CK(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
            enqueue_solve(pv, s, d_b, ldb, nrhs, chunk, which, nl);
            cudaGraph_t g = nullptr;
            CK(cudaStreamEndCapture(s, &g));
            CK(cudaGraphInstantiate(&exec, g, 0));
            cudaGraphDestroy(g);
            store_graph(key, exec, nl);
        } else {
            nl += graph_launches(key);
        }
        CK(cudaGraphLaunch(exec, s));
    } else {
        enqueue_solve(pv, s, d_b, ldb, nrhs, chunk, which, nl);
    }
    CK(cudaEventRecord(D.ev1, s));
    CK(cudaGetLastError());
    k_mailbox<<<1, 32, 0, s>>>(reinterpret_cast<const unsigned long long*>(D.st), (int)(sizeof(Stats) / 8),
                               D.mbox_dev);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(s));
    Stats hs;
    std::memcpy(&hs, D.mbox, sizeof(Stats));
    const int tri_timeout = hs.solve_timeout;
    CK(cudaEventElapsedTime(&timing.solve_ms, D.ev0, D.ev1));
    timing.solve_launches = nl;
    if (tri_timeout) {
        fprintf(stderr, "spr_b200: a triangle task of the solve gave up waiting for a block\n");
        return -4;
    }
    if (profile_) {
        for (int k = 9; k < 20; ++k) timing.phase_ms[k] = 0.f;
        for (size_t k = 0; k < marks_.size(); ++k) {
            float ms = 0.f;
            cudaEventElapsedTime(&ms, marks_[k].second, k + 1 < marks_.size() ? marks_[k + 1].second : D.ev1);
            timing.phase_ms[marks_[k].first] += ms;
            cudaEventDestroy(marks_[k].second);
        }
        marks_.clear();
    }
    return 0;
}

// ---------------------------------------------------------------------------
// Blocked LDL' of one dense front with caller-provided scratch (no device
// allocation).  Same kernels and step order as the large-front path of
// Engine::factor for a front with S = F = n.
// ---------------------------------------------------------------------------
size_t dense_scratch_bytes(int64_t n) {
    const int64_t nblk = (n + kNB - 1) / kNB;
    const int64_t njobs = 3 * nblk;
    size_t b = 0;
    auto add = [&](size_t bytes) { b += (bytes + 255) / 256 * 256; };
    add(sizeof(Stats));
    add(sizeof(double) * n);                       // original diagonal
    add(sizeof(double) * nblk * kNB * kNB);        // inverses of the diagonal blocks
    add(sizeof(Job) * njobs);
    add(sizeof(int32_t) * 16);                     // node arrays (one node)
    add(sizeof(int64_t) * 8);
    add(sizeof(double) * 4);
    return b;
}

int dense_factor_setup() {
    // k_trsm and the small-tile update use more than the default 48 KB of
    // dynamic shared memory; the opt-in is per function and per device.
    CK(cudaFuncSetAttribute(k_diag<kPivotLDL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDiagSmem));
    CK(cudaFuncSetAttribute(k_trsm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrsmSmem));
    CK(cudaFuncSetAttribute(K_GEMM_SMALL, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GemmSmall::smem));
    return 0;
}

int dense_factor_with_scratch(double* a, int64_t n, int64_t lda, double tol1, double* d, void* scratch,
                              size_t scratch_bytes, cudaStream_t s, double* out) {
    if (n <= 0 || lda < n || (lda % 4) != 0 || ((uintptr_t)a % 32) != 0) return -2;
    if (dense_scratch_bytes(n) > scratch_bytes) return -3;
    const int64_t nblk = (n + kNB - 1) / kNB;
    char* p = static_cast<char*>(scratch);
    auto take = [&](size_t bytes) {
        char* q = p;
        p += (bytes + 255) / 256 * 256;
        return q;
    };
    Stats* st = reinterpret_cast<Stats*>(take(sizeof(Stats)));
    double* adiag = reinterpret_cast<double*>(take(sizeof(double) * n));
    double* linv = reinterpret_cast<double*>(take(sizeof(double) * nblk * kNB * kNB));
    Job* jobs = reinterpret_cast<Job*>(take(sizeof(Job) * 3 * nblk));
    int32_t* i32 = reinterpret_cast<int32_t*>(take(sizeof(int32_t) * 16));
    int64_t* i64 = reinterpret_cast<int64_t*>(take(sizeof(int64_t) * 8));
    double* f64 = reinterpret_cast<double*>(take(sizeof(double) * 4));
    // node arrays: fst, S, F, buf_ld, sn_neg, sn_fail, sn_bad (int32); buf_off, linv_off (int64)
    int32_t hi32[16] = {0, (int32_t)n, (int32_t)n, (int32_t)lda, 0, -1, 0};
    int64_t hi64[8] = {0, 0};
    Stats init{};
    init.first_zero = 0x7fffffff;
    // jobs of every step (host side, fixed-size per block, no allocation)
    struct StepJobs {
        int64_t panel_begin, panel_tasks, upd_begin, upd_jobs, upd_tasks;
    };
    constexpr int kMaxBlocks = 1024;
    if (nblk > kMaxBlocks) return -3;
    static thread_local Job hjobs[3 * kMaxBlocks];
    static thread_local StepJobs steps[kMaxBlocks];
    int64_t nj = 0;
    auto tiles = [](int64_t c0, int64_t c_end, int64_t r_end) -> int64_t {
        const int64_t nct = (c_end - c0 + kTile - 1) / kTile, nr = (r_end - c0 + kTile - 1) / kTile;
        return nct * nr - nct * (nct - 1) / 2;
    };
    for (int64_t stp = 0; stp < nblk; ++stp) {
        const int32_t k0 = (int32_t)(stp * kNB);
        const int32_t nb = (int32_t)std::min<int64_t>(kNB, n - k0);
        const int32_t c0 = k0 + nb;
        StepJobs& sj = steps[stp];
        sj.panel_begin = nj;
        sj.panel_tasks = (n - c0 + kTRSMRows - 1) / kTRSMRows;
        hjobs[nj++] = Job{0, c0, c0, (int32_t)n, k0, c0, 0};
        sj.upd_begin = nj;
        sj.upd_jobs = 0;
        sj.upd_tasks = 0;
        const int32_t sp0 = (k0 / kSuperPanel) * kSuperPanel;
        const int32_t sp1 = (int32_t)std::min<int64_t>(sp0 + kSuperPanel, n);
        if (c0 < sp1) {
            hjobs[nj] = Job{0, c0, sp1, (int32_t)n, k0, c0, sj.upd_tasks};
            sj.upd_tasks += tiles(c0, sp1, n);
            ++nj;
            ++sj.upd_jobs;
        }
        if (c0 == sp1 && sp1 < n) {
            hjobs[nj] = Job{0, sp1, (int32_t)n, (int32_t)n, sp0, sp1, sj.upd_tasks};
            sj.upd_tasks += tiles(sp1, n, n);
            ++nj;
            ++sj.upd_jobs;
        }
    }
    CK(cudaMemcpyAsync(jobs, hjobs, sizeof(Job) * nj, cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(i32, hi32, sizeof(hi32), cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(i64, hi64, sizeof(hi64), cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(st, &init, sizeof(Stats), cudaMemcpyHostToDevice, s));
    CK(cudaMemsetAsync(f64, 0, sizeof(double) * 4, s));
    // the pivot test compares with the diagonal before factorisation (sprfc1.f:1272-1279)
    CK(cudaMemcpy2DAsync(adiag, sizeof(double), a, (lda + 1) * sizeof(double), sizeof(double), n,
                         cudaMemcpyDeviceToDevice, s));
    PV pv{};
    pv.fst = i32 + 0;
    pv.S = i32 + 1;
    pv.F = i32 + 2;
    pv.buf_ld = i32 + 3;
    pv.sn_neg = i32 + 4;
    pv.sn_fail = i32 + 5;
    pv.sn_bad = i32 + 6;
    pv.buf_off = i64 + 0;
    pv.linv_off = i64 + 1;
    pv.arena = a;
    pv.dvec = d;
    pv.lnz = nullptr;
    pv.adiag = adiag;
    pv.linv = linv;
    pv.sn_faild = f64 + 0;
    pv.sn_faila = f64 + 1;
    pv.st = st;
    pv.tol1 = tol1;
    for (int64_t stp = 0; stp < nblk; ++stp) {
        const StepJobs& sj = steps[stp];
        k_diag<kPivotLDL><<<1, 256, kDiagSmem, s>>>(jobs + sj.panel_begin, pv, 0);
        if (sj.panel_tasks > 0) k_trsm<<<(int)sj.panel_tasks, 128, kTrsmSmem, s>>>(jobs + sj.panel_begin, 1, nullptr, pv);
        if (sj.upd_tasks > 0)
            K_GEMM_SMALL<<<(int)sj.upd_tasks, GemmSmall::NT, GemmSmall::smem, s>>>(jobs + sj.upd_begin, sj.upd_jobs, nullptr,
                                                                                 pv);
    }
    CK(cudaGetLastError());
    Stats hs;
    int32_t hfail = -1;
    double hf[2] = {0.0, 0.0};
    CK(cudaMemcpyAsync(&hs, st, sizeof(Stats), cudaMemcpyDeviceToHost, s));
    CK(cudaMemcpyAsync(&hfail, i32 + 5, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    CK(cudaMemcpyAsync(hf, f64, sizeof(hf), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    // out[0]=NUMNEG out[1]=first failing column (1-based, 0 if none) out[2]=failing pivot out[3]=its a_jj
    // out[4]=max(a_jj/d_j)
    out[0] = (double)hs.numneg;
    out[1] = hs.pivot_fail ? (double)(hfail + 1) : 0.0;
    out[2] = hf[0];
    out[3] = hf[1];
    out[4] = hs.tol2;
    return 0;
}

// ---------------------------------------------------------------------------
// Autotuner of the mixed-mode factorisation: which Schur updates go to the
// tensor cores (launches of at least tc_min_flops; the rest stay on the FP64
// kernel) and how many SMs the side-stream tensor-core launches may take.
// Every candidate factors a copy of the assembled SM twice (the second,
// graph-replayed pass is timed); the fastest is kept.  out[0] = chosen
// tc_min_flops, out[1] = chosen quarters of the SMs, out[2] = its factor ms,
// out[3] = factor ms of the default choice, out[4] = candidates tried.
// ---------------------------------------------------------------------------
int Engine::autotune(const double* d_sm_assembled, double* out) {
    const int64_t n = P_.neq + P_.nzerol;
    double* work = nullptr;
    CK(cudaMalloc((void**)&work, n * sizeof(double)));
    const int mode0 = mixed_;
    const double t0 = tc_min_flops_;
    const int q0 = far_cap_q_;
    mixed_ = 1;
    const double mins[] = {0.0, 1.0e9, 1.0e10, 1.0e11, 1.0e300};
    const int caps[] = {2, 3, 4};
    double best = 1e300, best_min = 0.0, def_ms = 0.0;
    int best_cap = 3, tried = 0, rc = 0;
    for (double m : mins)
        for (int q : caps) {
            if (m >= 1.0e300 && q != 3) continue;              // no tensor-core launches: the cap is moot
            tc_min_flops_ = m;
            far_cap_q_ = q;
            float ms = 0.f;
            for (int rep = 0; rep < 2 && rc == 0; ++rep) {
                if (cudaMemcpyAsync(work, d_sm_assembled, n * sizeof(double), cudaMemcpyDeviceToDevice, stream_) !=
                    cudaSuccess) {
                    rc = -4;
                    break;
                }
                FactorResult r;
                rc = factor(work, 1.0e-12, r);
                ms = timing.factor_ms;
            }
            if (rc != 0) break;
            ++tried;
            if (m == 0.0 && q == 3) def_ms = ms;
            if (ms < best) {
                best = ms;
                best_min = m;
                best_cap = q;
            }
        }
    cudaFree(work);
    mixed_ = mode0;
    if (rc != 0) {
        tc_min_flops_ = t0;
        far_cap_q_ = q0;
        return rc;
    }
    tc_min_flops_ = best_min;
    far_cap_q_ = best_cap;
    out[0] = best_min;
    out[1] = best_cap;
    out[2] = best;
    out[3] = def_ms;
    out[4] = tried;
    return 0;
}

// Tile shape of the small Schur updates (those with fewer than 4 x 64 rows):
// each candidate (64 x 64 tiles, 32 x 32 tiles) factors a copy of the
// assembled SM twice and the faster one is kept.  out[0] = the tile chosen,
// out[1] / out[2] = factor ms with 64 / 32.
int Engine::autotune_tiles(const double* d_sm_assembled, double* out) {
    const int64_t n = P_.neq + P_.nzerol;
    double* work = nullptr;
    CK(cudaMalloc((void**)&work, n * sizeof(double)));
    const int t0 = small_tile_;
    const int cand[2] = {kTile, kTileTiny};
    double ms[2] = {0.0, 0.0};
    int rc = 0;
    for (int c = 0; c < 2 && rc == 0; ++c) {
        small_tile_ = cand[c];
        float best = 1e30f;
        for (int rep = 0; rep < 2 && rc == 0; ++rep) {
            if (cudaMemcpyAsync(work, d_sm_assembled, n * sizeof(double), cudaMemcpyDeviceToDevice, stream_) !=
                cudaSuccess) {
                rc = -4;
                break;
            }
            FactorResult r;
            rc = factor(work, 1.0e-12, r);
            best = std::min(best, timing.factor_ms);
        }
        ms[c] = best;
    }
    cudaFree(work);
    if (rc != 0) {
        small_tile_ = t0;
        return rc;
    }
    small_tile_ = ms[1] < ms[0] ? kTileTiny : kTile;
    out[0] = small_tile_;
    out[1] = ms[0];
    out[2] = ms[1];
    return 0;
}

// ---------------------------------------------------------------------------
// Iterative refinement against the FP64 matrix
// ---------------------------------------------------------------------------
int Engine::build_residual(const double* d_sm_assembled) {
    Dev& D = *d_;
    cudaStream_t s = stream_;
    PV pv = make_view(D, P_, const_cast<double*>(d_sm_assembled), 0.0);
    const int64_t neq = P_.neq;
    // the row arrays and the scratch stay with the handle (each asked for by itself: an
    // earlier call may have got some of them only); the entry arrays grow
    csr_.nnz = -1;                                       // no matrix until this one is complete
    if (!csr_.rowptr) CK(alloc((void**)&csr_.rowptr, (neq + 1) * sizeof(int64_t)));
    if (!csr_.fill) CK(alloc((void**)&csr_.fill, (neq + 1) * sizeof(int64_t)));
    if (!csr_.cnt) CK(alloc((void**)&csr_.cnt, neq * sizeof(int)));
    CK(cudaMemsetAsync(csr_.cnt, 0, neq * sizeof(int), s));
    CK(cudaMemsetAsync(D.hbuf, 0, sizeof(unsigned long long), s));
    const int grid = (int)std::min<int64_t>((neq * 32 + 255) / 256, 16 * (int64_t)std::max(sm_count_, 1));
    k_csr_count<<<grid, 256, 0, s>>>(pv, P_.nsuper, neq, csr_.cnt);
    k_csr_scan<<<1, 1024, 0, s>>>(csr_.cnt, neq, csr_.rowptr, csr_.fill);
    k_mailbox<<<1, 32, 0, s>>>(reinterpret_cast<const unsigned long long*>(csr_.rowptr + neq), 1, D.mbox_dev);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(s));
    const int64_t nnz = (int64_t)D.mbox[0];
    if (csr_.cap < nnz || !csr_.ci) {
        for (void* p : {(void*)csr_.ci, (void*)csr_.cv, (void*)csr_.ci2, (void*)csr_.cv2}) cudaFree(p);
        csr_.ci = csr_.ci2 = nullptr;
        csr_.cv = csr_.cv2 = nullptr;
        csr_.cap = 0;
        const int64_t n = std::max<int64_t>(nnz, 1);
        CK(alloc((void**)&csr_.ci, n * sizeof(int32_t)));
        CK(alloc((void**)&csr_.cv, n * sizeof(double)));
        CK(alloc((void**)&csr_.ci2, n * sizeof(int32_t)));
        CK(alloc((void**)&csr_.cv2, n * sizeof(double)));
        csr_.cap = nnz;
    }
    k_csr_fill<<<grid, 256, 0, s>>>(pv, P_.nsuper, neq, csr_.fill, csr_.ci2, csr_.cv2);
    k_csr_rank<<<grid, 256, 0, s>>>(csr_.rowptr, neq, csr_.ci2, csr_.cv2, csr_.ci, csr_.cv, D.hbuf);
    k_mailbox<<<1, 32, 0, s>>>(D.hbuf, 1, D.mbox_dev);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(s));
    std::memcpy(&csr_.norm_inf, D.mbox, sizeof(double));
    csr_.nnz = nnz;
    return 0;
}

int Engine::residual(const double* d_b, const double* d_x, double* d_r, int64_t ld, int64_t nrhs, double* berr) {
    if (csr_.nnz < 0) return -2;
    cudaStream_t s = stream_;
    if (nbuf_cap_ < 3 * nrhs) {
        if (nbuf_) cudaFree(nbuf_);
        nbuf_ = nullptr;
        nbuf_cap_ = 0;
        CK(alloc((void**)&nbuf_, 3 * nrhs * sizeof(double)));
        nbuf_cap_ = 3 * nrhs;
    }
    double* norms = nbuf_;
    CK(cudaMemsetAsync(norms, 0, 3 * nrhs * sizeof(double), s));
    const int64_t neq = P_.neq;
    constexpr int kW = kResThreads / 32;
    const int grid =
        (int)std::max<int64_t>(1, std::min<int64_t>((neq + kW - 1) / kW, 8 * (int64_t)std::max(sm_count_, 1)));
    for (int64_t q0 = 0; q0 < nrhs; q0 += kMaxRHS) {          // kMaxRHS right-hand sides per pass
        const int nq = (int)std::min<int64_t>(kMaxRHS, nrhs - q0);
        const int64_t o = q0 * ld;
        if (nq <= 4)
            k_residual<4><<<grid, kResThreads, 0, s>>>(csr_.rowptr, csr_.ci, csr_.cv, neq, d_b + o, d_x + o, d_r + o,
                                                       ld, nq, norms + 3 * q0);
        else
            k_residual<kMaxRHS><<<grid, kResThreads, 0, s>>>(csr_.rowptr, csr_.ci, csr_.cv, neq, d_b + o, d_x + o,
                                                             d_r + o, ld, nq, norms + 3 * q0);
    }
    CK(cudaGetLastError());
    std::vector<double> h(3 * nrhs);
    CK(cudaMemcpyAsync(h.data(), norms, 3 * nrhs * sizeof(double), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    double worst = 0.0;
    for (int64_t q = 0; q < nrhs; ++q) {
        const double den = csr_.norm_inf * h[3 * q + 1] + h[3 * q + 2];
        worst = std::max(worst, den > 0.0 ? h[3 * q] / den : 0.0);
    }
    *berr = worst;
    return 0;
}

int Engine::refine(const double* d_sm, const double* d_b, double* d_x, int64_t ld, int64_t nrhs, double tol,
                   int maxit, double* out) {
    Dev& D = *d_;
    cudaStream_t s = stream_;
    const int64_t n = ld * nrhs;
    if (rbuf_cap_ < n) {
        if (rbuf_) cudaFree(rbuf_);
        rbuf_ = nullptr;
        rbuf_cap_ = 0;
        CK(alloc((void**)&rbuf_, n * sizeof(double)));
        rbuf_cap_ = n;
    }
    (void)D;
    CK(cudaMemcpyAsync(d_x, d_b, n * sizeof(double), cudaMemcpyDeviceToDevice, s));
    if (solve(d_sm, d_x, ld, nrhs, 3) != 0) return -4;
    float solve_ms = timing.solve_ms;
    double berr = 0.0;
    int it = 0;
    for (;;) {
        if (residual(d_b, d_x, rbuf_, ld, nrhs, &berr) != 0) return -4;
        if (berr <= tol || it >= maxit) break;
        if (solve(d_sm, rbuf_, ld, nrhs, 3) != 0) return -4;
        solve_ms += timing.solve_ms;
        k_axpy<<<(int)((n + 255) / 256), 256, 0, s>>>(d_x, rbuf_, n);
        ++it;
    }
    CK(cudaStreamSynchronize(s));
    out[0] = it;
    out[1] = berr;
    out[2] = solve_ms;
    return 0;
}

// Self-test of recip_nr: out[2i] = recip_nr(x[i]), out[2i+1] = 1.0 / x[i]
// (host arrays, n values).
int recip_check(const double* h_x, int64_t n, double* h_out) {
    double *dx = nullptr, *dout = nullptr;
    CK(cudaMalloc((void**)&dx, std::max<int64_t>(n, 1) * sizeof(double)));
    CK(cudaMalloc((void**)&dout, std::max<int64_t>(2 * n, 1) * sizeof(double)));
    CK(cudaMemcpy(dx, h_x, n * sizeof(double), cudaMemcpyHostToDevice));
    if (n > 0) k_recip_check<<<(int)((n + 255) / 256), 256>>>(dx, n, dout);
    CK(cudaGetLastError());
    CK(cudaMemcpy(h_out, dout, 2 * n * sizeof(double), cudaMemcpyDeviceToHost));
    cudaFree(dx);
    cudaFree(dout);
    return 0;
}

}  // namespace sprb
