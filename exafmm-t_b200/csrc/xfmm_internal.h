// xfmm_internal.h -- shared internals of libexafmm_b200.so (not part of the ABI).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <memory>
#include <stdexcept>
#include <string>
#include <vector>

#include "xfmm.h"

namespace xfmm {

struct Error : std::exception {
  int code;
  std::string msg;
  Error(int c, std::string m) : code(c), msg(std::move(m)) {}
  const char* what() const noexcept override { return msg.c_str(); }
};

#define XFMM_STR2(x) #x
#define XFMM_STR(x) XFMM_STR2(x)
#define XCUDA(call)                                                                                         \
  do {                                                                                                      \
    cudaError_t e_ = (call);                                                                                \
    if (e_ != cudaSuccess)                                                                                  \
      throw ::xfmm::Error(e_ == cudaErrorMemoryAllocation ? XFMM_ERR_OOM : XFMM_ERR_CUDA,                   \
                          std::string(__FILE__ ":" XFMM_STR(__LINE__) " ") + #call + ": " + cudaGetErrorString(e_)); \
  } while (0)
#define XREQUIRE(cond, code, msg)                     \
  do {                                                \
    if (!(cond)) throw ::xfmm::Error((code), (msg));  \
  } while (0)
#define XLAUNCH() XCUDA(cudaGetLastError())

// Device memory of the buffers below (pool.cpp).  A cudaMalloc or cudaFree takes 50 to 100 us, and a set-up at new
// positions makes about a hundred of each: blocks that are released while an Fmm handle lives are kept for
// the next allocations, at most POOL_KEEP bytes per device; the kept blocks go back to the device when the last
// Fmm handle is freed, and whenever an allocation fails.  A block is kept only once nothing in flight can
// touch it, and any other goes to cudaFree.  Waiting for the whole device would tell, but CUDA forbids it while any
// stream captures, and breaks that capture; so every object knows the work that used it (Uses), and a release
// waits for that work alone.  Any thread may allocate and release.
cudaError_t pool_alloc(size_t bytes, void** p, size_t* capacity);
size_t pool_capacity(size_t bytes);  // of the block that an allocation takes
void pool_release(void* p, size_t capacity) noexcept;
void pool_hold();            // an Fmm handle was created
void pool_unhold() noexcept;  // ... was freed

// The device work that used an object: per stream (by its id) an event behind the last of it, and per call that was
// captured an event that every launch of the graph records.  Like the handles, for one thread at a time.
struct Uses {
  struct Event {
    cudaEvent_t e = nullptr;
    Event() = default;
    Event(const Event&) = delete;
    Event& operator=(const Event&) = delete;
    ~Event() {
      if (e) cudaEventDestroy(e);
    }
  };
  std::vector<std::pair<unsigned long long, std::shared_ptr<Event>>> last;
  std::vector<std::shared_ptr<Event>> graphs;
  bool unknown = false;        // work that no event tells the end of
  bool wait() const noexcept;  // waits for the work; false: unknown, or an error
};
// One call of the C API: its work on stream s uses the objects; they learn of it at the end of the scope.  Blocks that
// the scope allocated itself are idle once s is, others once the objects' earlier work is done too.
class UseScope {
 public:
  UseScope(cudaStream_t s, std::vector<Uses*> objects);
  ~UseScope();
  UseScope(const UseScope&) = delete;
  UseScope& operator=(const UseScope&) = delete;
  bool idle(uint64_t allocated) const noexcept;  // waits until a block with that allocation number is idle

 private:
  cudaStream_t s_;
  std::vector<Uses*> objects_;
  uint64_t begin_;
  bool capturing_;
  UseScope* outer_;
};
// The freeing of an object: waits for its work, and its blocks can be kept.
class FreeScope {
 public:
  explicit FreeScope(const Uses& u) noexcept;
  ~FreeScope();
  FreeScope(const FreeScope&) = delete;
  FreeScope& operator=(const FreeScope&) = delete;
};

// Owning device buffer (move-only).
template <class T>
struct DBuf {
  T* p = nullptr;
  size_t n = 0, cap = 0;  // elements; bytes of the block
  DBuf() = default;
  explicit DBuf(size_t count) { alloc(count); }
  DBuf(const DBuf&) = delete;
  DBuf& operator=(const DBuf&) = delete;
  DBuf(DBuf&& o) noexcept : p(o.p), n(o.n), cap(o.cap) { o.p = nullptr; o.n = o.cap = 0; }
  DBuf& operator=(DBuf&& o) noexcept {
    if (this != &o) {
      release();
      p = o.p;
      n = o.n;
      cap = o.cap;
      o.p = nullptr;
      o.n = o.cap = 0;
    }
    return *this;
  }
  ~DBuf() { release(); }
  void alloc(size_t count) {
    release();
    if (!count) return;
    void* block = nullptr;
    XCUDA(pool_alloc(count * sizeof(T), &block, &cap));
    p = static_cast<T*>(block);
    n = count;
  }
  // grow-only reallocation (contents not preserved)
  void reserve(size_t count) {
    if (count > n) alloc(count);
  }
  void release() {
    if (p) pool_release(p, cap);
    p = nullptr;
    n = cap = 0;
  }
  size_t bytes() const { return n * sizeof(T); }
  void upload(const T* h, size_t count, cudaStream_t s) {
    reserve(count);
    if (count) XCUDA(cudaMemcpyAsync(p, h, count * sizeof(T), cudaMemcpyHostToDevice, s));
  }
  void upload(const std::vector<T>& h, cudaStream_t s) { upload(h.data(), h.size(), s); }
  std::vector<T> download(cudaStream_t s, size_t count = (size_t)-1) const {
    if (count == (size_t)-1) count = n;
    std::vector<T> h(count);
    if (count) {
      XCUDA(cudaMemcpyAsync(h.data(), p, count * sizeof(T), cudaMemcpyDeviceToHost, s));
      XCUDA(cudaStreamSynchronize(s));
    }
    return h;
  }
};

constexpr int LMAX = 21;  // path keys hold 21 octant digits (63 bits): deepest supported level

inline int nsurf_of(int p) { return 6 * (p - 1) * (p - 1) + 2; }

struct Workspace;  // evaluate buffers, one per precision (evaluate.cu)
struct Tree;
void release_workspace(Tree& t);

// Tree + interaction lists on the device, node arrays in the reference's idx order.
struct Tree {
  Uses uses;
  Workspace* ws[2] = {nullptr, nullptr};  // evaluate workspace per precision
  Tree() = default;
  Tree(const Tree&) = delete;
  Tree& operator=(const Tree&) = delete;
  ~Tree() { release_workspace(*this); }
  int64_t nsrc = 0, ntrg = 0;
  int nnodes = 0, nleafs = 0, nnonleafs = 0, depth = 0, nonadaptive = 0, ncrit = 0, nsurf_lists = 0;
  double x0[3] = {0, 0, 0}, r0 = 0;
  // bodies in tree order: (x, y, z, Re q) and Im q for complex charges
  DBuf<double4> src4, trg4;
  DBuf<double> src_qim;
  DBuf<int> src_perm, trg_perm;
  // nodes
  DBuf<int> level, is_leaf, nsrcs, ntrgs, parent, octant, child0;
  DBuf<int64_t> sbeg, tbeg;
  DBuf<double4> center;  // x, y, z, r
  DBuf<uint64_t> key;    // the reference's Morton key with level offset (hilbert.h:79-107)
  DBuf<int> leafs, nonleafs;
  std::vector<int> h_level, h_is_leaf, h_child0, h_leafs, h_nonleafs, h_ntrgs, h_nsrcs;
  // lists
  bool lists_built = false;
  DBuf<int> colleagues, m2l;
  DBuf<int64_t> p2p_off, m2p_off, p2l_off;
  DBuf<int> p2p, m2p, p2l;
  int64_t np2p = 0, nm2p = 0, np2l = 0;
  // derived schedules
  DBuf<int> nl_by_level;              // nonleafs grouped by level (ascending), pre-order within a level
  std::vector<int> nl_level_off;      // depth+2 offsets into nl_by_level
  DBuf<int> eval_leafs;               // leaf positions (index into leafs) with ntrgs > 0
  int n_eval_leafs = 0;
  DBuf<int> p2l_nodes;                // nodes with a non-empty P2L list
  int n_p2l_nodes = 0;
  DBuf<float> leaf_scale;             // 0.5^level per leaf position (Laplace P2M/L2P scaling)
  DBuf<double> leaf_scale64;
  int64_t p2p_pairs = 0, m2p_pairs = 0, l2p_pairs = 0, m2l_pairs = 0;
  // M2L setup (fmm_scale_invariant.h:277-341 / fmm.h:265-333)
  bool m2l_ready = false;
  int m2l_grouped_by_level = 0;
  DBuf<int> m2l_src;                  // compact source list (node idx), grouped by level if per-level
  std::vector<int> m2l_src_off;       // group offsets
  DBuf<int> m2l_trg;                  // targets (nonleaf node idx), same grouping
  std::vector<int> h_m2l_trg;         // host copy
  std::vector<int> m2l_trg_off;
  DBuf<int> m2l_tab;                  // [n_trg][26] compact source index within its group, -1 if none
  std::vector<int> h_m2l_tab;
  DBuf<float> m2l_scale;              // per target 2^(level+1) (Laplace) else 1
  DBuf<double> m2l_scale64;
  int n_m2l_src = 0, n_m2l_trg = 0;
  // persistent staging for host-side charges and results (no allocation per call)
  DBuf<double> stage_q, stage_out;
  DBuf<int> stage_flag;               // non-finite charges found by the device-side check
  int hadr_tpc = 0;                   // M2L Hadamard, mixed path: target tiles per CTA (0: the built-in default)
};

// Precomputed operators of one level (or the single scale-invariant level).
struct LevelOps {
  // working precision copies (float for mixed, double for fp64); complex types stored as interleaved pairs
  // K(check, equiv) = U S V^H; the pseudo-inverse is applied in FP64 (both precisions), in two factors as the
  // reference does (UC2E_U then UC2E_V, DC2E_U then DC2E_V), never as one product: P = V S+ U^H
  // has entries up to ~1/s_min and a single dot product with it cancels catastrophically.
  DBuf<char> p2m_B1;   // [n][n]      y = U^H c        : B1[k][j] = conj(U[k][j])
  DBuf<char> p2m_B2;   // [n][n]      e = V S+ y       : B2[k][j] = conj(VH[k][j]) / s_k
  DBuf<char> l2p_B1;   // [n][n]      y = conj(VH) c   : B1[k][j] = conj(VH[j][k])
  DBuf<char> l2p_B2;   // [n][n]      e = conj(U) S+ y : B2[k][j] = conj(U[j][k]) / s_k
  DBuf<char> l2p_B1f;  // FP32 copy of l2p_B1 (mixed path, real kernels: the L2P first factor runs in FP32)
  DBuf<char> m2m_B;    // [8n][n]     B[c*n+k][j] = M2M[c][j][k], M2M[c] = (V S+)(U^H K_c)
  DBuf<char> l2l_B;    // [n][8n]     B[k][c*n+j] = M2M[c][k][j] (L2L = M2M^T)
  // M2L tables ([26][nfreq][64] complex, entry [s*8+t]; fmm_scale_invariant.h:549-551) as the Hadamard's
  // fragments per frequency: FP64, or FP16 head / tail for the mixed path (m2l_fragments)
  DBuf<char> m2l_frag;
  DBuf<float> m2l_binv;  // mixed: [window][nfreq][32], undoes the exponent of each block
  int m2l_windows = 1;   // mixed: windows of the factors' exponents (k_m2l_fragments)
  uint64_t m2l_id = 0;   // another number for every table built: memory addresses come again
  int rank = 0;        // singular values kept by the pinv threshold: B1 columns / B2 rows beyond are zero
  // the same operators in the form the translation GEMMs (translate.cu) read: real [K][N] row-major, a
  // complex operator expanded to [2K][2N] (expand_operator); FP64 for the pinv factors and the FP64
  // path, TF32 head / tail arrays for the mixed path's M2M, L2L and (real kernels) L2P first factor
  DBuf<double> tg_p2m1, tg_p2m2, tg_l2p1, tg_l2p2, tg_m2m, tg_l2l;
  DBuf<float> tg_m2m_h, tg_m2m_l, tg_l2l_h, tg_l2l_l, tg_l2p1_h, tg_l2p1_l;  // mixed: transposed [N][ld]
  int64_t ld_m2m = 0, ld_l2l = 0, ld_l2p1 = 0;
};

struct Fmm {
  Uses uses;
  int kernel = 0, p = 0, ncrit = 0, precision = 0;
  double k_re = 0, k_im = 0;
  int nsurf = 0, nconv = 0, nfreq = 0, n1 = 0;
  int depth = 0;
  double x0[3] = {0, 0, 0}, r0 = 0;
  std::string filename;               // operator file in the reference's .dat layout ("" : none)
  bool precomputed = false;
  double pre_r0 = -1;
  int pre_depth = -1;
  std::vector<LevelOps> ops;          // 1 (Laplace) or depth+1 (per-level kernels)
  DBuf<double> surf_base;             // [nsurf][3] unit surface (geometry.h:21-54 before scaling)
  DBuf<int> surf_perm;                // surface points line by line along x, then y (host_surface_lines)
  DBuf<double> surf_grid;             // [p] grid coordinates of the unit surface along one axis
  DBuf<int> map_up, map_dn;           // surface index -> conv-grid index (geometry.h:101-134)
  DBuf<int> conv_to_surf_up;          // conv-grid index -> surface index or -1
  DBuf<double> dft_tw;                // [n1] (cos, sin)(2 pi m / n1): factors of the M2L transforms
  std::vector<double> h_surf_base;
  double stage_ms[11] = {0};
  bool is_complex() const { return kernel == XFMM_HELMHOLTZ; }
  // the field falls off exponentially
  bool screened() const { return kernel == XFMM_MODIFIED_HELMHOLTZ || (kernel == XFMM_HELMHOLTZ && k_im != 0); }
  bool mixed() const { return precision == XFMM_MIXED; }
};

// tree.cu
void build_tree(Fmm& fmm, Tree& t, const double* src_xyz, const double* trg_xyz, int nonadaptive_depth,
                cudaStream_t s);
void build_lists(Fmm& fmm, Tree& t, cudaStream_t s);
void m2l_setup(Fmm& fmm, Tree& t, cudaStream_t s);
// precompute.cu
void precompute(Fmm& fmm, int depth, cudaStream_t s);
void host_surface_base(int p, std::vector<double>& out);
void host_surface_lines(int p, const std::vector<double>& base, std::vector<int>& perm, std::vector<double>& grid);
// evaluate.cu
void m2l_fragments(LevelOps& op, const double* T64, int nfreq, bool mixed, bool screened, cudaStream_t s);
void set_charges(Fmm& fmm, Tree& t, const double* q, bool on_device, cudaStream_t s);
void clear_values(Fmm& fmm, Tree& t, cudaStream_t s);
void upward_pass(Fmm& fmm, Tree& t, cudaStream_t s);
void downward_pass(Fmm& fmm, Tree& t, cudaStream_t s);
void get_values(Fmm& fmm, Tree& t, double* out_dev, cudaStream_t s);
void stage_times(Fmm& fmm, Tree& t, double* ms14);
void check_device_status(Fmm& f, Tree& t);
void selftest_bounded_wait(int64_t limit_cycles);
void gradient_p2p_raw(int kernel, double k_re, double k_im, int precision, const double* src, int64_t ns,
                      const double* q, const double* trg, int64_t nt, double* out, cudaStream_t s);
void verify(Fmm& fmm, Tree& t, int sample, double* err2, cudaStream_t s);
void gradient_p2p_scratch(int kernel, double k_re, double k_im, int precision, const double* src, int64_t ns,
                          const double* q, const double* trg, int64_t nt, double* out, double4* s4, double* qim,
                          double4* t4, cudaStream_t s);
// translate.cu: level-batched translation GEMMs with fused row gather / scale / scatter.
// C[coff[r] + j] (=|+=) alpha[r] * sum_k A[aoff[r] + k] * B[k * ldb + j] for r < M, j < N, k < K, on
// real views of the rows (complex rows as interleaved reals, operators expanded).
struct TGemm {
  int M = 0, N = 0, K = 0;
  const int64_t* aoff = nullptr;
  const int64_t* coff = nullptr;
  const double* alpha = nullptr;  // null: 1
  int64_t ldb = 0;
  int accumulate = 0;
  int64_t astep = 0;  // every A offset is a multiple of astep elements (alignment of the A rows)
  int* status = nullptr;  // device flag set by a tensor-core GEMM whose bounded wait ran out
  double* scratch = nullptr;  // tile counters (zero between uses) and partial sums of a GEMM whose K is split
  int64_t scratch_len = 0;
};
template <class TA, class TC>
void tgemm_f64(const TGemm& g, const TA* A, const double* B, TC* C, cudaStream_t s);
template <class TC>
void tgemm_tc(const TGemm& g, const float* A, const float* Bth, const float* Btl, int64_t ldbt, TC* C,
              cudaStream_t s);
int64_t tgemm_tc_scratch(int M, int N, int K, int accumulate);  // scratch of a split GEMM in doubles (0: unsplit)
int64_t tgemm_f64_scratch(int M, int N, int K);
void expand_operator_t(const void* B, bool b_single, int K, int N, int64_t ldb, bool cplx, int npad, int64_t ldbt,
                       float* ohi, float* olo, cudaStream_t s);
void expand_operator(const void* B, bool b_single, int K, int N, int64_t ldb, bool cplx, double* o64, float* ohi,
                     float* olo, cudaStream_t s);
void prepare_translation_operands(const Fmm& f, LevelOps& op, cudaStream_t s);
// evaluate.cu: many systems in one evaluate (xfmm_batch_*)
struct Batch;
Batch* batch_create(Fmm** fmms, Tree** trees, int n, cudaStream_t s);
void batch_free(Batch* b);
std::vector<Uses*> batch_uses(Batch* b);  // of the batch and its systems
void batch_schedule(const int64_t* sizes, int n, int nstreams, int* stream_of);
void batch_set_tuning(Batch* b, int option, int value);
void batch_evaluate(Batch* b, const double* const* charges, double* const* outs, int nstreams, cudaStream_t s);
// capi.cpp: record the message returned by xfmm_last_error() on this thread
void set_last_error(const char* msg);

}  // namespace xfmm
