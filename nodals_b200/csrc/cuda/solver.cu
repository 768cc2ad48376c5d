// Device SIMPLE solver: upload of the host setup, the pressure AMG V-cycle,
// the outer pressure solvers, one SIMPLE iteration, and the C ABI entry
// points nds_solver_*.  Numerics follow gpu/serial_cuda/h8_main_base.cu:
//   G4AMG::apply / explicit_vcycle        :544-564
//   smoothers cheb2 / jacobi / l1jacobi / mcgs  :425-542
//   pressure_pcg / richardson / cheb_poly  :569-611, :670-726
//   pressure_precond_power                 :613-668
//   g5_gpu_spectrum_refresh                :873-906
//   SIMPLE iteration                       :2046-2119
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <type_traits>
#include <vector>

#include "../capi_internal.hpp"
#include "../host/fem.hpp"
#include "common.cuh"
#include "kernels.cuh"
#include "krylov.cuh"
#include "mpnn.hpp"
#include "resident.cuh"
#include "split.cuh"

namespace nds {

unsigned long long g_launches = 0;

template <class T>
struct DBuf {
  T* p = nullptr;
  size_t n = 0;
  DBuf() = default;
  DBuf(const DBuf&) = delete;
  DBuf& operator=(const DBuf&) = delete;
  DBuf(DBuf&& o) noexcept : p(o.p), n(o.n) {
    o.p = nullptr;
    o.n = 0;
  }
  DBuf& operator=(DBuf&& o) noexcept {
    if (this != &o) {
      release();
      p = o.p;
      n = o.n;
      o.p = nullptr;
      o.n = 0;
    }
    return *this;
  }
  ~DBuf() { release(); }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
  }
  void alloc(size_t m) {
    release();
    n = m;
    if (m) NDS_CUDA(cudaMalloc((void**)&p, m * sizeof(T)));
  }
  template <class U>
  void upload(const std::vector<U>& h) {
    if constexpr (std::is_same<U, T>::value) {
      alloc(h.size());
      if (n) NDS_CUDA(cudaMemcpy(p, h.data(), n * sizeof(T), cudaMemcpyHostToDevice));
    } else {
      std::vector<T> t(h.begin(), h.end());
      alloc(t.size());
      if (n) NDS_CUDA(cudaMemcpy(p, t.data(), n * sizeof(T), cudaMemcpyHostToDevice));
    }
  }
  void zero(cudaStream_t s) {
    if (n) NDS_CUDA(cudaMemsetAsync(p, 0, n * sizeof(T), s));
  }
  size_t bytes() const { return n * sizeof(T); }
};

// Optional per-category CUDA-event timing of kernel launches on the solver's
// stream (the analogue of the reference's H0Profiler, h8_main_base.cu:58-99).
// fine_spmv: the physical fine operator (Krylov A p, power iterations);
// fine_spmv_amg: the fine-level operator inside the V-cycle
// fine_spmv_half: the V-cycle's fine-level operator in FP16 (amg_half)
enum ProfCat { P_FINE_SPMV = 0, P_COARSE_SPMV, P_REFRESH, P_ASSEMBLE, P_GS, P_CONTINUITY, P_TRANSFER, P_TERMINAL,
               P_VECTOR, P_FINE_AMG, P_FINE_HALF, P_RESIDENT, P_NCAT };
static const char* const kProfNames[P_NCAT] = {"fine_spmv", "coarse_spmv", "fine_refresh", "mom_assemble", "mom_gs",
                                               "continuity", "transfer", "terminal_dense", "vector_reduce",
                                               "fine_spmv_amg", "fine_spmv_half", "pcg_resident"};
struct Profiler {
  bool on = false;
  std::vector<cudaEvent_t> ev;
  std::vector<int> cat;
  int used = 0;
  double total[P_NCAT] = {};
  long long calls[P_NCAT] = {};
  ~Profiler() {
    for (auto e : ev) cudaEventDestroy(e);
  }
  int begin(cudaStream_t s, int c) {
    if (!on) return -1;
    if (2 * (size_t)used + 2 > ev.size()) {
      const size_t n = ev.size();
      ev.resize(n + 512);
      cat.resize(ev.size() / 2);
      for (size_t i = n; i < ev.size(); ++i) NDS_CUDA(cudaEventCreate(&ev[i]));
    }
    const int id = used++;
    cat[(size_t)id] = c;
    NDS_CUDA(cudaEventRecord(ev[2 * (size_t)id], s));
    return id;
  }
  void end(cudaStream_t s, int id) {
    if (id >= 0) NDS_CUDA(cudaEventRecord(ev[2 * (size_t)id + 1], s));
  }
  void collect() {
    if (!used) return;
    NDS_CUDA(cudaEventSynchronize(ev[2 * (size_t)used - 1]));
    for (int i = 0; i < used; ++i) {
      float ms = 0;
      NDS_CUDA(cudaEventElapsedTime(&ms, ev[2 * (size_t)i], ev[2 * (size_t)i + 1]));
      total[cat[(size_t)i]] += ms;
      ++calls[cat[(size_t)i]];
    }
    used = 0;
  }
  void reset() {
    used = 0;
    for (int c = 0; c < P_NCAT; ++c) { total[c] = 0; calls[c] = 0; }
  }
};
struct ProfScope {
  Profiler& p;
  cudaStream_t s;
  int id;
  ProfScope(Profiler& pp, cudaStream_t ss, int c) : p(pp), s(ss), id(pp.begin(ss, c)) {}
  ~ProfScope() { p.end(s, id); }
};

struct ISolver {
  virtual ~ISolver() = default;
  virtual void reset() = 0;
  virtual void step(nds_iter_report* rep) = 0;
  virtual void solve(nds_solve_report* rep) = 0;
  virtual void get_fields(double* u0, double* u1, double* u2, double* p) = 0;
  virtual void set_fields(const double* u0, const double* u1, const double* u2, const double* p) = 0;
  // set_fields(in), step, get_fields(out), with the read-back overlapped
  // with the step where the state type and the output memory allow it
  virtual void step_io(const double* const in[4], double* const out[4], nds_iter_report* rep) = 0;
  // device cell-plan arrays read by nds_continuity_noalloc; false unless the
  // state type is double
  virtual bool cell_arrays(const int32_t** ref, const double** bco, const double** fixed_div, int* nc,
                           int* device) const = 0;
  // learned pressure stage (precision mixed, FGMRES)
  virtual void load_stage(const float* host_params) = 0;
  virtual void stage_graph(int32_t* nbr, float* ew, float* dscale) = 0;
  virtual void pressure_pair(float* rhs, float* x) = 0;
  virtual void stage_counts(long long* applied, long long* fallbacks) = 0;
  virtual void apply_operator(const float* x, float* y) = 0;
  virtual void apply_operator_form(int form, const void* x, void* y) = 0;
  Profiler prof;
};

struct SolveFailure : std::runtime_error {
  int code;
  SolveFailure(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

namespace {

// Exceptions cannot leave an OpenMP region: the first message is kept and
// rethrown after the region.
struct OmpErr {
  bool bad = false;
  std::string msg;
  template <class F>
  void run(F&& f) {
    try {
      f();
    } catch (const std::exception& e) {
#pragma omp critical(nds_solver_omp_error)
      if (!bad) {
        bad = true;
        msg = e.what();
      }
    }
  }
  void rethrow() const {
    if (bad) throw std::runtime_error(msg);
  }
};

std::vector<int32_t> to_i32(const std::vector<int64_t>& v, const char* what) {
  std::vector<int32_t> o(v.size());
  for (size_t i = 0; i < v.size(); ++i) {
    if (v[i] > INT32_MAX) throw std::runtime_error(std::string(what) + " exceeds int32 offsets");
    o[i] = (int32_t)v[i];
  }
  return o;
}

// greedy colouring of a CSR graph in row order (h8_main_base.cu:125-180)
void greedy_color(int n, const std::vector<int32_t>& row, const std::vector<int32_t>& col, std::vector<int32_t>& rows_out,
                  std::vector<int>& off_out) {
  std::vector<int32_t> color((size_t)n, -1);
  std::vector<int> mark(64, -1);
  int nc = 0;
  for (int i = 0; i < n; ++i) {
    for (int k = row[(size_t)i]; k < row[(size_t)i + 1]; ++k) {
      const int j = col[(size_t)k];
      if (j == i) continue;
      const int cj = color[(size_t)j];
      if (cj >= 0) {
        if ((size_t)cj >= mark.size()) mark.resize((size_t)cj + 2, -1);
        mark[(size_t)cj] = i;
      }
    }
    int c = 0;
    while ((size_t)c < mark.size() && mark[(size_t)c] == i) ++c;
    if ((size_t)c >= mark.size()) mark.resize((size_t)c + 2, -1);
    color[(size_t)i] = c;
    nc = std::max(nc, c + 1);
  }
  off_out.assign((size_t)nc + 1, 0);
  for (int i = 0; i < n; ++i) ++off_out[(size_t)color[(size_t)i] + 1];
  for (int c = 0; c < nc; ++c) off_out[(size_t)c + 1] += off_out[(size_t)c];
  rows_out.resize((size_t)n);
  std::vector<int> next(off_out.begin(), off_out.end() - 1);
  for (int i = 0; i < n; ++i) rows_out[(size_t)next[(size_t)color[(size_t)i]]++] = i;
}

// Jacobi scaling and edge weights of the learned stage's graph from the
// current FP32 operator: dscale_i = 1 / sqrt(a_ii), e_ij = a_ij dscale_i dscale_j
// (a_ij read at its SELL offset off[4 i + k]; 0 for a boundary slot)
__global__ void stage_dscale(int n, const float* __restrict__ diag, float* __restrict__ dscale) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dscale[i] = diag[i] > 0.f ? rsqrtf(diag[i]) : 0.f;
}
__global__ void stage_edges(int n, const int32_t* __restrict__ nbr, const int32_t* __restrict__ off,
                            const float* __restrict__ val, const float* __restrict__ dscale, float* __restrict__ ew) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 4 * n) return;
  const int i = t >> 2, j = nbr[t];
  ew[t] = j >= 0 ? val[off[t]] * dscale[i] * dscale[j] : 0.f;
}
// after t = v - A z1: keep (t, z1) when ||t|| < ||v||, else fall back to the
// plain V-cycle (t = v, z1 = 0); counters: [0] applications, [1] fallbacks
__global__ void stage_select(int n, const float* __restrict__ v, float* __restrict__ t, float* __restrict__ z1,
                             const double* __restrict__ sc, int tt_slot, int vv_slot,
                             unsigned long long* __restrict__ cnt) {
  const bool bad = !(sc[tt_slot] < sc[vv_slot]);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    cnt[0] += 1;
    if (bad) cnt[1] += 1;
  }
  if (!bad) return;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    t[i] = v[i];
    z1[i] = 0.f;
  }
}
template <class Tin>
__global__ void to_float(int n, const Tin* __restrict__ a, float* __restrict__ b) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] = (float)a[i];
}

double cheb_root(double hi, double lo, int k, int degree) {
  const double centre = .5 * (hi + lo), radius = .5 * (hi - lo), pi = 3.141592653589793238462643383279502884;
  return centre - radius * std::cos(pi * (2.0 * (double)k + 1.0) / (2.0 * (double)degree));
}

}  // namespace

// T: state, momentum and pressure-operator precision (and the outer Krylov
// vectors); TA: precision of the AMG V-cycle (levels, transfers, smoothers,
// fine-level copy of the operator).  T == TA for the FP64 and FP32 modes;
// the mixed mode runs an FP32 V-cycle inside FP64 PCG.
template <class T, class TA>
class Solver final : public ISolver {
 public:
  static constexpr bool kSame = std::is_same<T, TA>::value;
  struct Level {  // explicit AMG level
    int n = 0;
    DBuf<int32_t> row, col, crows;
    std::vector<int> coff;
    DBuf<TA> val, diag, l1, b, x, r, tmp, corr, pong;
    // amg_half: FP16 copy of the level's CSR values, scaled by 1 / hinv,
    // and its columns as 16-bit deltas to the row when they all fit
    DBuf<__half> hval;
    DBuf<int16_t> hcol;
    double hinv = 1.0;
    // windows of x of the level's persistent SpMV (empty: not used)
    DBuf<int2> win;
    DBuf<int16_t> dcol;  // FP64 levels with windows: columns as 16-bit deltas to the row, when they fit
    int wrows = 0, wblocks = 0;
    size_t wsmem = 0;
  };
  struct Xfer {  // P (fine rows, ELL k-major) and R = P^T (coarse rows, CSR)
    int nf = 0, nc = 0, pw = 0;
    DBuf<int32_t> pcol, rrow, rcol;
    DBuf<TA> pval, rval;
  };

  Solver(const Problem& P) : P_(P), o_(P.opt) {
    NDS_CUDA(cudaSetDevice(o_.device));
    NDS_CUDA(cudaStreamCreateWithFlags(&st_, cudaStreamNonBlocking));
    NDS_CUDA(cudaStreamCreateWithFlags(&st2_, cudaStreamNonBlocking));
    NDS_CUDA(cudaStreamCreateWithFlags(&st_io_, cudaStreamNonBlocking));
    NDS_CUDA(cudaEventCreateWithFlags(&ev_io_, cudaEventDisableTiming));
    for (auto& e : ev_side_) NDS_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    for (auto& e : ev_) NDS_CUDA(cudaEventCreate(&e));
    upload();
  }
  ~Solver() override {
    for (auto& e : ev_)
      if (e) cudaEventDestroy(e);
    if (hsc_) cudaFreeHost(hsc_);
    if (hflags_) cudaFreeHost(hflags_);
    for (auto& e : ev_side_)
      if (e) cudaEventDestroy(e);
    if (ev_io_) cudaEventDestroy(ev_io_);
    if (st_io_) cudaStreamDestroy(st_io_);
    if (st2_) cudaStreamDestroy(st2_);
    if (st_) cudaStreamDestroy(st_);
  }

  // ------------------------------------------------------------------ setup
  void upload() {
    const Setup& S = P_.setup;
    const Hierarchy& H = P_.hier;
    StageTimer tm("device_upload");
    nc_ = S.nc;
    nv_ = S.nv;
    {
      // The momentum matrix is stored colour by colour: the Gauss-Seidel
      // pass of one colour then streams one contiguous block.  Each row
      // starts on a 32-byte boundary and is padded to a whole number of
      // 32-byte sectors (pad entries: column = the row itself, value 0), so
      // the assembly, which visits the rows in their natural order, writes
      // whole sectors.  The assembly and the audit address row i through
      // its span; the pads add zeros, so every value and sum is the one of
      // the natural order.  NDS_MOM_NATURAL_ORDER=1 keeps the natural CSR.
      const bool natural = std::getenv("NDS_MOM_NATURAL_ORDER") != nullptr;
      const int64_t pad = natural ? 1 : (int64_t)(32 / sizeof(T));
      int64_t nz = natural ? S.mom.row[(size_t)nv_] : 0;
      std::vector<int64_t> pos(natural ? 0 : (size_t)nv_);
      for (int q = 0; q < nv_ && !natural; ++q) {
        const int i = S.color_rows[(size_t)q];
        const int64_t len = S.mom.row[(size_t)i + 1] - S.mom.row[(size_t)i];
        pos[(size_t)i] = nz;
        nz += (len + pad - 1) / pad * pad;
      }
      if (nz > (int64_t)INT32_MAX) throw std::runtime_error("momentum CSR exceeds int32 offsets");
      std::vector<int32_t> col((size_t)nz), dpos((size_t)nv_);
      std::vector<int2> span((size_t)nv_);
      std::vector<T> kv((size_t)nz, T(0));
#pragma omp parallel for schedule(static)
      for (int i = 0; i < nv_; ++i) {
        const int64_t rb = S.mom.row[(size_t)i], re = S.mom.row[(size_t)i + 1];
        const int64_t cb = natural ? rb : pos[(size_t)i];
        const int64_t ce = natural ? re : cb + (re - rb + pad - 1) / pad * pad;
        span[(size_t)i] = make_int2((int)cb, (int)ce);
        dpos[(size_t)i] = (int32_t)(cb + (S.mom_diag_pos[(size_t)i] - rb));
        for (int64_t k = rb; k < re; ++k) {
          col[(size_t)(cb + (k - rb))] = S.mom.col[(size_t)k];
          kv[(size_t)(cb + (k - rb))] = (T)S.mom.val[(size_t)k];
        }
        for (int64_t k = cb + (re - rb); k < ce; ++k) col[(size_t)k] = i;
      }
      std::vector<int2> gspan((size_t)nv_);
#pragma omp parallel for schedule(static)
      for (int q = 0; q < nv_; ++q) gspan[(size_t)q] = span[(size_t)S.color_rows[(size_t)q]];
      mspan_.upload(span);
      gspan_.upload(gspan);
      mcol_.upload(col);
      mdpos_.upload(dpos);
      K_.upload(kv);
      A_.alloc((size_t)nz);
    }
    diag_.alloc((size_t)nv_);
    delta_.alloc((size_t)nv_);
    rau_.upload(S.init_rau);
    rau_pc_.upload(S.init_rau);
    inc_off_.upload(S.fine.inc_off);
    inc_.upload(S.fine.packed);
    ref_.upload(S.ref);
    slot_.upload(S.row_slot);
    det_.upload(S.det);
    invJ_.upload(S.invJ);
    bco_.upload(S.bco);
    fixed_.upload(S.fixed_value);
    fixed_div_.upload(S.fixed_div);
    for (int d = 0; d < 3; ++d) {
      s_[d].upload(S.static_rhs[(size_t)d]);
      b_[d].alloc((size_t)nv_);
      v_[d].alloc((size_t)nv_);
    }
    u3_.alloc((size_t)kVelComponents * nv_);
    NDS_CUDA(cudaMemset(u3_.p, 0, u3_.bytes()));
    p_.alloc((size_t)nc_);
    color_rows_.upload(S.color_rows);
    color_off_ = S.color_off;
    conv_table_.upload(conv_table());
    row_cap_ = 8;
    for (int i = 0; i < nv_; ++i) row_cap_ = std::max<int>(row_cap_, (int)(S.mom.row[(size_t)i + 1] - S.mom.row[(size_t)i]));
    row_cap_ = (row_cap_ + 7) / 8 * 8;
    mom_smem_ = (size_t)(kBlock / 8) * row_cap_ * sizeof(T);
    if (mom_smem_ > 200 * 1024) throw std::runtime_error("momentum row too long for the shared-memory assembly buffer");
    NDS_CUDA(cudaFuncSetAttribute(k::mom_assemble<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mom_smem_));
    NDS_CUDA(cudaFuncSetAttribute(k::mom_assemble<T, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(mom_smem_ + kConvTable * sizeof(T))));
    // The two-pass assembly by default: the cell pass writes each cell's
    // convection block row by row into the incidence slots of the velocity
    // rows (8 values per incidence, contiguous per row), the row pass
    // streams them.  NDS_FUSED_ASSEMBLY=1 (not with SUPG) evaluates the
    // convection rows inside the row pass instead.
    fused_assembly_ = !o_.supg && std::getenv("NDS_FUSED_ASSEMBLY") != nullptr;
    if (!fused_assembly_) {
      const size_t nz = S.fine.packed.size();
      std::vector<int32_t> zpos(8 * (size_t)nc_, -1);
      std::vector<uint8_t> slotz(8 * nz), fixz(nz, 0);
      std::vector<T> bz(3 * nz);
#pragma omp parallel for schedule(static)
      for (size_t z = 0; z < nz; ++z) {
        const uint32_t pa = S.fine.packed[z];
        const size_t c = pa >> 3, a = pa & 7u;
        zpos[8 * c + a] = (int32_t)z;
        for (int d = 0; d < 3; ++d) bz[3 * z + (size_t)d] = (T)S.bco[24 * c + 3 * a + (size_t)d];
        for (int b = 0; b < 8; ++b) {
          slotz[8 * z + (size_t)b] = S.row_slot[64 * c + 8 * a + (size_t)b];
          if (S.ref[8 * c + (size_t)b] < 0) fixz[z] |= (uint8_t)(1u << b);
        }
      }
      zpos_.upload(zpos);
      slotz_.upload(slotz);
      fixz_.upload(fixz);
      bz_.upload(bz);
      pz_.alloc(nz);
      cconv_.alloc(8 * nz);
    }

    if (o_.supg) {
      h2_.upload(S.h2);
      std::vector<double> rule;
      for (const auto& q : tet_rule_64()) {
        for (int k = 0; k < 4; ++k) rule.push_back(q.lam[(size_t)k]);
        rule.push_back(q.w);
      }
      supg_rule_.upload(rule);
    }

    tm.mark("momentum_and_cells");
    // The pressure operator: in split form, or as assembled rows (SELL) for
    // the smoothers that read a row's entries.
    split_ = o_.amg_smoother == NDS_SM_CHEB2 || o_.amg_smoother == NDS_SM_JACOBI;
    const FineTopo& F = S.fine;
    if (split_) upload_split();
    else upload_sell(tm);
    tm.mark("sell_layout");
    fdiag_.upload(H.fine_diag);
    const bool l1 = o_.amg_smoother == NDS_SM_L1JACOBI;
    if (l1) fl1_.alloc((size_t)nc_);
    if (o_.amg_smoother == NDS_SM_MCGS) {
      std::vector<int32_t> rows;
      greedy_color(nc_, F.row, F.col, rows, fine_coff_);
      fine_crows_.upload(rows);
    }
    for (auto* b : {&x_, &r_, &z_, &pp_, &q_, &rhs_}) b->alloc((size_t)nc_);
    tailpart_.alloc((size_t)std::max(grid_for(nc_), 1));
    ticket_.alloc(1);
    NDS_CUDA(cudaMemset(ticket_.p, 0, sizeof(unsigned)));
    for (auto* b : {&fr_, &ftmp_, &fcorr_, &frhs_, &fpong_}) b->alloc((size_t)nc_);
    if (!kSame) {
      rA_.alloc((size_t)nc_);
      zA_.alloc((size_t)nc_);
    }

    // AMG levels and transfers
    L_.resize(H.A.size());
    for (size_t l = 0; l < H.A.size(); ++l) {
      const CsrHost& A = H.A[l];
      Level& Lv = L_[l];
      Lv.n = A.n;
      Lv.row.upload(to_i32(A.row, "AMG level CSR"));
      Lv.col.upload(A.col);
      Lv.val.upload(A.val);
      Lv.diag.upload(A.diag);
      std::vector<double> l1h((size_t)A.n);
#pragma omp parallel for schedule(static)
      for (int i = 0; i < A.n; ++i) {
        double ss = 0.0;
        for (int64_t k = A.row[(size_t)i]; k < A.row[(size_t)i + 1]; ++k) ss += std::abs(A.val[(size_t)k]);
        l1h[(size_t)i] = ss;
      }
      Lv.l1.upload(l1h);
      for (auto* b : {&Lv.x, &Lv.r, &Lv.tmp, &Lv.corr, &Lv.pong}) b->alloc((size_t)A.n);
      Lv.b.alloc(dense_ld(A.n));  // the dense form reads up to the padding, which stays zero
      NDS_CUDA(cudaMemset(Lv.b.p, 0, Lv.b.bytes()));
      // the mixed path's V-cycle reads FP16 copies of the explicit levels
      // (the terminal level goes through its dense inverse)
      if (!kSame && o_.precision == NDS_MIXED && o_.amg_half && l + 1 < H.A.size()) level_to_half(Lv, A);
      if (l + 1 < H.A.size()) level_windows(Lv, A);
      if (o_.amg_smoother == NDS_SM_MCGS && l + 1 < H.A.size()) {
        std::vector<int32_t> rows;
        std::vector<int32_t> r32 = to_i32(A.row, "AMG level CSR");
        greedy_color(A.n, r32, A.col, rows, Lv.coff);
        Lv.crows.upload(rows);
      }
    }
    X_.resize(H.P.size());
    for (size_t l = 0; l < H.P.size(); ++l) {
      const Transfer& Ph = H.P[l];
      Xfer& X = X_[l];
      X.nf = Ph.nf;
      X.nc = Ph.nc;
      {
        // P in ELL, entry k of fine row i at k nf + i (coalesced across rows);
        // padding entries carry value 0 and coarse column 0
        int pw = 0;
        for (int i = 0; i < Ph.nf; ++i) pw = std::max<int>(pw, (int)(Ph.row[(size_t)i + 1] - Ph.row[(size_t)i]));
        std::vector<int32_t> ec((size_t)pw * Ph.nf, 0);
        std::vector<double> ev((size_t)pw * Ph.nf, 0.0);
#pragma omp parallel for schedule(static)
        for (int i = 0; i < Ph.nf; ++i)
          for (int64_t q = Ph.row[(size_t)i]; q < Ph.row[(size_t)i + 1]; ++q) {
            const size_t o = (size_t)(q - Ph.row[(size_t)i]) * Ph.nf + i;
            ec[o] = Ph.col[(size_t)q];
            ev[o] = Ph.val[(size_t)q];
          }
        X.pw = pw;
        X.pcol.upload(ec);
        X.pval.upload(ev);
      }
      // R = P^T, entries of each coarse row in ascending fine row
      std::vector<int32_t> rr((size_t)Ph.nc + 1, 0), rc(Ph.col.size());
      std::vector<double> rv(Ph.col.size());
      for (int32_t c : Ph.col) ++rr[(size_t)c + 1];
      for (int c = 0; c < Ph.nc; ++c) rr[(size_t)c + 1] += rr[(size_t)c];
      std::vector<int32_t> pos(rr.begin(), rr.end() - 1);
      for (int i = 0; i < Ph.nf; ++i)
        for (int64_t k = Ph.row[(size_t)i]; k < Ph.row[(size_t)i + 1]; ++k) {
          const int c = Ph.col[(size_t)k];
          rc[(size_t)pos[(size_t)c]] = i;
          rv[(size_t)pos[(size_t)c]++] = Ph.val[(size_t)k];
        }
      X.rrow.upload(rr);
      X.rcol.upload(rc);
      X.rval.upload(rv);
    }
    if (!L_.empty()) {  // rows padded for 16-byte loads
      const int n = L_.back().n;
      const size_t ld = dense_ld(n);
      std::vector<double> t(ld * (size_t)n, 0.0);
      for (int i = 0; i < n; ++i)
        std::copy_n(H.terminal_inv.begin() + (size_t)i * n, (size_t)n, t.begin() + (size_t)i * ld);
      tinv_.upload(t);
    }
    fine_lambda_ = H.fine_lambda;
    level_lambda_ = H.level_lambda;
    level_lambda_.resize(L_.size(), 0.0);

    part_.alloc((size_t)kMaxPartBlocks * 8);
    sc_.alloc(kScalars);
    flags_.alloc(1);
    ctl_.alloc(4);
    NDS_CUDA(cudaMallocHost((void**)&hsc_, sizeof(double) * kScalars));
    NDS_CUDA(cudaMallocHost((void**)&hflags_, sizeof(int) * 8));
    NDS_CUDA(cudaMemsetAsync(flags_.p, 0, sizeof(int), st_));

    if constexpr (!kSame) {
      mixed_ = o_.precision == NDS_MIXED;
      if (mixed_) alloc_mixed();
    }
    // setup-time state: fine CSR refreshed with the initial rAU
    tm.mark("levels_and_transfers");
    refresh_fine(rau_.p);
    if (mixed_ && o_.amg_half) {
      // FP16 copy: scale by a power of two that puts the largest setup-time
      // diagonal at 2^11 (the diagonal dominates its row; 2^4 headroom below
      // the FP16 maximum for later growth of rAU, values beyond saturate)
      std::vector<TA> d((size_t)nc_);
      NDS_CUDA(cudaMemcpyAsync(d.data(), fdiag_.p, sizeof(TA) * d.size(), cudaMemcpyDeviceToHost, st_));
      NDS_CUDA(cudaStreamSynchronize(st_));
      double dmax = 0.0;
      for (TA v : d) dmax = std::max(dmax, std::abs((double)v));
      if (!(dmax > 0.0) || !std::isfinite(dmax)) throw std::runtime_error("FP16 operator copy: no positive diagonal");
      hscale_ = std::ldexp(1.0, (int)std::floor(std::log2(2048.0 / dmax)));
      half_on_ = true;
      if (!split_) fvalH_.alloc(fval_.n);
      refresh_fine(rau_.p);
    }
    if (P_.power_its > 0) {
      fine_lambda_ = power_fine(P_.power_its, o_.amg_lambda_safety);
      for (size_t l = 0; l + 1 < L_.size(); ++l) level_lambda_[l] = power_level(L_[l], P_.power_its, o_.amg_lambda_safety);
    } else {
      fine_lambda_ = 1.0;
      for (auto& v : level_lambda_) v = 1.0;
    }
    build_dense_level();
    plan_resident();
    if (o_.pressure_solver == NDS_P_CHEB) p_cheb_lambda_ = precond_power(o_.p_power_its, o_.p_power_safety);
    NDS_CUDA(cudaStreamSynchronize(st_));
    tm.mark("refresh_and_spectrum");
    reset();
  }

  // assembled fine operator: refresh contributions and SELL layout
  void upload_sell(StageTimer& tm) {
    const Setup& S = P_.setup;
    const FineTopo& F = S.fine;
    // fine Schur refresh contributions, regrouped by destination slot in the
    // reference's order and laid out in runs (one run per fine entry, the
    // longest first) that never straddle a 32-contribution chunk of the row: a run that would
    // cross a chunk boundary starts the next chunk, the gap is filled with
    // pad entries.  Per contribution: the code word cs (basis a bits 0-2,
    // position in its run bits 3-5, run tail bit 6, slot bits 7-15; pads are
    // 0xFFFF) and the packed incidence (c2 << 3 | b) for the geometry.
    {
      std::vector<int32_t> plen((size_t)nc_ + 1, 0);
      std::vector<int32_t> poff((size_t)nc_ + 1, 0);
      OmpErr oerr;
      // pass 1: counts per slot and padded row lengths.  A row's runs are
      // laid out longest first (stable in slot order), so the few long runs
      // share a chunk and the chunks of short runs need few chain steps;
      // the order of the contributions inside a run is unchanged.
      std::vector<uint8_t> cnt(F.col.size(), 0);
      auto run_order = [&](int rb, int len, std::vector<int32_t>& ord) {
        ord.clear();
        for (int sl = 0; sl < len; ++sl)
          if (cnt[(size_t)rb + sl]) ord.push_back(sl);
        std::stable_sort(ord.begin(), ord.end(), [&](int32_t x, int32_t y) {
          return cnt[(size_t)rb + x] > cnt[(size_t)rb + y];
        });
      };
#pragma omp parallel
      {
        std::vector<int32_t> ord;
#pragma omp for schedule(dynamic, 1024)
        for (int c = 0; c < nc_; ++c) {
          oerr.run([&] {
            const int rb = F.row[(size_t)c], len = F.row[(size_t)c + 1] - rb;
            for (int q = F.contrib_off[(size_t)c]; q < F.contrib_off[(size_t)c + 1]; ++q) {
              // the code word holds a position in the run in three bits
              if (cnt[(size_t)rb + F.slot[(size_t)q]] == 8)
                throw std::runtime_error("more than 8 contributions to one fine entry");
              ++cnt[(size_t)rb + F.slot[(size_t)q]];
            }
            if (cnt[(size_t)F.diag_pos[(size_t)c]] == 0)
              throw std::runtime_error("fine Schur row without a diagonal contribution");
            run_order(rb, len, ord);
            int L = 0;
            for (const int32_t sl : ord) {
              const int n = cnt[(size_t)rb + sl];
              if ((L & 31) + n > 32) L = (L + 31) & ~31;
              L += n;
            }
            plen[(size_t)c + 1] = L;
          });
        }
      }
      oerr.rethrow();
      for (int c = 0; c < nc_; ++c) poff[(size_t)c + 1] = poff[(size_t)c] + plen[(size_t)c + 1];
      const size_t nq = (size_t)poff[(size_t)nc_];
      std::vector<uint16_t> cs(nq, 0xFFFF);
      std::vector<uint32_t> cpk(nq, 0);
      // pass 2: stable placement (the order of (a, incidence)) into the runs
#pragma omp parallel
      {
        std::vector<int32_t> start, fill, ord;
#pragma omp for schedule(dynamic, 1024)
        for (int c = 0; c < nc_; ++c) {
          const int rb = F.row[(size_t)c], len = F.row[(size_t)c + 1] - rb;
          start.assign((size_t)len, 0);
          fill.assign((size_t)len, 0);
          run_order(rb, len, ord);
          int L = 0;
          for (const int32_t sl : ord) {
            const int n = cnt[(size_t)rb + sl];
            if ((L & 31) + n > 32) L = (L + 31) & ~31;
            start[(size_t)sl] = L;
            L += n;
          }
          const size_t o = (size_t)poff[(size_t)c];
          int q = F.contrib_off[(size_t)c];
          for (int a = 0; a < 8; ++a) {
            const int g = S.ref[8 * (size_t)c + a];
            if (g < 0) continue;
            for (int k = F.inc_off[(size_t)g]; k < F.inc_off[(size_t)g + 1]; ++k, ++q) {
              const int sl = F.slot[(size_t)q], n = cnt[(size_t)rb + sl];
              const int pos = fill[(size_t)sl]++;
              const size_t at = o + (size_t)(start[(size_t)sl] + pos);
              cpk[at] = F.packed[(size_t)k];
              cs[at] = (uint16_t)(((unsigned)sl << 7) | ((pos == n - 1) ? 64u : 0u) | ((unsigned)pos << 3) | (unsigned)a);
            }
          }
        }
      }
      fcoff_.upload(poff);
      fcs_.upload(cs);
      DBuf<uint32_t> cpk_d;
      cpk_d.upload(cpk);
      fgeo_.alloc(nq);
      k::refresh_geometry<T><<<grid_for(nc_), kBlock, 0, st_>>>(nc_, fcoff_.p, cpk_d.p, fcs_.p, bco_.p, fgeo_.p);
      NDS_LAUNCH();
      NDS_CUDA(cudaStreamSynchronize(st_));
    }
    {
      tm.mark("refresh_contributions");
      // SELL-32x4 layout of the fine pattern (entry k of row 32 s + l at
      // base[s] + 128 (k/4) + 4 l + k%4, rows padded to a multiple of 4)
      const int ns = (nc_ + 31) / 32;
      std::vector<int32_t> width((size_t)ns, 0), base((size_t)ns + 1, 0), dslot((size_t)nc_);
      for (int c = 0; c < nc_; ++c) {
        const int len = F.row[(size_t)c + 1] - F.row[(size_t)c];
        width[(size_t)(c >> 5)] = std::max(width[(size_t)(c >> 5)], len);
        dslot[(size_t)c] = F.diag_pos[(size_t)c] - F.row[(size_t)c];
      }
      auto padded = [&](int q) { return (width[(size_t)q] + 3) & ~3; };
      auto offset = [&](int q, int l, int k) {
        return (size_t)base[(size_t)q] + 128 * (size_t)(k >> 2) + 4 * (size_t)l + (size_t)(k & 3);
      };
      for (int q = 0; q < ns; ++q) {
        const int64_t nb = (int64_t)base[(size_t)q] + 32LL * padded(q);
        if (nb > INT32_MAX) throw std::runtime_error("SELL fine operator exceeds int32 offsets");
        base[(size_t)q + 1] = (int32_t)nb;
      }
      // padding entries point at their own row; lanes past the last row of
      // the final slice point at row 0 (never read by a live thread)
      std::vector<int32_t> scol((size_t)base[(size_t)ns]);
#pragma omp parallel for schedule(static)
      for (int q = 0; q < ns; ++q)
        for (int l = 0; l < 32; ++l) {
          const int c = 32 * q + l;
          const int rb = c < nc_ ? F.row[(size_t)c] : 0, len = c < nc_ ? F.row[(size_t)c + 1] - rb : 0;
          for (int kk = 0; kk < padded(q); ++kk) scol[offset(q, l, kk)] = kk < len ? F.col[(size_t)rb + kk] : (c < nc_ ? c : 0);
        }
      swidth_.upload(width);
      int wmax = 0;
      for (int q = 0; q < ns; ++q) wmax = std::max(wmax, padded(q));
      refresh_smem_ = (size_t)33 * wmax * sizeof(T);
      if (refresh_smem_ > 200 * 1024) throw std::runtime_error("fine Schur row too long for the refresh slice buffer");
      NDS_CUDA(cudaFuncSetAttribute(k::sell_refresh<T, TA>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)refresh_smem_));
      sbase_.upload(base);
      fdslot_.upload(dslot);
      fval_.alloc(scol.size());
      NDS_CUDA(cudaMemset(fval_.p, 0, fval_.bytes()));
      if (!kSame) {
        fvalA_.alloc(scol.size());
        NDS_CUDA(cudaMemset(fvalA_.p, 0, fvalA_.bytes()));
      }
      // 16-bit column deltas when the ordering keeps every |column - row| < 2^15
      int too_far = 0;
      std::vector<int16_t> dcol(scol.size());
#pragma omp parallel for schedule(static) reduction(| : too_far)
      for (int q = 0; q < ns; ++q)
        for (int l = 0; l < 32; ++l) {
          const int row = 32 * q + l;
          for (int kk = 0; kk < padded(q); ++kk) {
            const size_t o = offset(q, l, kk);
            const int d = row < nc_ ? scol[o] - row : 0;
            if (d < -32767 || d > 32767) too_far = 1;
            else dcol[o] = (int16_t)d;
          }
        }
      const bool fits = too_far == 0;
      if (fits && !std::getenv("NDS_SELL_COL32")) {
        sdcol_.upload(dcol);
        sell_ = k::Sell{nc_, sbase_.p, swidth_.p, nullptr, sdcol_.p};
      } else {
        scol_.upload(scol);
        sell_ = k::Sell{nc_, sbase_.p, swidth_.p, scol_.p, nullptr};
      }
      sell_nnz_ = (long long)scol.size();
    }
  }
  // fine operator in split form (split.cuh): the free vertices' incidences,
  // the cells' vertices, face neighbours and gradients, in the precisions in
  // use; rAU-dependent parts are written by refresh_fine
  void upload_split() {
    const Setup& S = P_.setup;
    const FineTopo& F = S.fine;
    int nvert = 0;
    for (int v = 0; v < S.n_vert; ++v) nvert += S.g2free[(size_t)v] >= 0;
    svert_.n = nvert;
    const std::vector<int32_t> off(F.inc_off.begin(), F.inc_off.begin() + nvert + 1);
    const size_t nz = (size_t)off[(size_t)nvert];
    sp_off_.upload(off);
    svert_.off = sp_off_.p;
    const size_t n = (size_t)nc_;
    const bool half = !kSame && o_.precision == NDS_MIXED && o_.amg_half;
    auto vert = [&](int c, int a, int d) { return S.bco[24 * (size_t)c + 3 * (size_t)a + (size_t)d]; };
    std::vector<int4> vid(n), nid(n);
    std::vector<T> g4(4 * n);
    int too_far = 0;
#pragma omp parallel for schedule(static) reduction(| : too_far)
    for (int c = 0; c < nc_; ++c) {
      int v[4], nb[4];
      for (int a = 0; a < 4; ++a) {
        const int g = S.ref[8 * (size_t)c + (size_t)a], f = S.ref[8 * (size_t)c + 4 + (size_t)a];
        v[a] = g >= 0 ? g : nvert;
        nb[a] = -1;
        if (f >= 0)
          for (int k = F.inc_off[(size_t)f]; k < F.inc_off[(size_t)f + 1]; ++k) {
            const int q = (int)(F.packed[(size_t)k] >> 3);
            if (q != c) nb[a] = q;
          }
        if (nb[a] >= 0 && std::abs(nb[a] - c) > 32767) too_far = 1;
        double b2 = 0.0;
        for (int d = 0; d < 3; ++d) b2 += vert(c, a, d) * vert(c, a, d);
        g4[(size_t)a * n + (size_t)c] = (T)b2;
      }
      vid[(size_t)c] = make_int4(v[0], v[1], v[2], v[3]);
      nid[(size_t)c] = make_int4(nb[0], nb[1], nb[2], nb[3]);
    }
    sp_vid_.upload(vid);
    scell_.n = nc_;
    scell_.vid = sp_vid_.p;
    if (!too_far && !std::getenv("NDS_SELL_COL32")) {
      std::vector<short4> d16(n);
#pragma omp parallel for schedule(static)
      for (int c = 0; c < nc_; ++c) {
        const int4 q = nid[(size_t)c];
        auto d = [&](int j) { return (short)(j >= 0 ? j - c : 0); };
        d16[(size_t)c] = make_short4(d(q.x), d(q.y), d(q.z), d(q.w));
      }
      sp_nd16_.upload(d16);
      scell_.nd16 = sp_nd16_.p;
    } else {
      sp_nid_.upload(nid);
      scell_.nid = sp_nid_.p;
    }
    sp_g4_.upload(g4);
    // double: component arrays; float: 16-byte records (x, y, z, cell)
    auto records16 = [&](DBuf<float4>& out, auto&& value) {
      std::vector<float4> r(nz);
#pragma omp parallel for schedule(static)
      for (size_t z = 0; z < nz; ++z) {
        const uint32_t pa = F.packed[z];
        const int c = (int)(pa >> 3), a = (int)(pa & 7u);
        float cf;
        std::memcpy(&cf, &c, sizeof(cf));
        r[z] = make_float4(value(vert(c, a, 0)), value(vert(c, a, 1)), value(vert(c, a, 2)), cf);
      }
      out.upload(r);
    };
    auto geo_float = [&](DBuf<float4>& o4, DBuf<float>& o1) {
      std::vector<float4> q(2 * n);
      std::vector<float> l(n);
#pragma omp parallel for schedule(static)
      for (int c = 0; c < nc_; ++c) {
        float b[9];
        for (int k = 0; k < 9; ++k) b[k] = (float)vert(c, 1 + k / 3, k % 3);
        q[(size_t)c] = make_float4(b[0], b[1], b[2], b[3]);
        q[n + (size_t)c] = make_float4(b[4], b[5], b[6], b[7]);
        l[(size_t)c] = b[8];
      }
      o4.upload(q);
      o1.upload(l);
    };
    if constexpr (std::is_same<T, double>::value) {
      std::vector<double> b[3];
      std::vector<int32_t> cell(nz);
      for (auto& v : b) v.resize(nz);
#pragma omp parallel for schedule(static)
      for (size_t z = 0; z < nz; ++z) {
        const uint32_t pa = F.packed[z];
        const int c = (int)(pa >> 3), a = (int)(pa & 7u);
        cell[z] = c;
        for (int d = 0; d < 3; ++d) b[d][z] = vert(c, a, d);
      }
      for (int d = 0; d < 3; ++d) sp_b_[d].upload(b[d]);
      sp_cell_.upload(cell);
      svert_.bx = sp_b_[0].p;
      svert_.by = sp_b_[1].p;
      svert_.bz = sp_b_[2].p;
      svert_.cell = sp_cell_.p;
      std::vector<double2> q(4 * n);
      std::vector<double> l(n);
#pragma omp parallel for schedule(static)
      for (int c = 0; c < nc_; ++c) {
        for (int k = 0; k < 4; ++k)
          q[(size_t)k * n + (size_t)c] = make_double2(vert(c, 1 + 2 * k / 3, 2 * k % 3), vert(c, 1 + (2 * k + 1) / 3, (2 * k + 1) % 3));
        l[(size_t)c] = vert(c, 3, 2);
      }
      sp_gd2_.upload(q);
      sp_gd1_.upload(l);
    }
    if (std::is_same<TA, float>::value) {
      records16(sp_rec16_, [](double v) { return (float)v; });
      geo_float(sp_gf4_, sp_gf1_);
    }
    sp_rv_.alloc((size_t)std::max(nvert, 1));
    sp_tau_.alloc(4 * n);
    sp_w_.alloc(4 * (size_t)(nvert + 1));
    NDS_CUDA(cudaMemset(sp_w_.p, 0, sp_w_.bytes()));
    if (!kSame) {
      sp_rvA_.alloc((size_t)std::max(nvert, 1));
      sp_tauA_.alloc(4 * n);
      sp_wA_.alloc(4 * (size_t)(nvert + 1));
      NDS_CUDA(cudaMemset(sp_wA_.p, 0, sp_wA_.bytes()));
    }
    if (half) {
      // B of the free vertices scaled by the power of two that puts its largest
      // component at 2^14 .. 2^15 (the smallest normal half is 2^29 below).  A
      // fixed vertex's vector may be larger than a half holds; its w is zero,
      // so a cell keeps zero for it.
      double bmax = 0.0;
#pragma omp parallel for schedule(static) reduction(max : bmax)
      for (size_t z = 0; z < nz; ++z)
        for (int d = 0; d < 3; ++d) bmax = std::max(bmax, std::abs(vert((int)(F.packed[z] >> 3), (int)(F.packed[z] & 7u), d)));
      if (!std::isfinite(bmax)) throw std::runtime_error("FP16 operator copy: non-finite gradients");
      bscale_ = bmax > 0.0 ? std::ldexp(1.0, 14 - (int)std::floor(std::log2(bmax))) : 1.0;
      auto h = [&](double v) { return __float2half((float)(v * bscale_)); };
      auto bits = [](__half x) {
        unsigned short u;
        std::memcpy(&u, &x, sizeof(u));
        return (unsigned)u;
      };
      std::vector<int32_t> base((size_t)std::max(nvert, 1), 0);
      int wide = 0;
#pragma omp parallel for schedule(static) reduction(| : wide)
      for (int v = 0; v < nvert; ++v) {
        const int zb = off[(size_t)v], ze = off[(size_t)v + 1];
        if (zb == ze) continue;
        base[(size_t)v] = (int)(F.packed[(size_t)zb] >> 3);  // cells ascend
        if ((int)(F.packed[(size_t)ze - 1] >> 3) - base[(size_t)v] > 65535) wide = 1;
      }
      if (!wide && !std::getenv("NDS_SELL_COL32")) {
        std::vector<uint2> r(nz);
#pragma omp parallel for schedule(static)
        for (int v = 0; v < nvert; ++v)
          for (int z = off[(size_t)v]; z < off[(size_t)v + 1]; ++z) {
            const uint32_t pa = F.packed[(size_t)z];
            const int c = (int)(pa >> 3), a = (int)(pa & 7u);
            r[(size_t)z] = make_uint2(bits(h(vert(c, a, 0))) | bits(h(vert(c, a, 1))) << 16,
                                      bits(h(vert(c, a, 2))) | (unsigned)(c - base[(size_t)v]) << 16);
          }
        sp_rec8_.upload(r);
        sp_base_.upload(base);
      } else {
        records16(sp_rec16h_, [&](double v) { return __half2float(h(v)); });
      }
      std::vector<uint4> p(n);
      std::vector<uint2> q(n);
#pragma omp parallel for schedule(static)
      for (int c = 0; c < nc_; ++c) {
        unsigned w[6];
        auto value = [&](int q) {
          return S.ref[8 * (size_t)c + (size_t)(q / 3)] >= 0 ? bits(h(vert(c, q / 3, q % 3))) : 0u;
        };
        for (int k = 0; k < 6; ++k) w[k] = value(2 * k) | value(2 * k + 1) << 16;
        p[(size_t)c] = make_uint4(w[0], w[1], w[2], w[3]);
        q[(size_t)c] = make_uint2(w[4], w[5]);
      }
      sp_h4_.upload(p);
      sp_h2_.upload(q);
      sp_tauH_.alloc(4 * n);
    }
  }

  // ------------------------------------------------------------------ helpers
  static constexpr int kSms = 148;
  static constexpr int kMaxPartBlocks = 1184;  // 8 x 148 SMs
  static constexpr int kScalars = 128;
  enum { S_RHO = 0, S_PQ = 1, S_ALPHA = 2, S_RN2 = 3, S_RHON = 4, S_BETA = 5, S_R0 = 6, S_TARGET = 7, S_TMP = 8,
         S_TMP2 = 9, S_CONT2 = 10, S_WN = 11,
         S_AUDIT = 16, S_ST_T = 20, S_ST_V = 21,
         S_GUESS = 24 };  // 44 slots: Galerkin matrix (upper triangle) and right-hand side of the guess

  // CUDA graphs of fixed launch sequences (no host decisions inside)
  struct Graph {
    cudaGraphExec_t exec = nullptr;
    unsigned long long kernels = 0;
    ~Graph() {
      if (exec) cudaGraphExecDestroy(exec);
    }
  };
  template <class F>
  void capture(Graph& g, F&& body) {
    const bool was = prof.on;
    prof.on = false;
    const unsigned long long l0 = g_launches;
    NDS_CUDA(cudaStreamBeginCapture(st_, cudaStreamCaptureModeThreadLocal));
    try {
      body();
    } catch (...) {
      cudaGraph_t junk = nullptr;
      cudaStreamEndCapture(st_, &junk);
      if (junk) cudaGraphDestroy(junk);
      prof.on = was;
      throw;
    }
    cudaGraph_t graph = nullptr;
    NDS_CUDA(cudaStreamEndCapture(st_, &graph));
    const cudaError_t e = cudaGraphInstantiate(&g.exec, graph, 0);
    cudaGraphDestroy(graph);
    NDS_CUDA(e);
    g.kernels = g_launches - l0;
    g_launches = l0;
    prof.on = was;
  }
  void replay(Graph& g) {
    NDS_CUDA(cudaGraphLaunch(g.exec, st_));
    g_launches += g.kernels;
  }
  bool use_graphs_ = std::getenv("NDS_NO_GRAPHS") == nullptr;
  Graph g_amg_;
  // a whole Krylov loop as one graph: a conditional while node whose body is
  // one iteration; its last kernel sets the condition
  struct LoopGraph {
    cudaGraphExec_t exec = nullptr;
    unsigned long long body_kernels = 0;
    bool failed = false;
    ~LoopGraph() {
      if (exec) cudaGraphExecDestroy(exec);
    }
  };
  LoopGraph g_loop_;
  // z = M b with b, z in the state precision (casts around the V-cycle in
  // the mixed mode)
  void amg_T(const T* b, T* z) {
    if constexpr (kSame) {
      amg_apply(b, z);
    } else if (o_.amg_smoother != NDS_SM_MCGS) {
      // the cast also takes the fine pre-smoother's diagonal step
      const PolyPlan pl = fine_plan();
      pdl_launch(k::cast_jacobi<T, TA>, grid_for(nc_), kBlock, 0, st_, nc_, b, rA_.p, TA(pl.w0), pl.den0,
                 fine_first(zA_.p));
      NDS_LAUNCH();
      amg_apply(rA_.p, zA_.p, true);
      pdl_launch(k::cast_copy<TA, T>, grid_for(nc_), kBlock, 0, st_, nc_, zA_.p, z);
      NDS_LAUNCH();
    } else {
      pdl_launch(k::cast_copy<T, TA>, grid_for(nc_), kBlock, 0, st_, nc_, b, rA_.p);
      NDS_LAUNCH();
      amg_apply(rA_.p, zA_.p);
      pdl_launch(k::cast_copy<TA, T>, grid_for(nc_), kBlock, 0, st_, nc_, zA_.p, z);
      NDS_LAUNCH();
    }
  }
  // z = M r on the solver's fixed PCG buffers, replayed from a graph
  void amg_rz() {
    if (!use_graphs_) return amg_T(r_.p, z_.p);
    if (!g_amg_.exec) capture(g_amg_, [&] { amg_T(r_.p, z_.p); });
    replay(g_amg_);
  }

  int red_grid(long long n, int per = kBlock) const { return std::min(grid_for(n, per), kMaxPartBlocks); }
  template <int NV>
  void reduce_to(int nblocks, int slot) {
    pdl_launch(k::reduce_partials<NV>, 1, kBlock, 0, st_, part_.p, nblocks, sc_.p + slot);
    NDS_LAUNCH();
  }
  // a sum that the host needs: the reduction writes it to page-locked memory
  k::ReduceTail host_tail(int slot) {
    k::ReduceTail t = tail(slot);
    t.out = hsc_ + slot;
    return t;
  }
  template <class V>
  double dot_fetch(const V* x, const V* y, int n, int slot) {
    pdl_launch(k::dot_step<V, V, k::SUM_ONLY>, red_grid(n), kBlock, 0, st_, n, x, y, host_tail(slot));
    NDS_LAUNCH();
    NDS_CUDA(cudaStreamSynchronize(st_));
    return hsc_[slot];
  }
  // block partials in part summed straight into hsc_[slot ..]
  template <int NV>
  void reduce_host(const double* part, int nblocks, int slot) {
    pdl_launch(k::reduce_partials<NV>, 1, kBlock, 0, st_, part, nblocks, hsc_ + slot);
    NDS_LAUNCH();
    NDS_CUDA(cudaStreamSynchronize(st_));
  }
  k::HostWords host_words() const { return k::HostWords{hsc_ + S_RN2, hflags_}; }
  k::SolveInit solve_init(double target, double r0, int first, int cap) const {
    return k::SolveInit{sc_.p, ctl_.p, flags_.p, S_R0, S_TARGET, first, cap, r0, target};
  }
  template <class V>
  void dot_dev(const V* x, const V* y, int n, int slot) {
    const int g = red_grid(n);
    pdl_launch(k::dot<V>, g, kBlock, 0, st_, n, x, y, part_.p);
    NDS_LAUNCH();
    reduce_to<1>(g, slot);
  }

  // operator view: the fine Schur matrix in SELL-32, AMG levels in CSR
  template <class V>
  struct OpView {
    int n;
    bool sell;
    k::Sell s;
    const int32_t* rp;
    const int32_t* ci;
    const V* v;
    int cat;                     // profiler category
    const __half* vh = nullptr;  // FP16 copy of the values, scaled by 1 / vinv
    double vinv = 1.0;
    const int16_t* ch = nullptr;  // CSR levels with vh: columns as deltas to the row
    const int2* win = nullptr;    // CSR levels: windows of x (level_window)
    int wrows = 0, wblocks = 0;
    size_t wsmem = 0;
    const int16_t* dc = nullptr;  // with win: columns as deltas to the row
    // fine operator in split form (sell is set too)
    bool split = false, half = false;
    k::SplitVerts sv{};
    k::SplitCells sc{};
    const V* rv = nullptr;
    V* w = nullptr;
    double wscale = 1.0, tinv = 1.0;
  };
  // the two steps of a product in split form
  template <int MODE, class V>
  void split_launch(const OpView<V>& A, const V* x, const V* b, const V* den, double w, V* y, V* y2) {
    static_assert(MODE != k::SELL_DOT, "split_dot forms p.q");
    split_vertices(A, x);
    split_types(A, [&](auto mt, auto d16) {
      pdl_launch(k::split_cell<V, MODE, decltype(d16)::value, decltype(mt)>, grid_for(A.n), kBlock, 0, st_, A.sc,
                 A.w, x, b, den, V(w), y, y2, V(A.tinv),
                 (const V*)nullptr, k::ReduceTail{}, (const int*)nullptr);
    });
  }
  template <class V>
  void split_vertices(const OpView<V>& A, const V* x) {
    if (A.sv.n <= 0) return;
    auto go = [&](auto rec) {
      constexpr int REC = decltype(rec)::value;
      const int gv = std::min(grid_for(8LL * A.sv.n), kSms * k::split_vertex_blocks<REC>());
      pdl_launch(k::split_vertex<V, REC>, gv, kBlock, 0, st_, A.sv, A.rv, x, A.w, V(A.wscale));
    };
    if constexpr (std::is_same<V, double>::value) go(std::integral_constant<int, k::REC_SOA>{});
    else if (A.sv.rec8) go(std::integral_constant<int, k::REC_8>{});
    else go(std::integral_constant<int, k::REC_16>{});
    NDS_LAUNCH();
  }
  // f(value type of the cells' data, 16-bit neighbour deltas)
  template <class V, class F>
  void split_types(const OpView<V>& A, F&& f) {
    auto width = [&](auto mt) {
      if (A.sc.nd16) f(mt, std::true_type{});
      else f(mt, std::false_type{});
    };
    if constexpr (std::is_same<V, float>::value) {
      if (A.half) {
        width(__half{});
        return;
      }
    }
    width(V{});
  }
  // the last smoothing step of the V-cycle, z = x + w (b - A x) / den or
  // (add_to given) add_to += that, with r.z and the step rho of PCG
  template <class V, class R>
  void split_smooth_rho(const OpView<V>& A, const V* x, const V* b, const V* den, double w, V* z, V* add_to,
                        const R* r) {
    ProfScope ps(prof, st_, A.cat);
    split_vertices(A, x);
    split_types(A, [&](auto mt, auto d16) {
      pdl_launch(k::split_cell<V, k::SELL_SMOOTH, decltype(d16)::value, decltype(mt), k::PCG_RHO, R>, grid_for(A.n),
                 kBlock, 0, st_, A.sc, A.w, x, b, den, V(w), z, add_to, V(A.tinv), r, tail(S_RHON),
                 (const int*)nullptr);
    });
    NDS_LAUNCH();
  }
  // q = A p with p.q and the step alpha of PCG
  template <class V>
  void split_dot(const OpView<V>& A, const V* p, V* q) {
    ProfScope ps(prof, st_, A.cat);
    split_vertices(A, p);
    if (A.sc.nd16)
      pdl_launch(k::split_cell_dot<V, true>, red_grid(A.n), kBlock, 0, st_, A.sc, A.w, p, q, V(A.tinv), tail(S_PQ));
    else
      pdl_launch(k::split_cell_dot<V, false>, red_grid(A.n), kBlock, 0, st_, A.sc, A.w, p, q, V(A.tinv), tail(S_PQ));
    NDS_LAUNCH();
  }
  // a reduction into sc[slot] taken by the producing kernel's last block
  k::ReduceTail tail(int slot, cudaGraphConditionalHandle h = {}) {
    return k::ReduceTail{tailpart_.p, ticket_.p, sc_.p + slot,
                         k::PcgScalars{sc_.p, flags_.p, ctl_.p, S_RN2, S_R0, S_TARGET, h, in_graph_, host_words()}};
  }
  template <int MODE, class V>
  void sell_launch(const OpView<V>& A, int grid, const V* x, const V* b, const V* den, double w, V* y, V* y2) {
    if constexpr (MODE != k::SELL_DOT) {
      if (A.split) {
        split_launch<MODE, V>(A, x, b, den, w, y, y2);
        return;
      }
    }
    if constexpr (std::is_same<V, float>::value) {
      if (A.vh) {
        if (A.s.dcol)
          pdl_launch(k::sell_spmv<V, MODE, true, __half>, grid, kBlock, 0, st_, A.s, A.vh, x, b, den, V(w), y, y2,
                     part_.p, V(A.vinv));
        else
          pdl_launch(k::sell_spmv<V, MODE, false, __half>, grid, kBlock, 0, st_, A.s, A.vh, x, b, den, V(w), y, y2,
                     part_.p, V(A.vinv));
        return;
      }
    }
    if (A.s.dcol)
      pdl_launch(k::sell_spmv<V, MODE, true>, grid, kBlock, 0, st_, A.s, A.v, x, b, den, V(w), y, y2, part_.p, V(1));
    else
      pdl_launch(k::sell_spmv<V, MODE, false>, grid, kBlock, 0, st_, A.s, A.v, x, b, den, V(w), y, y2, part_.p, V(1));
  }
  // physical operator (precision T) and the AMG's fine operator (precision TA)
  OpView<T> fine_op() {
    OpView<T> A{nc_, true, sell_, nullptr, nullptr, fval_.p, P_FINE_SPMV};
    if (split_) set_split(A, sp_rv_.p, sp_w_.p, sp_tau_.p);
    return A;
  }
  // the split form in the precision of V (FP64 or FP32 data)
  template <class V>
  void set_split(OpView<V>& A, const V* rv, V* w, const V* tau) {
    A.split = true;
    A.sv = svert_;
    A.sc = scell_;
    A.rv = rv;
    A.w = w;
    A.sc.tau = tau;
    if constexpr (std::is_same<V, double>::value) {
      A.sc.g0 = sp_gd2_.p;
      A.sc.g2 = sp_gd1_.p;
    } else {
      A.sv.rec16 = sp_rec16_.p;
      A.sc.g0 = sp_gf4_.p;
      A.sc.g1 = sp_gf4_.p + nc_;
      A.sc.g2 = sp_gf1_.p;
    }
  }
  OpView<TA> fine_opA() {
    if (split_) {
      if constexpr (kSame) {
        OpView<TA> A = fine_op();
        A.cat = P_FINE_AMG;
        return A;
      } else {
        OpView<TA> A{nc_, true, sell_, nullptr, nullptr, nullptr, P_FINE_AMG};
        set_split(A, (const TA*)sp_rvA_.p, sp_wA_.p, (const TA*)sp_tauA_.p);
        return A;
      }
    }
    if constexpr (kSame) return {nc_, true, sell_, nullptr, nullptr, fval_.p, P_FINE_AMG};
    else return {nc_, true, sell_, nullptr, nullptr, fvalA_.p, P_FINE_AMG};
  }
  // the fine operator of the V-cycle: the FP16 copy when amg_half is on
  OpView<TA> fine_opV() {
    OpView<TA> A = fine_opA();
    if (split_ && half_on_) {
      A.half = true;
      A.sv.rec16 = sp_rec16h_.p;
      A.sv.rec8 = sp_rec8_.p;
      A.sv.base = sp_base_.p;
      A.sc.g0 = sp_h4_.p;
      A.sc.g1 = sp_h2_.p;
      A.sc.tau = sp_tauH_.p;
      A.wscale = 1.0 / (bscale_ * bscale_);
      A.tinv = 1.0 / hscale_;
      A.cat = P_FINE_HALF;
    } else if (fvalH_.p) {
      A.vh = fvalH_.p;
      A.vinv = 1.0 / hscale_;
      A.cat = P_FINE_HALF;
    }
    return A;
  }
  OpView<TA> level_op(const Level& A) const {
    OpView<TA> V{A.n, false, k::Sell{}, A.row.p, A.col.p, A.val.p, P_COARSE_SPMV};
    if (A.hval.p) {
      V.vh = A.hval.p;
      V.vinv = A.hinv;
      V.ch = A.hcol.p;
    }
    V.win = A.win.p;
    V.wrows = A.wrows;
    V.wblocks = A.wblocks;
    V.wsmem = A.wsmem;
    V.dc = A.dcol.p;
    return V;
  }
  // windows of a level's rows (FP64 levels): from kWinRows rows on, when a
  // window fits the block's share of shared memory.  The line: with fewer rows
  // than about two per lane group of the 296 blocks there is no next row to
  // look ahead to.  Microseconds of a PCG iteration, a lane group a row / this:
  // 12,419 rows 130.9 / 128.7, 17,736 rows 165.4 / 155.2, 23,192 rows 218.7 /
  // 204.7, 74,540 rows 612 / 557 (a product there 25 / 20 us on average).
  static constexpr int kWinRows = 16384;
  static constexpr size_t kWinBytes = 72 * 1024;
  void level_windows(Level& Lv, const CsrHost& A) {
    if (A.n < stream_rows(kWinRows) || !std::is_same<TA, double>::value) return;
    int sms = 0;
    NDS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, o_.device));
    const int blocks = sms * k::kWinPerSm, rows = (A.n + blocks - 1) / blocks;
    std::vector<int2> win((size_t)blocks, make_int2(0, 0));
    int most = 0;
#pragma omp parallel for schedule(static) reduction(max : most)
    for (int q = 0; q < blocks; ++q) {
      const int r0 = std::min(A.n, q * rows), r1 = std::min(A.n, r0 + rows);
      int lo = A.n, hi = 0;
      for (int i = r0; i < r1; ++i) {
        lo = std::min(lo, i);
        hi = std::max(hi, i + 1);
        for (int64_t k = A.row[(size_t)i]; k < A.row[(size_t)i + 1]; ++k) {
          lo = std::min(lo, (int)A.col[(size_t)k]);
          hi = std::max(hi, (int)A.col[(size_t)k] + 1);
        }
      }
      if (lo < hi) win[(size_t)q] = make_int2(lo, hi);
      most = std::max(most, hi - lo + 4);  // staged from a 16-byte boundary
    }
    if ((size_t)most * sizeof(double) > kWinBytes) return;
    std::vector<int16_t> dc(A.col.size());
    int too_far = 0;
#pragma omp parallel for schedule(static) reduction(| : too_far)
    for (int i = 0; i < A.n; ++i)
      for (int64_t k = A.row[(size_t)i]; k < A.row[(size_t)i + 1]; ++k) {
        const int d = A.col[(size_t)k] - i;
        if (d < -32767 || d > 32767) too_far = 1;
        else dc[(size_t)k] = (int16_t)d;
      }
    if (!too_far && !std::getenv("NDS_SELL_COL32")) Lv.dcol.upload(dc);
    Lv.win.upload(win);
    Lv.wrows = rows;
    Lv.wblocks = blocks;
    Lv.wsmem = (size_t)most * sizeof(double);
  }
  // a product of a level with windows; false when it has none
  template <int MODE, class V>
  bool window_launch(const OpView<V>& A, const V* x, const V* b, const V* den, double w, V* y, V* y2) {
    if (!A.win) return false;
    if constexpr (std::is_same<V, double>::value) {
      auto go = [&](auto* ci) {
        using CT = std::remove_const_t<std::remove_pointer_t<decltype(ci)>>;
        auto* kernel = k::level_window<MODE, CT>;
        NDS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWinBytes));
        pdl_launch(kernel, A.wblocks, k::kWinBlock, A.wsmem, st_, A.n, A.wrows, A.win, A.rp, ci, A.v, x, b, den, w, y,
                   y2);
      };
      if (A.dc) go(A.dc);
      else go(A.ci);
      return true;
    }
    return false;
  }
  // FP16 copy of an explicit level's CSR values (a setup snapshot), scaled by
  // the power of two that puts its largest diagonal at 2^11
  void level_to_half(Level& Lv, const CsrHost& A) {
    double dmax = 0.0;
    for (double d : A.diag) dmax = std::max(dmax, std::abs(d));
    if (!(dmax > 0.0) || !std::isfinite(dmax)) throw std::runtime_error("FP16 level copy: no positive diagonal");
    const double scale = std::ldexp(1.0, (int)std::floor(std::log2(2048.0 / dmax)));
    std::vector<__half> hv(A.val.size());
#pragma omp parallel for schedule(static)
    for (size_t k = 0; k < hv.size(); ++k)
      hv[k] = __float2half((float)std::min(std::max(A.val[k] * scale, -65504.0), 65504.0));
    Lv.hval.alloc(hv.size());
    NDS_CUDA(cudaMemcpy(Lv.hval.p, hv.data(), hv.size() * sizeof(__half), cudaMemcpyHostToDevice));
    Lv.hinv = 1.0 / scale;
    std::vector<int16_t> dc(A.col.size());
    int too_far = 0;
#pragma omp parallel for schedule(static) reduction(| : too_far)
    for (int i = 0; i < A.n; ++i)
      for (int64_t k = A.row[(size_t)i]; k < A.row[(size_t)i + 1]; ++k) {
        const int d = A.col[(size_t)k] - i;
        if (d < -32767 || d > 32767) too_far = 1;
        else dc[(size_t)k] = (int16_t)d;
      }
    const bool fits = too_far == 0;
    if (fits && !std::getenv("NDS_SELL_COL32")) Lv.hcol.upload(dc);
  }
  // launch f with the lanes per row of the FP16 level kernels
  template <class V, class F>
  void level_half_launch(const OpView<V>& A, F&& f) {
    if (level_lanes_ == 8) f(std::integral_constant<int, 8>{});
    else if (level_lanes_ == 16) f(std::integral_constant<int, 16>{});
    else f(std::integral_constant<int, 32>{});
  }
  template <class V>
  void op_spmv(const OpView<V>& A, const V* x, V* y) {
    ProfScope ps(prof, st_, A.cat);
    if (A.sell) sell_launch<k::SELL_Y, V>(A, grid_for(A.n), x, nullptr, nullptr, 0.0, y, nullptr);
    else if (window_launch<k::LEV_Y, V>(A, x, nullptr, nullptr, 0.0, y, nullptr)) {
    } else if (A.vh && A.ch && std::is_same<V, float>::value)
      level_half_launch(A, [&](auto gl) {
        constexpr int GL = decltype(gl)::value;
        pdl_launch(k::spmv<V, __half, int16_t, GL>, grid_for((long long)A.n * GL), kBlock, 0, st_, A.n, A.rp, A.ch,
                   A.vh, x, y, V(A.vinv));
      });
    else if (A.vh && std::is_same<V, float>::value)
      level_half_launch(A, [&](auto gl) {
        constexpr int GL = decltype(gl)::value;
        pdl_launch(k::spmv<V, __half, int32_t, GL>, grid_for((long long)A.n * GL), kBlock, 0, st_, A.n, A.rp, A.ci,
                   A.vh, x, y, V(A.vinv));
      });
    else pdl_launch(k::spmv<V>, grid_for((long long)A.n * k::kRowLanes), kBlock, 0, st_, A.n, A.rp, A.ci, A.v, x, y,
                    V(1));
    NDS_LAUNCH();
  }
  // r = b - A x; r2 = r, or (den given) the first Jacobi step w r / den
  template <class V>
  void op_resid(const OpView<V>& A, const V* x, const V* b, V* r, V* r2 = nullptr, const V* den = nullptr,
                double w = 0.0) {
    ProfScope ps(prof, st_, A.cat);
    if (A.sell) sell_launch<k::SELL_RESID, V>(A, grid_for(A.n), x, b, den, w, r, r2);
    else if (window_launch<k::LEV_RESID, V>(A, x, b, den, w, r, r2)) {
    } else if (A.vh && A.ch && std::is_same<V, float>::value)
      level_half_launch(A, [&](auto gl) {
        constexpr int GL = decltype(gl)::value;
        pdl_launch(k::spmv_resid<V, __half, int16_t, GL>, grid_for((long long)A.n * GL), kBlock, 0, st_, A.n, A.rp,
                   A.ch, A.vh, x, b, r, r2, den, V(w), V(A.vinv));
      });
    else if (A.vh && std::is_same<V, float>::value)
      level_half_launch(A, [&](auto gl) {
        constexpr int GL = decltype(gl)::value;
        pdl_launch(k::spmv_resid<V, __half, int32_t, GL>, grid_for((long long)A.n * GL), kBlock, 0, st_, A.n, A.rp,
                   A.ci, A.vh, x, b, r, r2, den, V(w), V(A.vinv));
      });
    else
      pdl_launch(k::spmv_resid<V>, grid_for((long long)A.n * k::kRowLanes), kBlock, 0, st_, A.n, A.rp, A.ci, A.v, x,
                 b, r, r2, den, V(w), V(1));
    NDS_LAUNCH();
  }
  // xout = xin + w (b - A xin) / den, or (add_to given) add_to += that
  template <class V>
  void op_smooth(const OpView<V>& A, const V* xin, const V* b, const V* den, double w, V* xout, V* add_to = nullptr) {
    ProfScope ps(prof, st_, A.cat);
    if (A.sell) sell_launch<k::SELL_SMOOTH, V>(A, grid_for(A.n), xin, b, den, w, xout, add_to);
    else if (window_launch<k::LEV_SMOOTH, V>(A, xin, b, den, w, xout, add_to)) {
    } else if (A.vh && A.ch && std::is_same<V, float>::value)
      level_half_launch(A, [&](auto gl) {
        constexpr int GL = decltype(gl)::value;
        pdl_launch(k::spmv_smooth<V, __half, int16_t, GL>, grid_for((long long)A.n * GL), kBlock, 0, st_, A.n, A.rp,
                   A.ch, A.vh, xin, b, den, V(w), xout, add_to, V(A.vinv));
      });
    else if (A.vh && std::is_same<V, float>::value)
      level_half_launch(A, [&](auto gl) {
        constexpr int GL = decltype(gl)::value;
        pdl_launch(k::spmv_smooth<V, __half, int32_t, GL>, grid_for((long long)A.n * GL), kBlock, 0, st_, A.n, A.rp,
                   A.ci, A.vh, xin, b, den, V(w), xout, add_to, V(A.vinv));
      });
    else
      pdl_launch(k::spmv_smooth<V>, grid_for((long long)A.n * k::kRowLanes), kBlock, 0, st_, A.n, A.rp, A.ci, A.v,
                 xin, b, den, V(w), xout, add_to, V(1));
    NDS_LAUNCH();
  }
  template <class V>
  void vcopy(int n, const V* a, V* b) {
    k::copy<V><<<grid_for(n), kBlock, 0, st_>>>(n, a, b);
    NDS_LAUNCH();
  }
  template <class V>
  void vaxpy(int n, double a, const V* x, V* y) {
    pdl_launch(k::axpy<V>, grid_for(n), kBlock, 0, st_, n, V(a), x, y);
    NDS_LAUNCH();
  }

  // fine Schur operator
  void refresh_fine(const T* rau, cudaStream_t s = nullptr) {
    if (!s) s = st_;
    ProfScope ps(prof, s, P_REFRESH);
    if (split_) {
      k::split_refresh<T, TA><<<grid_for(std::max(nc_, svert_.n)), kBlock, 0, s>>>(
          nc_, svert_.n, ref_.p, sp_g4_.p, rau, sp_rv_.p, kSame ? nullptr : sp_rvA_.p, sp_tau_.p,
          kSame ? nullptr : sp_tauA_.p, half_on_ ? sp_tauH_.p : nullptr, (float)hscale_, fdiag_.p);
      NDS_LAUNCH();
      return;
    }
    k::sell_refresh<T, TA><<<(nc_ + 31) / 32, k::kRefreshBlock, refresh_smem_, s>>>(
        nc_, fcoff_.p, fcs_.p, fgeo_.p, ref_.p, rau, fdslot_.p, sbase_.p, swidth_.p, fval_.p,
        kSame ? nullptr : fvalA_.p, fdiag_.p, fl1_.p, fvalH_.p, (float)hscale_);
    NDS_LAUNCH();
  }
  void fine_apply(const T* x, T* y) { op_spmv(fine_op(), x, y); }

  // ------------------------------------------------------------- smoothers
  // x = S(b) from a zero initial guess.  Jacobi-type steps write to a second
  // buffer (xin is read by every row), then the result is copied back.
  // Polynomial (Chebyshev or damped-Jacobi) smoother from a zero guess:
  // x = S(b).  One diagonal step, then m Jacobi-type steps ping-ponging
  // between two buffers; the first buffer is chosen by the parity of m so
  // that the last step writes x (no copy-back).
  struct PolyPlan {
    int m;            // Jacobi-type steps after the diagonal one
    double w0;        // weight of the diagonal step
    const TA* den0;   // its denominator
  };
  PolyPlan poly_plan(double lambda, bool cheb, const TA* diag, const TA* den_jac, int sweeps) const {
    if (cheb) {
      const int deg = o_.amg_cheb_degree;
      const double lo = o_.amg_lambda_low_fraction * lambda;
      if (!(lambda > lo && lo > 0)) throw SolveFailure(NDS_E_BREAKDOWN, "Chebyshev smoother interval invalid");
      return {deg - 1, 1.0 / cheb_root(lambda, lo, 0, deg), diag};
    }
    return {sweeps - 1, o_.amg_jacobi_omega, den_jac};
  }
  static TA* poly_first(const PolyPlan& pl, TA* x, TA* pong) { return (pl.m % 2 == 0) ? x : pong; }
  // first_done: the diagonal step is already in poly_first(x, pong) (written
  // by the residual kernel); add_to: the result is added to add_to instead
  // of stored in x.
  void poly_smooth(const OpView<TA>& A, const TA* diag, const TA* b, TA* x, TA* pong, double lambda, bool cheb,
                   const TA* den_jac, int sweeps, bool first_done = false, TA* add_to = nullptr) {
    const int n = A.n;
    const PolyPlan pl = poly_plan(lambda, cheb, diag, den_jac, sweeps);
    TA* cur = poly_first(pl, x, pong);
    TA* nxt = (pl.m % 2 == 0) ? pong : x;
    if (!first_done) {
      pdl_launch(k::jacobi_zero<TA>, grid_for(n), kBlock, 0, st_, n, TA(pl.w0), b, pl.den0, cur);
      NDS_LAUNCH();
    }
    const double lo = cheb ? o_.amg_lambda_low_fraction * lambda : 0.0;
    for (int kk = 1; kk <= pl.m; ++kk) {
      const double w = cheb ? 1.0 / cheb_root(lambda, lo, kk, o_.amg_cheb_degree) : o_.amg_jacobi_omega;
      op_smooth(A, cur, b, cheb ? diag : den_jac, w, nxt, kk == pl.m ? add_to : nullptr);
      std::swap(cur, nxt);
    }
    if (pl.m == 0 && add_to) vaxpy(n, 1.0, (const TA*)x, add_to);
  }
  void mcgs(const OpView<TA>& A, const TA* diag, const TA* b, TA* x, const DBuf<int32_t>& crows,
            const std::vector<int>& coff, int sweeps) {
    const int n = A.n;
    NDS_CUDA(cudaMemsetAsync(x, 0, sizeof(TA) * (size_t)n, st_));
    const int ncol = (int)coff.size() - 1;
    auto pass = [&](bool reverse) {
      for (int qq = 0; qq < ncol; ++qq) {
        const int c = reverse ? ncol - 1 - qq : qq;
        const int cnt = coff[(size_t)c + 1] - coff[(size_t)c];
        if (cnt <= 0) continue;
        if (A.sell && A.s.dcol)
          k::sell_gs_color<TA, true><<<grid_for(cnt), kBlock, 0, st_>>>(cnt, crows.p + coff[(size_t)c], A.s, A.v, diag, b,
                                                                     x, TA(o_.amg_mcgs_omega));
        else if (A.sell)
          k::sell_gs_color<TA, false><<<grid_for(cnt), kBlock, 0, st_>>>(cnt, crows.p + coff[(size_t)c], A.s, A.v, diag,
                                                                      b, x, TA(o_.amg_mcgs_omega));
        else
          k::amg_gs_color<TA><<<grid_for((long long)cnt * 32), kBlock, 0, st_>>>(cnt, crows.p + coff[(size_t)c], A.rp, A.ci,
                                                                                A.v, diag, b, x, TA(o_.amg_mcgs_omega));
        NDS_LAUNCH();
      }
    };
    for (int s = 0; s < sweeps; ++s) {
      if (o_.amg_mcgs_order == NDS_MCGS_FORWARD) pass(false);
      else if (o_.amg_mcgs_order == NDS_MCGS_BACKWARD) pass(true);
      else { pass(false); pass(true); }
    }
  }
  // first_done: the diagonal step of the polynomial smoother is already in
  // place (taken by the kernel that produced b); never set for MCGS
  void smooth_fine(const TA* b, TA* x, bool first_done = false) {
    const int sm = o_.amg_smoother;
    if (sm == NDS_SM_MCGS) {
      mcgs(fine_opV(), fdiag_.p, b, x, fine_crows_, fine_coff_, o_.amg_mcgs_fine_sweeps);
      return;
    }
    const TA* den = sm == NDS_SM_L1JACOBI ? fl1_.p : fdiag_.p;
    poly_smooth(fine_opV(), fdiag_.p, b, x, fpong_.p, fine_lambda_, sm == NDS_SM_CHEB2, den, o_.amg_jacobi_fine_sweeps,
                first_done);
  }
  void smooth_level(Level& A, const TA* b, TA* x, double lambda, bool first_done = false) {
    const int sm = o_.amg_smoother;
    if (sm == NDS_SM_MCGS) {
      mcgs(level_op(A), A.diag.p, b, x, A.crows, A.coff, o_.amg_mcgs_coarse_sweeps);
      return;
    }
    const TA* den = sm == NDS_SM_L1JACOBI ? A.l1.p : A.diag.p;
    poly_smooth(level_op(A), A.diag.p, b, x, A.pong.p, lambda, sm == NDS_SM_CHEB2, den, o_.amg_jacobi_coarse_sweeps,
                first_done);
  }
  // plan of the pre-smoother of level l (polynomial smoothers only)
  PolyPlan level_plan(int l) const {
    const Level& A = L_[(size_t)l];
    const int sm = o_.amg_smoother;
    const TA* den = sm == NDS_SM_L1JACOBI ? A.l1.p : A.diag.p;
    return poly_plan(level_lambda_[(size_t)l], sm == NDS_SM_CHEB2, A.diag.p, den, o_.amg_jacobi_coarse_sweeps);
  }
  PolyPlan fine_plan() const {
    const int sm = o_.amg_smoother;
    const TA* den = sm == NDS_SM_L1JACOBI ? fl1_.p : fdiag_.p;
    return poly_plan(fine_lambda_, sm == NDS_SM_CHEB2, fdiag_.p, den, o_.amg_jacobi_fine_sweeps);
  }
  // whether the pre-smoother of level l can take its diagonal step in the
  // restriction that feeds it (a polynomial smoother, not the terminal level)
  bool fuse_pre(int l) const { return o_.amg_smoother != NDS_SM_MCGS && l < (int)L_.size() - 1 && l != dense_level_; }
  // coarse rows from which the restriction streams: more than a wave of warps, so
  // that there is a next row to load ahead (fewer rows: a lane group a row).
  // Microseconds of a PCG iteration, a lane group a row / streaming: 6,411 rows
  // FP64 81.4 / 80.0, FP32 72.9 / 70.7; 12,419 rows 132.5 / 130.6, 102.9 / 101.7;
  // 74,540 rows 569 / 556, 406 / 398.
  static constexpr int kStreamRows = 8192;
  // NDS_STREAM_ROWS overrides the row counts from which the streaming kernels
  // of the levels and the restriction are used
  static int stream_rows(int rows) {
    const char* e = std::getenv("NDS_STREAM_ROWS");
    return e ? std::atoi(e) : rows;
  }
  int rest_rows_ = stream_rows(kStreamRows);
  // lanes per coarse row of the restriction (the FP16 levels' count on the
  // mixed FP16 path, a warp otherwise)
  int restrict_lanes() const { return mixed_ && o_.amg_half ? level_lanes_ : 32; }
  // c = R f; with level >= 0 also the diagonal step of that level's
  // pre-smoother (see fuse_pre)
  void restrict_to(const Xfer& X, const TA* f, TA* c, int level = -1) {
    ProfScope ps(prof, st_, P_TRANSFER);
    const TA* den0 = nullptr;
    TA* x1 = nullptr;
    double w0 = 0.0;
    if (level >= 0) {
      Level& C = L_[(size_t)level];
      const PolyPlan pl = level_plan(level);
      den0 = pl.den0;
      w0 = pl.w0;
      x1 = poly_first(pl, C.x.p, C.pong.p);
    }
    if (X.nc >= rest_rows_) {
      const int g = std::min(grid_for(X.nc, kBlock / 32), kSms * k::rest_blocks<TA>());
      pdl_launch(k::restrict_stream<TA>, g, kBlock, 0, st_, X.nc, X.rrow.p, X.rcol.p, X.rval.p, f, c, den0, TA(w0), x1);
    } else if (restrict_lanes() != 32) {
      auto run = [&](auto gl) {
        constexpr int GL = decltype(gl)::value;
        pdl_launch(k::restrict_rows<TA, GL>, grid_for((long long)X.nc * GL), kBlock, 0, st_, X.nc, X.rrow.p,
                   X.rcol.p, X.rval.p, f, c, den0, TA(w0), x1);
      };
      if (restrict_lanes() == 8) run(std::integral_constant<int, 8>{});
      else run(std::integral_constant<int, 16>{});
    } else {
      pdl_launch(k::restrict_rows<TA>, grid_for((long long)X.nc * k::kRowLanes), kBlock, 0, st_, X.nc, X.rrow.p,
                 X.rcol.p, X.rval.p, f, c, den0, TA(w0), x1);
    }
    NDS_LAUNCH();
  }
  void prolong(const Xfer& X, const TA* c, TA* f) {
    ProfScope ps(prof, st_, P_TRANSFER);
    pdl_launch(k::prolong_add<TA>, grid_for(X.nf), kBlock, 0, st_, X.nf, X.pw, X.pcol.p, X.pval.p, c, f);
    NDS_LAUNCH();
  }

  // ------------------------------------------- dense form of coarse levels
  // The first level whose V-cycle matrix takes at most kDenseBytes is applied
  // as that matrix (polynomial smoothers; not the terminal level, which is
  // dense already).  One product replaces the level's four SpMVs and all
  // launches below it.  Microseconds of a PCG iteration, level by level /
  // dense: 278 rows (0.3 MB) 66.5 / 51.9, 2,090 FP64 (35 MB) 72.5 / 58.3,
  // 2,893 FP32 (33 MB) 81.4 / 65.1, 1,449 FP32 below 23,192 (8 MB) 195 / 179,
  // 2,893 FP64 (67 MB) 75.6 / 72.9, 4,660 FP32 (87 MB) 390 / 382; nothing
  // gained at 104 MB (3,614 FP64) and 174 MB (4,660 FP64), hence the limit.
  // NDS_DENSE_MB overrides it (0: none).
  static constexpr size_t kDenseBytes = (size_t)96 << 20;
  static size_t dense_ld(int n) { return ((size_t)n + 3) / 4 * 4; }
  void build_dense_level() {
    dense_level_ = -1;
    if (o_.amg_smoother == NDS_SM_MCGS) return;
    const size_t lim = std::getenv("NDS_DENSE_MB") ? (size_t)std::atoi(std::getenv("NDS_DENSE_MB")) << 20 : kDenseBytes;
    int l = 0;
    const int last = (int)L_.size() - 1;
    while (l < last && dense_ld(L_[(size_t)l].n) * (size_t)L_[(size_t)l].n * sizeof(TA) > lim) ++l;
    if (l >= last) return;
    const int m = L_[(size_t)l].n;
    std::vector<DBuf<TA>> B((size_t)(last - l + 1)), X((size_t)(last - l + 1));
    for (int q = l; q <= last; ++q) {
      B[(size_t)(q - l)].alloc((size_t)L_[(size_t)q].n * m);
      X[(size_t)(q - l)].alloc((size_t)L_[(size_t)q].n * m);
    }
    DBuf<TA> r, t0, t1;
    for (auto* b : {&r, &t0, &t1}) b->alloc((size_t)m * m);
    const size_t total = (size_t)m * m;
    k::block_unit<TA><<<grid_for((long long)total), kBlock, 0, st_>>>(total, m, B[0].p);
    NDS_LAUNCH();
    block_cycle(l, l, m, B, X, r.p, t0.p, t1.p);
    const size_t ld = dense_ld(m);
    dense_.alloc(ld * (size_t)m);
    NDS_CUDA(cudaMemsetAsync(dense_.p, 0, dense_.bytes(), st_));
    NDS_CUDA(cudaMemcpy2DAsync(dense_.p, ld * sizeof(TA), X[0].p, (size_t)m * sizeof(TA), (size_t)m * sizeof(TA),
                               (size_t)m, cudaMemcpyDeviceToDevice, st_));
    NDS_CUDA(cudaStreamSynchronize(st_));
    dense_level_ = l;
  }
  dim3 block_grid(int n, int m) const { return dim3((unsigned)grid_for(m), (unsigned)std::min(n, 65535)); }
  // y = epilogue(A x) of level q on m columns, with the values the level's SpMVs read
  template <int MODE>
  void block_op(const Level& A, int m, const TA* x, const TA* b, const TA* den, double w, TA* y) {
    const dim3 g = block_grid(A.n, m);
    auto run = [&](auto* ci, auto* v, double vinv) {
      using CT = std::remove_const_t<std::remove_pointer_t<decltype(ci)>>;
      using MT = std::remove_const_t<std::remove_pointer_t<decltype(v)>>;
      k::block_spmm<TA, MT, CT, MODE><<<g, kBlock, 0, st_>>>(A.n, m, A.row.p, ci, v, TA(vinv), x, b, den, TA(w), y);
    };
    if (A.hval.p && A.hcol.p) run(A.hcol.p, A.hval.p, A.hinv);
    else if (A.hval.p) run(A.col.p, A.hval.p, A.hinv);
    else run(A.col.p, A.val.p, 1.0);
    NDS_LAUNCH();
  }
  // x = S b of level q (poly_smooth on m columns; t the second buffer).  The
  // last step writes x.
  void block_smooth(int q, int m, const TA* b, TA* x, TA* t) {
    const Level& A = L_[(size_t)q];
    const PolyPlan pl = level_plan(q);
    const bool cheb = o_.amg_smoother == NDS_SM_CHEB2;
    const double lam = level_lambda_[(size_t)q], lo = cheb ? o_.amg_lambda_low_fraction * lam : 0.0;
    const size_t total = (size_t)A.n * m;
    TA* cur = poly_first(pl, x, t);
    TA* nxt = cur == x ? t : x;
    k::block_jacobi<TA><<<grid_for((long long)total), kBlock, 0, st_>>>(total, m, TA(pl.w0), b, pl.den0, cur);
    NDS_LAUNCH();
    for (int kk = 1; kk <= pl.m; ++kk) {
      const double w = cheb ? 1.0 / cheb_root(lam, lo, kk, o_.amg_cheb_degree) : o_.amg_jacobi_omega;
      block_op<k::BLK_SMOOTH>(A, m, cur, b, pl.den0, w, nxt);
      std::swap(cur, nxt);
    }
  }
  // vcycle(q, ...) on m columns; B[q - l], X[q - l]: right-hand sides and results
  void block_cycle(int l, int q, int m, std::vector<DBuf<TA>>& B, std::vector<DBuf<TA>>& X, TA* r, TA* t0, TA* t1) {
    const Level& A = L_[(size_t)q];
    TA* b = B[(size_t)(q - l)].p;
    TA* x = X[(size_t)(q - l)].p;
    if (q == (int)L_.size() - 1) {
      k::block_dense<TA><<<block_grid(A.n, m), kBlock, 0, st_>>>(A.n, (int)dense_ld(A.n), m, tinv_.p, b, x);
      NDS_LAUNCH();
      return;
    }
    const size_t total = (size_t)A.n * m;
    block_smooth(q, m, b, x, t0);
    block_op<k::BLK_RESID>(A, m, x, b, nullptr, 0.0, r);
    const Xfer& P = X_[(size_t)q + 1];
    k::block_spmm<TA, TA, int32_t, k::BLK_Y><<<block_grid(P.nc, m), kBlock, 0, st_>>>(
        P.nc, m, P.rrow.p, P.rcol.p, P.rval.p, TA(1), r, nullptr, nullptr, TA(0), B[(size_t)(q - l) + 1].p);
    NDS_LAUNCH();
    block_cycle(l, q + 1, m, B, X, r, t0, t1);
    k::block_prolong_add<TA><<<block_grid(P.nf, m), kBlock, 0, st_>>>(P.nf, m, P.pw, P.pcol.p, P.pval.p,
                                                                      X[(size_t)(q - l) + 1].p, x);
    NDS_LAUNCH();
    block_op<k::BLK_RESID>(A, m, x, b, nullptr, 0.0, r);
    block_smooth(q, m, r, t1, t0);
    k::block_add<TA><<<grid_for((long long)total), kBlock, 0, st_>>>(total, t1, x);
    NDS_LAUNCH();
  }

  // -------------------------------------------------------------- V-cycle
  // pre_done: the diagonal step of this level's pre-smoother is already in
  // place (taken by the restriction that produced b)
  void vcycle(int l, const TA* b, TA* x, bool pre_done = false) {
    Level& A = L_[(size_t)l];
    if (l == dense_level_) {
      ProfScope ps(prof, st_, P_TERMINAL);
      pdl_launch(k::dense_rows<TA>, A.n, 32 * k::kDenseWarps, 0, st_, A.n, (int)dense_ld(A.n), dense_.p, b, x);
      NDS_LAUNCH();
      return;
    }
    if (l == (int)L_.size() - 1) {
      ProfScope ps(prof, st_, P_TERMINAL);
      pdl_launch(k::dense_rows<TA>, A.n, 32 * k::kDenseWarps, 0, st_, A.n, (int)dense_ld(A.n), tinv_.p, b, x);
      NDS_LAUNCH();
      return;
    }
    smooth_level(A, b, x, level_lambda_[(size_t)l], pre_done);
    op_resid(level_op(A), x, b, A.r.p);
    Level& C = L_[(size_t)l + 1];
    const bool fuse = fuse_pre(l + 1);
    restrict_to(X_[(size_t)l + 1], A.r.p, C.b.p, fuse ? l + 1 : -1);
    vcycle(l + 1, C.b.p, C.x.p, fuse);
    prolong(X_[(size_t)l + 1], C.x.p, x);
    // r = b - A x into b (b is no longer needed), then the post-smoother
    // solves A corr = r and x += corr
    const double lam = level_lambda_[(size_t)l];
    const int sm = o_.amg_smoother;
    if (sm == NDS_SM_MCGS) {
      op_resid(level_op(A), x, b, A.r.p, A.b.p);
      smooth_level(A, A.b.p, A.corr.p, lam);
      vaxpy(A.n, 1.0, A.corr.p, x);
      return;
    }
    // the residual kernel also takes the smoother's diagonal step, and the
    // last smoothing step adds the correction to x
    const bool cheb = sm == NDS_SM_CHEB2;
    const TA* den = sm == NDS_SM_L1JACOBI ? A.l1.p : A.diag.p;
    const PolyPlan pl = poly_plan(lam, cheb, A.diag.p, den, o_.amg_jacobi_coarse_sweeps);
    op_resid(level_op(A), x, b, A.b.p, poly_first(pl, A.corr.p, A.pong.p), pl.den0, pl.w0);
    poly_smooth(level_op(A), A.diag.p, A.b.p, A.corr.p, A.pong.p, lam, cheb, den, o_.amg_jacobi_coarse_sweeps, true, x);
  }
  // where the fine pre-smoother's diagonal step goes: with one step only
  // (m = 0, split form) the cycle works in ftmp_, so that the post-smoothing
  // step can write z from it in one product
  TA* fine_first(TA* z) {
    const PolyPlan pl = fine_plan();
    return split_ && pl.m == 0 ? ftmp_.p : poly_first(pl, z, fpong_.p);
  }
  // z = M b.  pre_done: the fine pre-smoother's diagonal step is already in
  // fine_first(z).  With r (split form only) the last kernel also takes r.z
  // and the step rho of PCG.
  template <class R = TA>
  void amg_apply(const TA* b, TA* z, bool pre_done = false, const R* r = nullptr) {
    const int sm = o_.amg_smoother;
    const bool one = split_ && fine_plan().m == 0;
    TA* x = one ? ftmp_.p : z;
    smooth_fine(b, x, pre_done);
    op_resid(fine_opV(), x, b, fr_.p);
    Level& C = L_[0];
    const bool fuse = fuse_pre(0);
    restrict_to(X_[0], fr_.p, C.b.p, fuse ? 0 : -1);
    vcycle(0, C.b.p, C.x.p, fuse);
    prolong(X_[0], C.x.p, x);
    if (sm == NDS_SM_MCGS) {
      op_resid(fine_opV(), z, b, fr_.p, frhs_.p);
      smooth_fine(frhs_.p, fcorr_.p);
      vaxpy(nc_, 1.0, fcorr_.p, z);
      return;
    }
    const bool cheb = sm == NDS_SM_CHEB2;
    const TA* den = sm == NDS_SM_L1JACOBI ? fl1_.p : fdiag_.p;
    const PolyPlan pl = poly_plan(fine_lambda_, cheb, fdiag_.p, den, o_.amg_jacobi_fine_sweeps);
    if (one) {  // z = x + w0 (b - A x) / den
      if (r) split_smooth_rho(fine_opV(), (const TA*)x, b, pl.den0, pl.w0, z, (TA*)nullptr, r);
      else op_smooth(fine_opV(), (const TA*)x, b, pl.den0, pl.w0, z);
      return;
    }
    // post-smoothing as on the levels: residual with the diagonal step, last
    // step added to z
    op_resid(fine_opV(), z, b, frhs_.p, poly_first(pl, fcorr_.p, fpong_.p), pl.den0, pl.w0);
    if (r && pl.m >= 1) {
      TA* cur = poly_first(pl, fcorr_.p, fpong_.p);
      TA* nxt = cur == fcorr_.p ? fpong_.p : fcorr_.p;
      const double lo = cheb ? o_.amg_lambda_low_fraction * fine_lambda_ : 0.0;
      for (int kk = 1; kk <= pl.m; ++kk) {
        const double w = cheb ? 1.0 / cheb_root(fine_lambda_, lo, kk, o_.amg_cheb_degree) : o_.amg_jacobi_omega;
        if (kk < pl.m) op_smooth(fine_opV(), (const TA*)cur, (const TA*)frhs_.p, pl.den0, w, nxt);
        else split_smooth_rho(fine_opV(), (const TA*)cur, (const TA*)frhs_.p, pl.den0, w, (TA*)nullptr, z, r);
        std::swap(cur, nxt);
      }
      return;
    }
    poly_smooth(fine_opV(), fdiag_.p, frhs_.p, fcorr_.p, fpong_.p, fine_lambda_, cheb, den, o_.amg_jacobi_fine_sweeps,
                true, z);
  }

  // ------------------------------------------------------ spectrum estimates
  double power_fine(int its, double safety) {
    TA* v = fcorr_.p;
    TA* u = frhs_.p;
    TA* au = ftmp_.p;
    TA* w = fr_.p;
    k::power_init<TA><<<grid_for(nc_), kBlock, 0, st_>>>(nc_, v);
    NDS_LAUNCH();
    const double vn = std::sqrt(dot_fetch((const TA*)v, (const TA*)v, nc_, S_TMP));
    k::scale<TA><<<grid_for(nc_), kBlock, 0, st_>>>(nc_, TA(1.0 / vn), v);
    NDS_LAUNCH();
    double ray = 0.0;
    for (int it = 0; it < its; ++it) {
      k::div_sqrt<TA><<<grid_for(nc_), kBlock, 0, st_>>>(nc_, v, fdiag_.p, u);
      op_spmv(fine_opV(), (const TA*)u, au);
      k::div_sqrt<TA><<<grid_for(nc_), kBlock, 0, st_>>>(nc_, au, fdiag_.p, w);
      NDS_LAUNCH();
      const double num = dot_fetch((const TA*)v, (const TA*)w, nc_, S_TMP),
                   den = dot_fetch((const TA*)v, (const TA*)v, nc_, S_TMP2);
      ray = num / std::max(den, 1e-300);
      const double wn = std::sqrt(dot_fetch((const TA*)w, (const TA*)w, nc_, S_TMP));
      if (!(ray > 0.0) || !(wn > 0.0) || !std::isfinite(ray) || !std::isfinite(wn))
        throw SolveFailure(NDS_E_BREAKDOWN, "fine GPU power iteration failed");
      vcopy(nc_, (const TA*)w, v);
      k::scale<TA><<<grid_for(nc_), kBlock, 0, st_>>>(nc_, TA(1.0 / wn), v);
      NDS_LAUNCH();
    }
    return safety * ray;
  }
  double power_level(Level& A, int its, double safety) {
    const int n = A.n;
    k::power_init<TA><<<grid_for(n), kBlock, 0, st_>>>(n, A.corr.p);
    NDS_LAUNCH();
    const double vn = std::sqrt(dot_fetch((const TA*)A.corr.p, (const TA*)A.corr.p, n, S_TMP));
    k::scale<TA><<<grid_for(n), kBlock, 0, st_>>>(n, TA(1.0 / vn), A.corr.p);
    NDS_LAUNCH();
    double ray = 0.0;
    for (int it = 0; it < its; ++it) {
      k::div_sqrt<TA><<<grid_for(n), kBlock, 0, st_>>>(n, A.corr.p, A.diag.p, A.b.p);
      op_spmv(level_op(A), (const TA*)A.b.p, A.tmp.p);
      k::div_sqrt<TA><<<grid_for(n), kBlock, 0, st_>>>(n, A.tmp.p, A.diag.p, A.r.p);
      NDS_LAUNCH();
      const double num = dot_fetch((const TA*)A.corr.p, (const TA*)A.r.p, n, S_TMP),
                   den = dot_fetch((const TA*)A.corr.p, (const TA*)A.corr.p, n, S_TMP2);
      ray = num / std::max(den, 1e-300);
      const double wn = std::sqrt(dot_fetch((const TA*)A.r.p, (const TA*)A.r.p, n, S_TMP));
      if (!(ray > 0.0) || !(wn > 0.0) || !std::isfinite(ray) || !std::isfinite(wn))
        throw SolveFailure(NDS_E_BREAKDOWN, "coarse GPU power iteration failed");
      vcopy(n, (const TA*)A.r.p, A.corr.p);
      k::scale<TA><<<grid_for(n), kBlock, 0, st_>>>(n, TA(1.0 / wn), A.corr.p);
      NDS_LAUNCH();
    }
    return safety * ray;
  }
  // lambda_max(M^-1 A) for the outer Chebyshev solver
  double precond_power(int its, double safety) {
    k::power_init<T><<<grid_for(nc_), kBlock, 0, st_>>>(nc_, pp_.p);
    NDS_LAUNCH();
    const double vn = std::sqrt(dot_fetch(pp_.p, pp_.p, nc_, S_TMP));
    k::scale<T><<<grid_for(nc_), kBlock, 0, st_>>>(nc_, T(1.0 / vn), pp_.p);
    NDS_LAUNCH();
    double est = 0.0;
    for (int kk = 0; kk < its; ++kk) {
      fine_apply(pp_.p, q_.p);
      amg_T(q_.p, z_.p);
      const double zn = std::sqrt(dot_fetch(z_.p, z_.p, nc_, S_TMP));
      const double ray = dot_fetch(pp_.p, z_.p, nc_, S_TMP2);
      if (!(zn > 0.0) || !std::isfinite(zn) || !std::isfinite(ray)) throw SolveFailure(NDS_E_BREAKDOWN, "preconditioned power failed");
      est = std::max(est, std::max(std::abs(ray), zn));
      vcopy(nc_, z_.p, pp_.p);
      k::scale<T><<<grid_for(nc_), kBlock, 0, st_>>>(nc_, T(1.0 / zn), pp_.p);
      NDS_LAUNCH();
    }
    const double hi = safety * est;
    if (!(hi > 0.0) || !std::isfinite(hi)) throw SolveFailure(NDS_E_BREAKDOWN, "preconditioned lambda invalid");
    return hi;
  }

  // ------------------------------------------------------ pressure solvers
  struct PRes {
    int its = 0;
    double rel = 1;
    bool ok = false;
  };
  // ||r0|| and the zero solution
  double p_start(const T* rhs) {
    pdl_launch(k::solve_start<T>, red_grid(nc_), kBlock, 0, st_, nc_, rhs, r_.p, x_.p, host_tail(S_TMP));
    NDS_LAUNCH();
    NDS_CUDA(cudaStreamSynchronize(st_));
    const double r0 = std::sqrt(hsc_[S_TMP]);
    if (!std::isfinite(r0)) throw SolveFailure(NDS_E_BREAKDOWN, "pressure initial norm nonfinite");
    return r0;
  }
  // r.z taken by the V-cycle's last kernel up to this many cells: it saves a
  // launch there, but each of that kernel's blocks waits for its stores before
  // it leaves its partial sum.  Microseconds of an iteration, a pass of its own /
  // the tail: FP64 47,880 cells 58.6 / 56.9, 105,984 82.2 / 80.0, 205,320 131.0 /
  // 130.9, 383,040 207.4 / 208.1; FP32 V-cycle 205,320 101.6 / 100.1, 383,040
  // 149.8 / 152.1, 1.23M 400 / 407.  The line holds for the defect's norm too
  // (fast configuration: 205,320 cells 99.7 / 98.7, 383,040 136.7 / 138.4).
  static constexpr int kRhoCells = 200000;
  // Vectors of a PCG solve in precision S (the preconditioner runs in TA):
  // rA the residual in TA when the precisions differ.
  template <class S>
  struct PcgVecs {
    S *x, *r, *q, *p;
    TA *z, *rA;
  };
  // the PCG loops take the fine pre-smoother's first step in the kernels that
  // produce r (plain V-cycle with a polynomial smoother only)
  bool pre_fused() const { return !stage_ && o_.amg_smoother != NDS_SM_MCGS; }
  // start of a PCG loop from the residual in v.r, or (from given) from s times
  // the FP64 residual `from`, scaled into v.r with v.x zeroed
  template <class S>
  void pcg_first(const PcgVecs<S>& v, double target, double r0, int cap, const double* from = nullptr, double s = 1.0) {
    const TA* den0 = nullptr;
    TA w0 = 0, *x1 = nullptr, *rA = nullptr;
    if (!resident_) {
      if (pre_fused()) {
        const PolyPlan pl = fine_plan();
        den0 = pl.den0;
        w0 = TA(pl.w0);
        x1 = fine_first(v.z);
      }
      rA = v.rA;
    }
    const k::SolveInit init = solve_init(target, r0, 1, cap);
    if (from)
      pdl_launch(k::loop_start<double, S, TA>, grid_for(nc_), kBlock, 0, st_, nc_, from, s, v.r, (S*)nullptr, v.x, rA,
                 den0, w0, x1, init);
    else
      pdl_launch(k::loop_start<S, S, TA>, rA || x1 ? grid_for(nc_) : 1, kBlock, 0, st_, rA || x1 ? nc_ : 0, v.r, 1.0,
                 (S*)nullptr, (S*)nullptr, (S*)nullptr, rA, den0, w0, x1, init);
    NDS_LAUNCH();
  }
  // One pass of a PCG loop: z = M r; rho (first pass: p = z) and beta; q = A p;
  // alpha; x and r; ||r||^2 and the stopping test.  In split form the scalar
  // steps are taken by the kernels before them.
  template <class S>
  void pcg_body(const PcgVecs<S>& v, const OpView<S>& A, cudaGraphConditionalHandle h) {
    const int g = red_grid(nc_);
    const bool fused = pre_fused();
    const TA* r = v.rA;
    if constexpr (std::is_same<S, TA>::value) r = v.r;
    if (split_ && nc_ <= kRhoCells) {
      amg_apply<S>(r, v.z, fused, v.r);
    } else {
      amg_apply(r, v.z, fused);
      pdl_launch(k::dot_step<S, TA, k::PCG_RHO>, g, kBlock, 0, st_, nc_, v.r, v.z, tail(S_RHON));
      NDS_LAUNCH();
    }
    pdl_launch(k::p_update_dev<S, TA>, grid_for(nc_), kBlock, 0, st_, nc_, sc_.p + S_BETA, ctl_.p, v.z, v.p);
    NDS_LAUNCH();
    if (split_) {
      split_dot(A, (const S*)v.p, v.q);
    } else {
      {
        ProfScope ps(prof, st_, A.cat);
        sell_launch<k::SELL_DOT, S>(A, g, v.p, nullptr, nullptr, 0.0, v.q, nullptr);
        NDS_LAUNCH();
      }
      pdl_launch(k::reduce_alpha, 1, kBlock, 0, st_, part_.p, g, sc_.p, flags_.p);
      NDS_LAUNCH();
    }
    const TA* den0 = nullptr;
    TA w0 = 0, *x1 = nullptr;
    if (fused) {
      const PolyPlan pl = fine_plan();
      den0 = pl.den0;
      w0 = TA(pl.w0);
      x1 = fine_first(v.z);
    }
    pdl_launch(k::xr_update<S, TA, k::PCG_CHECK>, g, kBlock, 0, st_, nc_, 0.0, sc_.p + S_ALPHA, v.p, v.q, v.x, v.r,
               tail(S_RN2, h), den0, w0, x1, v.rA);
    NDS_LAUNCH();
    if (!fused && v.rA) {
      pdl_launch(k::cast_copy<S, TA>, grid_for(nc_), kBlock, 0, st_, nc_, v.r, v.rA);
      NDS_LAUNCH();
    }
  }
  PcgVecs<T> pcg_vecs() {
    if constexpr (kSame) return {x_.p, r_.p, q_.p, pp_.p, z_.p, nullptr};
    else return {x_.p, r_.p, q_.p, pp_.p, zA_.p, rA_.p};
  }
  // The whole PCG loop as one kernel of one cluster (resident.cuh): the split
  // operator with a coarse level applied as a dense matrix, on meshes of up to
  // kResidentCells cells whose vectors fit the cluster's shared memory.
  // Microseconds of an iteration, loop of kernels / this: 720 cells FP64 35.5 /
  // 19.9, FP32 37 / 20, mixed FP16 46 / 30; 2,688 cells 37 / 29, 35.5 / 25.5,
  // 41 / 30.5; 3,840 to 4,032 cells of four shapes FP64 37 to 38.5 / 33 to 40,
  // FP32 36 / 29 to 34, mixed FP16 38 to 40 / 31 to 36; 4,608 cells 38 / 42,
  // 35 / 35, 42 / 40; at 9,600 cells half as fast, as eight SMs no longer keep
  // up.  NDS_RESIDENT overrides the line (0:
  // none).  It is an ordinary launch, taken with graphs off and under the
  // profiler too, so that those runs have the same sums.
  static constexpr int kResidentCells = 4000;
  // The coarse matrix is read from L2 by the eight SMs, 64 rows a block of 512:
  // with the classical hierarchy, which keeps a quarter of the cells, its rows
  // set the line.  Loop / this: 500 rows FP64 30.4 / 29.5, FP32 30.3 / 24.1; 536
  // rows 31.1 / 32.4, 30.9 / 29.5; 602 rows 32.4 / 34.8, 30.0 / 31.6; 834 rows
  // 31.7 / 52.5, 30.1 / 40.8.  SA hierarchies have 244 rows at 4,000 cells.
  static constexpr int kResidentRows = 512;
  // entries of n per block (at least 2: res_inverse)
  static int res_part(int n) { return std::max(2, (n + k::kResCluster - 1) / k::kResCluster); }
  void plan_resident() {
    resident_ = false;
    const bool dense0 = dense_level_ == 0 || L_.size() == 1;
    if (!split_ || !dense0 || o_.learned || (mixed_ && fg_m_ > 0)) return;
    if (o_.pressure_solver != NDS_P_PCG || fine_plan().m >= k::kResSteps) return;
    int cells = kResidentCells;
    if (const char* e = std::getenv("NDS_RESIDENT")) cells = std::atoi(e);
    const size_t ld = dense_ld(L_[0].n);
    if (nc_ > cells || L_[0].n > kResidentRows) return;
    const int chunk = res_part(nc_), vchunk = res_part(svert_.n);
    res_smem_ = mixed_ ? k::res_smem<float, TA>(chunk, vchunk, (int)ld) : k::res_smem<T, TA>(chunk, vchunk, (int)ld);
    int most = 0;
    NDS_CUDA(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, o_.device));
    most -= 2048;  // the kernel's static arrays
    if ((long long)res_smem_ > (long long)most) return;
    // the operators' copies, as far as they fit
    res_zmax_ = 0;
    for (int v = 0; v < svert_.n; v += vchunk)
      res_zmax_ = std::max(res_zmax_, P_.setup.fine.inc_off[(size_t)std::min(v + vchunk, svert_.n)] -
                                          P_.setup.fine.inc_off[(size_t)v]);
    const bool d16 = scell_.nd16 != nullptr;
    const size_t ca = mixed_ && o_.amg_half ? k::res_copy_bytes<TA, __half>(chunk, vchunk, res_zmax_, d16, sp_rec8_.p)
                                            : k::res_copy_bytes<TA, TA>(chunk, vchunk, res_zmax_, d16, false);
    const size_t cs = mixed_ ? k::res_copy_bytes<float, float>(chunk, vchunk, res_zmax_, d16, false)
                             : k::res_copy_bytes<T, T>(chunk, vchunk, res_zmax_, d16, false);
    const bool shared = (kSame || mixed_) && !(mixed_ && o_.amg_half);  // one operator for both
    res_copy_a_ = res_smem_ + ca <= (size_t)most;
    if (res_copy_a_) res_smem_ += ca;
    res_copy_s_ = !shared && res_copy_a_ && res_smem_ + cs <= (size_t)most;
    if (res_copy_s_) res_smem_ += cs;
    // one limit for every solver of the process: the attribute is the kernel's
    auto allow = [&](auto* kernel) {
      NDS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    };
    if constexpr (kSame) {
      allow(k::pcg_resident<T, TA, TA>);
    } else if (mixed_) {
      if (o_.amg_half) allow(k::pcg_resident<float, float, __half>);
      else allow(k::pcg_resident<float, float, float>);
    } else {
      allow(k::pcg_resident<T, TA, TA>);
    }
    resident_ = true;
  }
  template <class S>
  void pcg_on_chip(const PcgVecs<S>& v, const OpView<S>& A) {
    k::Resident<S, TA> a{};
    const OpView<TA> V = fine_opV();
    a.nc = nc_;
    a.chunk = res_part(nc_);
    a.inv_chunk = k::res_inverse(a.chunk);
    a.vchunk = res_part(svert_.n);
    a.inv_vchunk = k::res_inverse(a.vchunk);
    a.vs = A.sv;
    a.cs = A.sc;
    a.rvs = A.rv;
    a.va = V.sv;
    a.ca = V.sc;
    a.rva = V.rv;
    a.wscale = TA(V.wscale);
    a.tinv = TA(V.tinv);
    const PolyPlan pl = fine_plan();
    const bool cheb = o_.amg_smoother == NDS_SM_CHEB2;
    const double lo = cheb ? o_.amg_lambda_low_fraction * fine_lambda_ : 0.0;
    a.den = pl.den0;
    a.m = pl.m;
    a.w[0] = TA(pl.w0);
    for (int q = 1; q <= pl.m; ++q)
      a.w[q] = TA(cheb ? 1.0 / cheb_root(fine_lambda_, lo, q, o_.amg_cheb_degree) : o_.amg_jacobi_omega);
    const Xfer& X = X_[0];
    a.nk = L_[0].n;
    a.kchunk = (a.nk + k::kResCluster - 1) / k::kResCluster;
    a.ld = (int)dense_ld(a.nk);
    a.dense = dense_level_ == 0 ? dense_.p : tinv_.p;
    a.rr = X.rrow.p;
    a.rc = X.rcol.p;
    a.rv = X.rval.p;
    a.pw = X.pw;
    a.pc = X.pcol.p;
    a.pv = X.pval.p;
    a.zmax = res_zmax_;
    a.copy_a = res_copy_a_;
    a.copy_s = res_copy_s_;
    a.r = v.r;
    a.x = v.x;
    a.sc = sc_.p;
    a.r0_slot = S_R0;
    a.target_slot = S_TARGET;
    a.flags = flags_.p;
    a.ctl = ctl_.p;
    a.host = host_words();
    static_assert(S_RN2 == 3, "result slot of the kernel");
    {
      ProfScope ps(prof, st_, P_RESIDENT);
      if constexpr (std::is_same<S, float>::value && std::is_same<TA, float>::value && !kSame) {
        if (V.half) k::pcg_resident<S, TA, __half><<<k::kResCluster, k::kResBlock, res_smem_, st_>>>(a);
        else k::pcg_resident<S, TA, TA><<<k::kResCluster, k::kResBlock, res_smem_, st_>>>(a);
      } else {
        k::pcg_resident<S, TA, TA><<<k::kResCluster, k::kResBlock, res_smem_, st_>>>(a);
      }
      NDS_LAUNCH();
    }
    NDS_CUDA(cudaStreamSynchronize(st_));
  }
  // PCG with the iteration loop on the device: two host synchronisations per
  // solve (initial norm, final state) instead of one per iteration.  With
  // graphs off or the profiler on the same body runs launch by launch.
  PRes pcg(const T* rhs) {
    const double r0 = p_start(rhs);
    start_readback();
    if (r0 <= o_.p_atol) return {0, 0.0, true};
    pcg_first(pcg_vecs(), std::max(o_.p_atol, o_.p_rtol * r0), r0, o_.p_max);
    if (resident_) pcg_on_chip(pcg_vecs(), fine_op());
    else run_loop(g_loop_, [&](cudaGraphConditionalHandle h) { pcg_body(pcg_vecs(), fine_op(), h); });
    const int f = hflags_[0];
    if (f & 8) throw SolveFailure(NDS_E_BREAKDOWN, "pressure PCG initial rho nonpositive");
    if (f & 1) throw SolveFailure(NDS_E_BREAKDOWN, "pressure PCG pAp nonpositive");
    if (f & 2) throw SolveFailure(NDS_E_BREAKDOWN, "pressure PCG rho nonpositive");
    PRes R;
    R.its = hflags_[4];
    R.rel = std::sqrt(hsc_[S_RN2]) / std::max(r0, 1e-300);
    if ((f & 4) || !std::isfinite(R.rel)) throw SolveFailure(NDS_E_BREAKDOWN, "pressure PCG residual nonfinite");
    R.ok = hflags_[5] != 0;
    return R;
  }
  // Richardson (omega fixed) and outer Chebyshev (omega = 1/root_k)
  PRes stationary(const T* rhs, bool cheb) {
    const double r0 = p_start(rhs);
    start_readback();
    if (r0 <= o_.p_atol) return {0, 0.0, true};
    const double target = std::max(o_.p_atol, o_.p_rtol * r0);
    double centre = 0, radius = 0;
    if (cheb) {
      const double lo = o_.p_cheb_low_fraction * p_cheb_lambda_;
      centre = .5 * (p_cheb_lambda_ + lo);
      radius = .5 * (p_cheb_lambda_ - lo);
    }
    const double pi = 3.141592653589793238462643383279502884;
    PRes R;
    for (int kk = 0; kk < o_.p_max; ++kk) {
      double omega = o_.p_richardson_omega;
      if (cheb) {
        const int ri = kk % o_.p_cheb_degree;
        omega = 1.0 / (centre - radius * std::cos(pi * (2.0 * (double)ri + 1.0) / (2.0 * (double)o_.p_cheb_degree)));
      }
      amg_rz();
      fine_apply(z_.p, q_.p);
      const int g = red_grid(nc_);
      k::ReduceTail to{};
      to.part = part_.p;
      pdl_launch(k::xr_update<T, T, 0>, g, kBlock, 0, st_, nc_, omega, nullptr, z_.p, q_.p, x_.p, r_.p, to, nullptr,
                 T(0),
                 nullptr, nullptr);
      NDS_LAUNCH();
      reduce_host<1>(part_.p, g, S_RN2);
      const double rn = std::sqrt(hsc_[S_RN2]);
      R.its = kk + 1;
      R.rel = rn / std::max(r0, 1e-300);
      if (!std::isfinite(R.rel)) throw SolveFailure(NDS_E_BREAKDOWN, "pressure stationary residual nonfinite");
      if (rn <= target) {
        R.ok = true;
        break;
      }
    }
    return R;
  }

  // ------------------------------------------- mixed-precision pressure solve
  // (precision NDS_MIXED: Solver<double, float>).  No reference counterpart.
  // FP64 defect correction around FP32 inner Krylov solves:
  //   target = max(atol, rtol ||b||); x = Galerkin guess (or 0); r = b - A x
  //   while ||r|| > target:  solve A d = r / ||r|| in FP32 (PCG or FGMRES,
  //   FP32 operator copy and V-cycle) to max(inner_rtol, target / (2 ||r||));
  //   x += ||r|| d;  r = b - A x in FP64 on the FP64 operator.
  // The stopping rule is the reference's ||r|| <= max(atol, rtol ||r0||)
  // with r0 = b (its zero initial guess), checked on the FP64 residual.
  void alloc_mixed() {
    const size_t n = (size_t)nc_;
    for (auto* b : {&xf_, &rf_, &zf_, &pf_, &qf_}) b->alloc(n);
    fg_m_ = o_.p_krylov == NDS_KRYLOV_FGMRES ? o_.p_restart : 0;
    if (fg_m_ > 0) {
      fgV_.alloc((size_t)(fg_m_ + 1) * n);
      fgZ_.alloc((size_t)fg_m_ * n);
      fg_.alloc((size_t)k::FgLayout{fg_m_}.size());
      fgtick_.alloc((size_t)fg_m_ + 1);
      NDS_CUDA(cudaMemsetAsync(fgtick_.p, 0, fgtick_.bytes(), st_));
      fg_.zero(st_);
    }
    fgpart_.alloc((size_t)kMaxPartBlocks * std::max(fg_m_ + 1, 48));
    if (o_.p_guess > 0) {
      gY_.alloc((size_t)o_.p_guess * n);
      gW_.alloc((size_t)o_.p_guess * n);
      if (o_.p_guess_fresh) gYf_.alloc((size_t)o_.p_guess * n);
    }
  }
  // the preconditioner of the inner solves: z = M v (FP32).  With the
  // learned stage: z1 = N(v), t = v - A z1; the V-cycle then solves for t and
  // z = z1 + V(t) -- or, when the stage did not reduce the residual
  // (||t|| >= ||v||), z = V(v) (the plain preconditioner as fallback).
  void precond_f(const float* v, float* z) {
    if constexpr (!kSame) {
      if (!stage_) {
        amg_apply(v, z);
        return;
      }
      mpnn_forward(*stage_, stage_view(), v, st_z1_.p);
      op_resid(fine_opA(), (const float*)st_z1_.p, v, st_t_.p);
      dot_dev((const float*)st_t_.p, (const float*)st_t_.p, nc_, S_ST_T);
      dot_dev(v, v, nc_, S_ST_V);
      stage_select<<<red_grid(nc_), kBlock, 0, st_>>>(nc_, v, st_t_.p, st_z1_.p, sc_.p, S_ST_T, S_ST_V, st_cnt_.p);
      NDS_LAUNCH();
      amg_apply(st_t_.p, z);
      vaxpy(nc_, 1.0, (const float*)st_z1_.p, z);
    }
  }
  nds_mpnn_graph stage_view() const { return nds_mpnn_graph{nc_, sg_nbr_.p, sg_ew_.p, sg_dscale_.p}; }
  // face graph of the cells and the SELL offsets of its edges
  void build_stage_graph() {
    const Mesh& M = P_.mesh;
    const FineTopo& F = P_.setup.fine;
    std::vector<int32_t> nbr(4 * (size_t)nc_, -1), off(4 * (size_t)nc_, -1);
    std::vector<int> cnt((size_t)nc_, 0);
    auto add = [&](int a, int b) {
      if (cnt[(size_t)a] >= 4) throw std::runtime_error("learned stage: a cell with more than four face neighbours");
      nbr[4 * (size_t)a + cnt[(size_t)a]++] = b;
    };
    for (size_t f = 0; f < M.neighbour.size(); ++f) {
      add(M.owner[f], M.neighbour[f]);
      add(M.neighbour[f], M.owner[f]);
    }
    if (split_) {
      // position of each face in its cell (the edge weights' face couplings)
      std::vector<uint8_t> face(4 * (size_t)nc_, 0);
      std::vector<int> at((size_t)nc_, 0);
      auto local = [&](int c, size_t f) {
        for (int a = 0; a < 4; ++a)
          if ((size_t)M.opp[(size_t)c][(size_t)a] == f) return (uint8_t)a;
        throw std::runtime_error("learned stage: a face missing from its cell");
      };
      for (size_t f = 0; f < M.neighbour.size(); ++f)
        for (const int c : {M.owner[f], M.neighbour[f]}) face[4 * (size_t)c + (size_t)at[(size_t)c]++] = local(c, f);
      sg_face_.upload(face);
    }
    std::vector<int32_t> base((size_t)(nc_ + 31) / 32 + 1);
    if (!split_) NDS_CUDA(cudaMemcpy(base.data(), sbase_.p, sizeof(int32_t) * base.size(), cudaMemcpyDeviceToHost));
    for (int i = 0; i < nc_ && !split_; ++i)
      for (int k = 0; k < 4; ++k) {
        const int j = nbr[4 * (size_t)i + k];
        if (j < 0) continue;
        int pos = -1;
        for (int q = F.row[(size_t)i]; q < F.row[(size_t)i + 1]; ++q)
          if (F.col[(size_t)q] == j) pos = q - F.row[(size_t)i];
        if (pos < 0) throw std::runtime_error("learned stage: face neighbour missing from the pressure operator");
        off[4 * (size_t)i + k] = base[(size_t)(i >> 5)] + 128 * (pos >> 2) + 4 * (i & 31) + (pos & 3);
      }
    sg_nbr_.upload(nbr);
    if (!split_) sg_off_.upload(off);
    sg_ew_.alloc(4 * (size_t)nc_);
    sg_dscale_.alloc((size_t)nc_);
    st_z1_.alloc((size_t)nc_);
    st_t_.alloc((size_t)nc_);
    st_cnt_.alloc(2);
    st_cnt_.zero(st_);
  }
  // edge weights and scaling from the operator of the last refresh
  void update_stage_graph() {
    if constexpr (!kSame) {
      stage_dscale<<<grid_for(nc_), kBlock, 0, st_>>>(nc_, fdiag_.p, sg_dscale_.p);
      NDS_LAUNCH();
      if (split_)
        k::split_edges<T><<<grid_for(4LL * nc_), kBlock, 0, st_>>>(nc_, sg_nbr_.p, sg_face_.p, ref_.p, bco_.p,
                                                                   sp_rv_.p, sp_tau_.p, sg_dscale_.p, sg_ew_.p);
      else
        stage_edges<<<grid_for(4LL * nc_), kBlock, 0, st_>>>(nc_, sg_nbr_.p, sg_off_.p, fvalA_.p, sg_dscale_.p, sg_ew_.p);
      NDS_LAUNCH();
    }
  }
  void load_stage(const float* host) override {
    if constexpr (kSame) {
      throw SolveFailure(NDS_E_INVALID, "the learned stage needs precision mixed");
    } else {
      if (!mixed_ || fg_m_ == 0) throw SolveFailure(NDS_E_INVALID, "the learned stage needs precision mixed and FGMRES");
      if (!sg_nbr_.p) build_stage_graph();
      if (!stage_) stage_ = make_mpnn(nc_, false, st_);
      mpnn_set_params(*stage_, host);
      // the FGMRES loop body is captured with the stage: rebuild it
      if (g_fgmres_.exec) cudaGraphExecDestroy(g_fgmres_.exec);
      g_fgmres_.exec = nullptr;
      g_fgmres_.failed = false;
    }
  }
  void stage_graph(int32_t* nbr, float* ew, float* dscale) override {
    if constexpr (kSame) {
      throw SolveFailure(NDS_E_INVALID, "the learned stage needs precision mixed");
    } else {
      if (!sg_nbr_.p) build_stage_graph();
      update_stage_graph();
      if (nbr) NDS_CUDA(cudaMemcpyAsync(nbr, sg_nbr_.p, sg_nbr_.bytes(), cudaMemcpyDeviceToDevice, st_));
      if (ew) NDS_CUDA(cudaMemcpyAsync(ew, sg_ew_.p, sg_ew_.bytes(), cudaMemcpyDeviceToDevice, st_));
      if (dscale) NDS_CUDA(cudaMemcpyAsync(dscale, sg_dscale_.p, sg_dscale_.bytes(), cudaMemcpyDeviceToDevice, st_));
      NDS_CUDA(cudaStreamSynchronize(st_));
    }
  }
  void pressure_pair(float* rhs, float* x) override {
    if (rhs) {
      to_float<T><<<grid_for(nc_), kBlock, 0, st_>>>(nc_, rhs_.p, rhs);
      NDS_LAUNCH();
    }
    if (x) {
      to_float<T><<<grid_for(nc_), kBlock, 0, st_>>>(nc_, x_.p, x);
      NDS_LAUNCH();
    }
    NDS_CUDA(cudaStreamSynchronize(st_));
  }
  void apply_operator(const float* x, float* y) override {
    if constexpr (kSame) {
      throw SolveFailure(NDS_E_INVALID, "the FP32 operator product needs precision mixed or amg_fp32");
    } else {
      op_spmv(fine_opA(), x, y);
      NDS_CUDA(cudaStreamSynchronize(st_));
    }
  }
  void apply_operator_form(int form, const void* x, void* y) override {
    if (form == NDS_OP_STATE) op_spmv(fine_op(), static_cast<const T*>(x), static_cast<T*>(y));
    else if (form == NDS_OP_VCYCLE) op_spmv(fine_opV(), static_cast<const TA*>(x), static_cast<TA*>(y));
    else throw SolveFailure(NDS_E_INVALID, "unknown operator form");
    NDS_CUDA(cudaStreamSynchronize(st_));
  }
  void stage_counts(long long* applied, long long* fallbacks) override {
    unsigned long long c[2] = {0, 0};
    if (st_cnt_.p) {
      NDS_CUDA(cudaMemcpyAsync(c, st_cnt_.p, sizeof(c), cudaMemcpyDeviceToHost, st_));
      NDS_CUDA(cudaStreamSynchronize(st_));
    }
    if (applied) *applied = (long long)c[0];
    if (fallbacks) *fallbacks = (long long)c[1];
  }
  // one Arnoldi step of FGMRES: z_j = M v_j, w = A z_j, classical Gram-Schmidt
  // with FP64 dot products, Givens update of the least-squares problem
  void fg_body(cudaGraphConditionalHandle h) {
    if constexpr (!kSame) {
      const int g = red_grid(nc_);
      const k::FgLayout L{fg_m_};
      // rf_ holds v_j, and with pre_fused() the pre-smoother's first step is taken
      if (pre_fused()) amg_apply(rf_.p, zf_.p, true);
      else precond_f(rf_.p, zf_.p);
      if (split_) {  // w = A z_j, Z_j = z_j
        const OpView<float> A = fine_opA();
        ProfScope ps(prof, st_, A.cat);
        split_vertices(A, (const float*)zf_.p);
        split_types(A, [&](auto mt, auto d16) {
          pdl_launch(k::split_cell<float, k::SELL_Y, decltype(d16)::value, decltype(mt)>, grid_for(nc_), kBlock, 0,
                     st_, A.sc, A.w, zf_.p, nullptr, nullptr, 0.f, qf_.p, fgZ_.p, 1.f, (const float*)nullptr,
                     k::ReduceTail{}, ctl_.p);
        });
        NDS_LAUNCH();
      } else {
        pdl_launch(k::fg_store, grid_for(nc_), kBlock, 0, st_, nc_, zf_.p, ctl_.p, fgZ_.p);
        NDS_LAUNCH();
        op_spmv(fine_opA(), (const float*)zf_.p, qf_.p);
      }
      pdl_launch(k::fg_dots, dim3(g, std::min(fg_m_ + 1, k::kDotRows)), kBlock, 0, st_, nc_, fgV_.p, qf_.p, ctl_.p,
                 fgpart_.p, fgtick_.p, L, fg_.p);
      NDS_LAUNCH();
      pdl_launch(k::fg_orth, g, kBlock, 0, st_, nc_, fgV_.p, fg_.p, L, qf_.p, part_.p, ticket_.p, k::FgScalars{sc_.p,
                 S_RN2, S_WN, S_TARGET, ctl_.p, flags_.p, h, in_graph_, host_words()});
      NDS_LAUNCH();
      const PolyPlan pl = pre_fused() ? fine_plan() : PolyPlan{};
      pdl_launch(k::fg_normalize, grid_for(nc_), kBlock, 0, st_, nc_, qf_.p, sc_.p, S_WN, ctl_.p, fgV_.p, rf_.p,
                 pl.den0, float(pl.w0), pre_fused() ? fine_first(zf_.p) : nullptr);
      NDS_LAUNCH();
    }
  }
  template <class Body>
  bool build_loop(LoopGraph& G, Body&& body) {
    const bool was = prof.on;
    prof.on = false;
    cudaGraph_t graph = nullptr;
    bool ok = cudaGraphCreate(&graph, 0) == cudaSuccess;
    cudaGraphConditionalHandle h{};
    cudaGraphNodeParams cp{};
    cudaGraphNode_t node{};
    if (ok) ok = cudaGraphConditionalHandleCreate(&h, graph, 1, cudaGraphCondAssignDefault) == cudaSuccess;
    if (ok) {
      cp.type = cudaGraphNodeTypeConditional;
      cp.conditional.handle = h;
      cp.conditional.type = cudaGraphCondTypeWhile;
      cp.conditional.size = 1;
      ok = cudaGraphAddNode(&node, graph, nullptr, 0, &cp) == cudaSuccess;
    }
    const unsigned long long l0 = g_launches;
    if (ok) ok = cudaStreamBeginCaptureToGraph(st_, cp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                               cudaStreamCaptureModeThreadLocal) == cudaSuccess;
    if (ok) {
      bool body_ok = true;
      in_graph_ = 1;
      try {
        body(h);
      } catch (...) {
        body_ok = false;
      }
      in_graph_ = 0;
      ok = cudaStreamEndCapture(st_, nullptr) == cudaSuccess && body_ok;
    }
    G.body_kernels = g_launches - l0;
    g_launches = l0;
    if (ok) ok = cudaGraphInstantiate(&G.exec, graph, 0) == cudaSuccess;
    if (graph) cudaGraphDestroy(graph);
    if (!ok) {
      if (G.exec) cudaGraphExecDestroy(G.exec);
      G.exec = nullptr;
      G.failed = true;
      cudaGetLastError();
    }
    prof.on = was;
    return ok;
  }
  // Runs a device loop (or, with graphs off or the profiler on, the same
  // body launch by launch with a host-side test of the loop condition).
  // ctl[0..3] must be set by the caller; returns after the loop ends.
  template <class Body>
  void run_loop(LoopGraph& G, Body&& body) {
    if (use_graphs_ && !prof.on && !G.failed && (G.exec || build_loop(G, body))) {
      NDS_CUDA(cudaGraphLaunch(G.exec, st_));
      NDS_CUDA(cudaStreamSynchronize(st_));
      g_launches += (unsigned long long)hflags_[4] * G.body_kernels;
      return;
    }
    // host-driven: the body's check kernel (launched with in_graph_ = 0)
    // leaves the decision to this loop, which reads ctl and the flags
    for (;;) {
      body(cudaGraphConditionalHandle{});
      NDS_CUDA(cudaStreamSynchronize(st_));
      prof.collect();
      const int its = hflags_[4], conv = hflags_[5], cap = hflags_[7];
      if (conv || hflags_[0] != 0 || its >= cap) break;
    }
  }
  // inner FP32 PCG on r_ / rn from zero to ||r|| <= tol within cap iterations;
  // returns the iterations
  int inner_pcg(double rn, double tol, int cap) {
    if constexpr (!kSame) {
      const PcgVecs<float> v{xf_.p, rf_.p, qf_.p, pf_.p, zf_.p, nullptr};
      pcg_first(v, tol, 1.0, cap, r_.p, 1.0 / rn);
      if (resident_) pcg_on_chip(v, fine_opA());
      else run_loop(g_loopf_, [&](cudaGraphConditionalHandle h) { pcg_body(v, fine_opA(), h); });
    }
    const int f = hflags_[0];
    if (f & 8) throw SolveFailure(NDS_E_BREAKDOWN, "inner FP32 PCG initial rho nonpositive");
    if (f & 1) throw SolveFailure(NDS_E_BREAKDOWN, "inner FP32 PCG pAp nonpositive");
    if (f & 2) throw SolveFailure(NDS_E_BREAKDOWN, "inner FP32 PCG rho nonpositive");
    if (f & 4) throw SolveFailure(NDS_E_BREAKDOWN, "inner FP32 PCG residual nonfinite");
    return hflags_[4];
  }
  // one FGMRES pass on V_0 = r / rn: x += rn sum y_i z_i; returns the
  // Arnoldi steps taken
  int inner_fgmres(double rn, double tol, int cap) {
    const k::FgLayout L{fg_m_};
    if constexpr (!kSame) {
      const PolyPlan pl = pre_fused() ? fine_plan() : PolyPlan{};
      pdl_launch(k::loop_start<double, float, float>, grid_for(nc_), kBlock, 0, st_, nc_, r_.p, 1.0 / rn, fgV_.p,
                 rf_.p, (float*)nullptr, (float*)nullptr, pl.den0, float(pl.w0),
                 pre_fused() ? fine_first(zf_.p) : nullptr, solve_init(tol, 1.0, 0, cap));
      NDS_LAUNCH();
    }
    k::fg_start<<<1, 1, 0, st_>>>(fg_.p, L);
    NDS_LAUNCH();
    run_loop(g_fgmres_, [&](cudaGraphConditionalHandle h) { fg_body(h); });
    if (hflags_[0] & 16) throw SolveFailure(NDS_E_BREAKDOWN, "inner FGMRES breakdown or nonfinite value");
    const int k_done = hflags_[4];
    k::fg_backsolve<<<1, 1, 0, st_>>>(fg_.p, L, ctl_.p);
    NDS_LAUNCH();
    k::fg_combine<<<grid_for(nc_), kBlock, 0, st_>>>(nc_, fgZ_.p, fg_.p, L, ctl_.p, rn, x_.p);
    NDS_LAUNCH();
    return k_done;
  }
  // Galerkin guess over the stored corrections and their stored products:
  // sets x_ and the exact FP64 residual r_ = b - A x_; returns ||r|| (or a
  // negative value when the guess is not usable: then nothing is set)
  template <int K>
  double guess_k(const double* rhs) {
    constexpr int NG = K * (K + 1) / 2 + K;
    const int g = red_grid(nc_);
    if constexpr (!kSame) {
      if (o_.p_guess_fresh) {
        // products with this iteration's operator (FP32 copy), widened to FP64
        const size_t n = (size_t)nc_;
        for (int a = 0; a < K; ++a) {
          op_spmv(fine_opA(), (const float*)(gYf_.p + a * n), qf_.p);
          pdl_launch(k::cast_copy<float, double>, grid_for(nc_), kBlock, 0, st_, nc_, qf_.p, gW_.p + a * n);
          NDS_LAUNCH();
        }
      }
    }
    pdl_launch(k::guess_dots<K>, g, kBlock, 0, st_, nc_, gY_.p, gW_.p, rhs, fgpart_.p);
    NDS_LAUNCH();
    reduce_host<NG>(fgpart_.p, g, S_GUESS);
    // G c = f by Cholesky (no guess when G is not numerically positive
    // definite, e.g. for dependent corrections)
    double G[K][K], f[K], c[K];
    int q = 0;
    for (int a = 0; a < K; ++a)
      for (int b = a; b < K; ++b) G[a][b] = G[b][a] = hsc_[S_GUESS + q++];
    for (int a = 0; a < K; ++a) f[a] = hsc_[S_GUESS + q++];
    double Lc[K][K] = {};
    for (int a = 0; a < K; ++a) {
      for (int b = 0; b <= a; ++b) {
        double sum = G[a][b];
        for (int e = 0; e < b; ++e) sum -= Lc[a][e] * Lc[b][e];
        if (a == b) {
          if (!(sum > 1e-12 * std::max(G[a][a], 1e-300)) || !std::isfinite(sum)) return -1.0;
          Lc[a][a] = std::sqrt(sum);
        } else {
          Lc[a][b] = sum / Lc[b][b];
        }
      }
    }
    for (int a = 0; a < K; ++a) {
      double sum = f[a];
      for (int e = 0; e < a; ++e) sum -= Lc[a][e] * c[e];
      c[a] = sum / Lc[a][a];
    }
    for (int a = K - 1; a >= 0; --a) {
      double sum = c[a];
      for (int e = a + 1; e < K; ++e) sum -= Lc[e][a] * c[e];
      c[a] = sum / Lc[a][a];
    }
    k::GuessCoef<K> coef;
    for (int a = 0; a < K; ++a) {
      if (!std::isfinite(c[a])) return -1.0;
      coef.c[a] = c[a];
    }
    pdl_launch(k::guess_combine<K>, grid_for(nc_), kBlock, 0, st_, nc_, gY_.p, coef, x_.p);
    NDS_LAUNCH();
    return defect_norm(rhs);
  }
  // r_ = b - A x_ on the FP64 operator; returns ||r||
  double defect_norm(const double* rhs) {
    if constexpr (std::is_same<T, double>::value) {
      if (split_ && nc_ <= kRhoCells) {
        const OpView<double> A = fine_op();
        ProfScope ps(prof, st_, A.cat);
        split_vertices(A, (const double*)x_.p);
        split_types(A, [&](auto mt, auto d16) {
          pdl_launch(k::split_cell<double, k::SELL_RESID, decltype(d16)::value, decltype(mt), k::SUM_ONLY>,
                     grid_for(A.n), kBlock, 0, st_, A.sc, A.w, x_.p, rhs, (const double*)nullptr, 0.0, r_.p,
                     (double*)nullptr, A.tinv, (const double*)nullptr, host_tail(S_TMP), (const int*)nullptr);
        });
        NDS_LAUNCH();
        NDS_CUDA(cudaStreamSynchronize(st_));
        return std::sqrt(hsc_[S_TMP]);
      }
    }
    op_resid(fine_op(), (const T*)x_.p, (const T*)rhs, r_.p);
    return std::sqrt(dot_fetch((const T*)r_.p, (const T*)r_.p, nc_, S_TMP));
  }
  double apply_guess(const double* rhs) {
    switch (std::min(o_.p_guess, nguess_)) {
      case 1: return guess_k<1>(rhs);
      case 2: return guess_k<2>(rhs);
      case 3: return guess_k<3>(rhs);
      case 4: return guess_k<4>(rhs);
      case 5: return guess_k<5>(rhs);
      case 6: return guess_k<6>(rhs);
      case 7: return guess_k<7>(rhs);
      case 8: return guess_k<8>(rhs);
      default: return -1.0;
    }
  }
  // keep the solution and its product with this iteration's operator,
  // w = b - r (r_ holds the final FP64 defect b - A x)
  void store_guess(const double* rhs) {
    if (o_.p_guess <= 0) return;
    const size_t o = (size_t)guess_head_ * nc_;
    pdl_launch(k::guess_store, grid_for(nc_), kBlock, 0, st_, nc_, x_.p, rhs, r_.p, gY_.p + o, gW_.p + o);
    NDS_LAUNCH();
    if (gYf_.p) {
      pdl_launch(k::cast_copy<double, float>, grid_for(nc_), kBlock, 0, st_, nc_, x_.p, gYf_.p + o);
      NDS_LAUNCH();
    }
    guess_head_ = (guess_head_ + 1) % o_.p_guess;
    nguess_ = std::min(nguess_ + 1, o_.p_guess);
  }
  PRes mixed_solve(const T* rhs_t) {
    PRes R;
    if constexpr (!kSame) {
      const double* rhs = rhs_t;
      // ||b|| = ||B u + fixedDiv||: the continuity norm this iteration already read back
      const double bn = std::sqrt(hsc_[S_CONT2]);
      if (!std::isfinite(bn)) throw SolveFailure(NDS_E_BREAKDOWN, "pressure initial norm nonfinite");
      const double target = std::max(o_.p_atol, o_.p_rtol * bn);
      start_readback();
      if (bn <= o_.p_atol) {
        x_.zero(st_);
        R.ok = true;
        R.rel = 0.0;
        return R;
      }
      if (o_.learned && !stage_) throw SolveFailure(NDS_E_STATE, "learned stage enabled but no parameters loaded");
      if (stage_) update_stage_graph();
      double rn = -1.0;
      if (o_.p_guess > 0 && nguess_ > 0) rn = apply_guess(rhs);
      // a guess that does not reduce the residual is dropped
      if (!(rn >= 0.0) || !std::isfinite(rn) || rn >= bn) {
        x_.zero(st_);
        vcopy(nc_, rhs, r_.p);
        rn = bn;
      }
      int passes = 0;
      for (;;) {
        if (rn <= target) {
          R.ok = true;
          break;
        }
        if (passes >= o_.p_refine_max || R.its >= o_.p_max) break;
        const double tol = std::max(o_.p_inner_rtol, 0.5 * target / rn);
        const int cap = o_.p_max - R.its;
        if (fg_m_ > 0) {
          R.its += inner_fgmres(rn, tol, std::min(cap, fg_m_));
        } else {
          R.its += inner_pcg(rn, tol, cap);
          pdl_launch(k::axpy_from_float, grid_for(nc_), kBlock, 0, st_, nc_, rn, xf_.p, x_.p);
          NDS_LAUNCH();
        }
        ++passes;
        rn = defect_norm(rhs);
        if (!std::isfinite(rn)) throw SolveFailure(NDS_E_BREAKDOWN, "pressure defect nonfinite");
      }
      R.rel = rn / std::max(bn, 1e-300);
      last_passes_ = passes;
      if (stage_) mpnn_check(*stage_);
      if (R.ok) store_guess(rhs);
    }
    return R;
  }

  // ------------------------------------------------------ SIMPLE iteration
  void assemble() {
    k::MomArgs<T> a;
    a.nrows = nv_;
    a.span = mspan_.p;
    a.dpos = mdpos_.p;
    a.K = K_.p;
    a.inc_off = inc_off_.p;
    a.inc = inc_.p;
    a.ref = ref_.p;
    a.slot = slot_.p;
    a.C = cconv_.p;
    a.slotz = slotz_.p;
    a.Bz = bz_.p;
    a.pz = pz_.p;
    a.fixz = fixz_.p;
    a.bco = bco_.p;
    a.fixed = fixed_.p;
    a.u0 = uc(0);
    a.u1 = uc(1);
    a.u2 = uc(2);
    a.p = p_.p;
    a.s0 = s_[0].p;
    a.s1 = s_[1].p;
    a.s2 = s_[2].p;
    a.alpha_u = T(o_.alpha_u);
    a.rau_scale = T(o_.rau_scale);
    a.row_cap = row_cap_;
    a.A = A_.p;
    a.delta = delta_.p;
    a.diag = diag_.p;
    a.rau = rau_.p;
    a.b0 = b_[0].p;
    a.b1 = b_[1].p;
    a.b2 = b_[2].p;
    a.invJ = invJ_.p;
    a.det = det_.p;
    a.table = conv_table_.p;
    ProfScope ps(prof, st_, P_ASSEMBLE);
    if (fused_assembly_) {
      // one pass: each incidence's convection row is evaluated in place
      pdl_launch(k::mom_assemble<T, 1>, grid_for(nv_, kBlock / 8), kBlock, mom_smem_ + kConvTable * sizeof(T), st_, a);
      NDS_LAUNCH();
      return;
    }
    // cell blocks: a grid of 4 blocks per SM amortises the load of the shared table
    k::SupgArgs sa{P_.setup.pipe.nu, o_.supg_tau_scale, o_.supg_magic};
    const int gc = std::min(grid_for(nc_, kBlock / 4), 4 * kSms);
    k::mom_cell_conv<T><<<gc, kBlock, 0, st_>>>(nc_, ref_.p, fixed_.p, uc(0), uc(1), uc(2), invJ_.p, det_.p,
                                                 conv_table_.p, zpos_.p, cconv_.p, p_.p, pz_.p);
    if (o_.supg) {
      NDS_LAUNCH();
      k::mom_cell_supg<T><<<gc, kBlock, 0, st_>>>(nc_, ref_.p, fixed_.p, uc(0), uc(1), uc(2), invJ_.p, det_.p, zpos_.p,
                                                  cconv_.p, supg_rule_.p, h2_.p, sa);
    }
    NDS_LAUNCH();
    pdl_launch(k::mom_assemble<T>, grid_for(nv_, kBlock / 8), kBlock, mom_smem_, st_, a);
    NDS_LAUNCH();
  }
  void gs_pass(bool reverse) {
    const int ncol = (int)color_off_.size() - 1;
    for (int qq = 0; qq < ncol; ++qq) {
      const int c = reverse ? ncol - 1 - qq : qq;
      const int s = color_off_[(size_t)c], n = color_off_[(size_t)c + 1] - s;
      if (!n) continue;
      ProfScope ps(prof, st_, P_GS);
      pdl_launch(k::mom_gs_color<T>, grid_for((long long)n * 8), kBlock, 0, st_, n, color_rows_.p + s, gspan_.p + s,
                 mcol_.p, A_.p, diag_.p, b_[0].p, b_[1].p, b_[2].p, uc(0), uc(1), uc(2), T(o_.mom_omega));
      NDS_LAUNCH();
    }
  }
  std::array<double, 3> audit() {
    const int g = red_grid((long long)nv_ * 8);
    k::mom_audit<T><<<g, kBlock, 0, st_>>>(nv_, mspan_.p, mcol_.p, A_.p, b_[0].p, b_[1].p, b_[2].p, uc(0), uc(1),
                                           uc(2), part_.p);
    NDS_LAUNCH();
    reduce_host<6>(part_.p, g, S_AUDIT);
    std::array<double, 3> q{};
    for (int d = 0; d < 3; ++d) {
      double bn = std::sqrt(std::max(0.0, hsc_[S_AUDIT + d]));
      if (bn == 0.0) bn = 1.0;
      q[(size_t)d] = std::sqrt(std::max(0.0, hsc_[S_AUDIT + 3 + d])) / bn;
    }
    return q;
  }
  double rau_snapshot_rel() {
    // ||rau - rau_setup|| / ||rau_setup||, in double on the host copies
    std::vector<T> a((size_t)nv_), b((size_t)nv_);
    NDS_CUDA(cudaMemcpyAsync(a.data(), rau_.p, sizeof(T) * nv_, cudaMemcpyDeviceToHost, st_));
    NDS_CUDA(cudaMemcpyAsync(b.data(), rau_pc_.p, sizeof(T) * nv_, cudaMemcpyDeviceToHost, st_));
    NDS_CUDA(cudaStreamSynchronize(st_));
    long double d = 0, r = 0;
    for (int i = 0; i < nv_; ++i) {
      const long double q = (long double)a[(size_t)i] - (long double)b[(size_t)i];
      d += q * q;
      r += (long double)b[(size_t)i] * b[(size_t)i];
    }
    return std::sqrt((double)d) / std::max(std::sqrt((double)r), 1e-300);
  }

  void reset() override {
    u3_.zero(st_);
    p_.zero(st_);
    it_ = 0;
    nguess_ = 0;
    guess_head_ = 0;
    cont0_ = -1.0;
    cont_rel_ = 1.0;
    NDS_CUDA(cudaStreamSynchronize(st_));
  }

  void step(nds_iter_report* rep) override {
    const int it = ++it_;
    nds_iter_report R{};
    R.it = it;
    NDS_CUDA(cudaEventRecord(ev_[0], st_));
    assemble();
    NDS_CUDA(cudaEventRecord(ev_[1], st_));
    // The fine Schur refresh needs only rAU from the assembly: it runs on the
    // side stream while the momentum sweep and the continuity residual run
    // on the main stream (it writes only the pressure operator, which
    // nothing reads until the pressure solve waits for it).
    NDS_CUDA(cudaEventRecord(ev_side_[0], st_));
    NDS_CUDA(cudaStreamWaitEvent(st2_, ev_side_[0], 0));
    refresh_fine(rau_.p, st2_);
    NDS_CUDA(cudaEventRecord(ev_side_[1], st2_));
    if (it == 1) {
      const double rr = rau_snapshot_rel();
      if (!(rr < o_.snapshot_tol))
        throw SolveFailure(NDS_E_SETUP, "setup rAU snapshot mismatch (rel " + std::to_string(rr) + ")");
    }
    const bool converge = o_.run_mode == NDS_RUN_CONVERGE;
    if (converge && it > 1 && cont_rel_ <= o_.simple_tol) {
      auto q = audit();
      R.audited = 1;
      for (int d = 0; d < 3; ++d) R.audit_rel[d] = q[(size_t)d];
    }
    if (o_.momentum_work == NDS_MOM_FGS1) gs_pass(false);
    else if (o_.momentum_work == NDS_MOM_ALTGS1) gs_pass((it & 1) == 0);
    else { gs_pass(false); gs_pass(true); }
    NDS_CUDA(cudaEventRecord(ev_[2], st_));
    {
      const int g = red_grid(nc_);
      ProfScope ps(prof, st_, P_CONTINUITY);
      pdl_launch(k::continuity<T>, g, kBlock, 0, st_, nc_, ref_.p, bco_.p, fixed_div_.p, uc(0), uc(1), uc(2), rhs_.p,
                 part_.p);
      NDS_LAUNCH();
      reduce_host<1>(part_.p, g, S_CONT2);
    }
    const double cn = std::sqrt(hsc_[S_CONT2]);
    if (it == 1) cont0_ = cn;
    cont_rel_ = cn / std::max(cont0_, 1e-300);
    R.cont_norm = cn;
    R.rel_cont = cont_rel_;
    NDS_CUDA(cudaEventRecord(ev_[3], st_));
    NDS_CUDA(cudaStreamWaitEvent(st_, ev_side_[1], 0));
    NDS_CUDA(cudaEventRecord(ev_[6], st_));
    PRes pr;
    if (mixed_) pr = mixed_solve(rhs_.p);
    else if (o_.pressure_solver == NDS_P_PCG) pr = pcg(rhs_.p);
    else pr = stationary(rhs_.p, o_.pressure_solver == NDS_P_CHEB);
    R.p_its = pr.its;
    R.p_rel = pr.rel;
    NDS_CUDA(cudaEventRecord(ev_[4], st_));
    if (!pr.ok) {
      last_ = R;
      throw SolveFailure(NDS_E_NOT_CONVERGED, "pressure solve failed its requested target");
    }
    vaxpy(nc_, o_.alpha_p, x_.p, p_.p);
    NDS_CUDA(cudaEventRecord(ev_[5], st_));
    if constexpr (std::is_same<T, double>::value) {
      if (io_out_ && io_out_[3]) NDS_CUDA(cudaMemcpyAsync(io_out_[3], p_.p, p_.bytes(), cudaMemcpyDeviceToHost, st_));
    }
    NDS_CUDA(cudaStreamSynchronize(st_));
    if (io_pending_) {
      NDS_CUDA(cudaEventSynchronize(ev_io_));
      io_pending_ = false;
    }
    prof.collect();
    float ms[5];
    for (int q = 0; q < 5; ++q) NDS_CUDA(cudaEventElapsedTime(&ms[q], ev_[q], ev_[q + 1]));
    R.ms_assembly = ms[0];
    R.ms_momentum = ms[1];
    R.ms_continuity = ms[2];
    R.ms_pressure = ms[3];
    R.ms_update = ms[4];
    float msr = 0.f;
    NDS_CUDA(cudaEventElapsedTime(&msr, ev_[3], ev_[6]));
    R.ms_refresh = msr;
    const bool finite = std::isfinite(R.rel_cont) && std::isfinite(R.p_rel) &&
                        (!R.audited || (std::isfinite(R.audit_rel[0]) && std::isfinite(R.audit_rel[1]) &&
                                        std::isfinite(R.audit_rel[2])));
    finite_all_ = finite_all_ && finite;
    if (R.audited)
      R.all_momentum_met = R.audit_rel[0] <= o_.simple_tol && R.audit_rel[1] <= o_.simple_tol &&
                           R.audit_rel[2] <= o_.simple_tol;
    R.converged = converge && finite_all_ && R.rel_cont <= o_.simple_tol && R.audited && R.all_momentum_met;
    last_ = R;
    if (rep) *rep = R;
  }

  void solve(nds_solve_report* rep) override {
    nds_solve_report S{};
    S.pressure_all = 1;
    finite_all_ = true;
    long long sumP = 0;
    for (int it = 1; it <= o_.max_outer; ++it) {
      nds_iter_report R{};
      step(&R);
      sumP += R.p_its;
      S.outer_its = R.it;
      S.final_rel_cont = R.rel_cont;
      if (R.audited)
        for (int d = 0; d < 3; ++d) S.final_audit_rel[d] = R.audit_rel[d];
      S.assembly_ms += R.ms_assembly;
      S.momentum_ms += R.ms_momentum;
      S.continuity_ms += R.ms_continuity;
      S.pressure_ms += R.ms_pressure;
      S.update_ms += R.ms_update;
      if (o_.verbose)
        std::printf(
            "NODALS_GPU_H8_SIMPLE it=%d relCont=%.12e pCG=%d pTrueRel=%.3e residualAudit=%s auditInitRel=[%.3e,%.3e,%.3e] "
            "allMomentumMet=%d converged=%d\n",
            R.it, R.rel_cont, R.p_its, R.p_rel, R.audited ? "DONE" : "SKIPPED", R.audit_rel[0], R.audit_rel[1],
            R.audit_rel[2], R.all_momentum_met, R.converged);
      if (R.converged) {
        S.converged = 1;
        break;
      }
    }
    S.finite_all = finite_all_;
    S.avg_pressure_its = S.outer_its ? (double)sumP / S.outer_its : 0.0;
    S.loop_ms = S.assembly_ms + S.momentum_ms + S.continuity_ms + S.pressure_ms + S.update_ms;
    if (rep) *rep = S;
  }

  bool cell_arrays(const int32_t** ref, const double** bco, const double** fixed_div, int* nc,
                   int* device) const override {
    if constexpr (std::is_same<T, double>::value) {
      *ref = ref_.p;
      *bco = bco_.p;
      *fixed_div = fixed_div_.p;
      *nc = nc_;
      *device = o_.device;
      return true;
    } else {
      return false;
    }
  }
  void get_fields(double* u0, double* u1, double* u2, double* p) override {
    std::vector<T> h;
    auto get = [&](const DBuf<T>& b, double* out) {
      if (!out) return;
      if (std::is_same<T, double>::value) {  // straight DMA into the caller's buffer
        NDS_CUDA(cudaMemcpyAsync(out, b.p, b.bytes(), cudaMemcpyDeviceToHost, st_));
        NDS_CUDA(cudaStreamSynchronize(st_));
        return;
      }
      h.resize(b.n);
      NDS_CUDA(cudaMemcpyAsync(h.data(), b.p, b.bytes(), cudaMemcpyDeviceToHost, st_));
      NDS_CUDA(cudaStreamSynchronize(st_));
      for (size_t i = 0; i < b.n; ++i) out[i] = (double)h[i];
    };
    if (u0 || u1 || u2) {
      k::deinterleave3<T><<<grid_for(nv_), kBlock, 0, st_>>>(nv_, u3_.p, v_[0].p, v_[1].p, v_[2].p);
      NDS_LAUNCH();
    }
    get(v_[0], u0);
    get(v_[1], u1);
    get(v_[2], u2);
    get(p_, p);
  }
  void set_fields(const double* u0, const double* u1, const double* u2, const double* p) override {
    auto put = [&](DBuf<T>& b, const double* in) {
      if (!in) return;
      if (std::is_same<T, double>::value) {
        NDS_CUDA(cudaMemcpyAsync(b.p, in, b.bytes(), cudaMemcpyHostToDevice, st_));
        NDS_CUDA(cudaStreamSynchronize(st_));
        return;
      }
      std::vector<T> h(in, in + b.n);
      NDS_CUDA(cudaMemcpyAsync(b.p, h.data(), b.bytes(), cudaMemcpyHostToDevice, st_));
      NDS_CUDA(cudaStreamSynchronize(st_));
    };
    put(v_[0], u0);
    put(v_[1], u1);
    put(v_[2], u2);
    if (u0 || u1 || u2) {
      k::interleave3<T><<<grid_for(nv_), kBlock, 0, st_>>>(nv_, u0 ? v_[0].p : nullptr, u1 ? v_[1].p : nullptr,
                                                           u2 ? v_[2].p : nullptr, u3_.p);
      NDS_LAUNCH();
      NDS_CUDA(cudaStreamSynchronize(st_));
    }
    put(p_, p);
  }

  // step_io: the velocity is final after the momentum sweep (event ev_[2]);
  // it is read back on the I/O stream once the pressure solve has read its
  // initial norm, so that the copy runs under the device-side Krylov loop.
  // (Issued earlier, it would hold up the small reads the host waits for
  // between the sweep and the loop: they share the copy engine.)
  void start_readback() {
    if constexpr (std::is_same<T, double>::value) {
      if (!io_out_ || io_issued_ || !(io_out_[0] || io_out_[1] || io_out_[2])) return;
      io_issued_ = true;
      NDS_CUDA(cudaStreamWaitEvent(st_io_, ev_[2], 0));
      k::deinterleave3<T><<<grid_for(nv_), kBlock, 0, st_io_>>>(nv_, u3_.p, v_[0].p, v_[1].p, v_[2].p);
      NDS_LAUNCH();
      for (int d = 0; d < 3; ++d)
        if (io_out_[d]) NDS_CUDA(cudaMemcpyAsync(io_out_[d], v_[d].p, v_[d].bytes(), cudaMemcpyDeviceToHost, st_io_));
      NDS_CUDA(cudaEventRecord(ev_io_, st_io_));
      io_pending_ = true;
    }
  }
  void step_io(const double* const in[4], double* const out[4], nds_iter_report* rep) override {
    set_fields(in[0], in[1], in[2], in[3]);
    // Overlapped read-back needs an FP64 state (no host-side conversion) and
    // page-locked outputs (a copy into pageable memory would block the host
    // before the rest of the step is queued).
    bool overlap = std::is_same<T, double>::value;
    for (int q = 0; q < 4 && overlap; ++q) {
      if (!out[q]) continue;
      cudaPointerAttributes a{};
      if (cudaPointerGetAttributes(&a, out[q]) != cudaSuccess || a.type != cudaMemoryTypeHost) {
        cudaGetLastError();
        overlap = false;
      }
    }
    if (!overlap) {
      step(rep);
      get_fields(out[0], out[1], out[2], out[3]);
      return;
    }
    io_out_ = out;
    io_issued_ = false;
    try {
      step(rep);
      start_readback();  // no-op unless the pressure stage did not issue it
      if (io_pending_) {
        NDS_CUDA(cudaEventSynchronize(ev_io_));
        io_pending_ = false;
      }
    } catch (...) {
      // no copy may write the caller's arrays after the call returns
      io_out_ = nullptr;
      cudaStreamSynchronize(st_io_);
      cudaStreamSynchronize(st_);
      io_pending_ = false;
      throw;
    }
    io_out_ = nullptr;
  }

  nds_iter_report last_{};

 private:
  const Problem& P_;
  nds_options o_;
  cudaStream_t st_ = nullptr;
  cudaStream_t st2_ = nullptr;      // side stream of the fine Schur refresh
  cudaEvent_t ev_side_[2] = {};     // assembly done -> refresh; refresh done -> pressure
  cudaStream_t st_io_ = nullptr;    // read-back of step_io
  cudaEvent_t ev_io_ = nullptr;
  double* const* io_out_ = nullptr;  // outputs of the step_io call in progress
  bool io_pending_ = false, io_issued_ = false;
  cudaEvent_t ev_[7] = {};
  int nc_ = 0, nv_ = 0, row_cap_ = 0, it_ = 0;
  size_t mom_smem_ = 0, refresh_smem_ = 0;
  double cont0_ = -1, cont_rel_ = 1, fine_lambda_ = 1, p_cheb_lambda_ = 1;
  bool finite_all_ = true;
  bool fused_assembly_ = false;
  // lanes per row of the FP16 level SpMVs and of the restriction in the
  // mixed FP16 V-cycle (16 measured best at pipe1m: 0.25 ms per SIMPLE
  // iteration less than 32 or 8); NDS_LEVEL_LANES=8|16|32 overrides
  int level_lanes_ = std::getenv("NDS_LEVEL_LANES") ? std::atoi(std::getenv("NDS_LEVEL_LANES")) : 16;
  std::vector<double> level_lambda_;
  // momentum
  DBuf<int32_t> mcol_, mdpos_, inc_off_, ref_, color_rows_;
  DBuf<uint32_t> inc_;
  DBuf<int32_t> zpos_;  // incidence of (cell, basis), -1 for a fixed dof
  DBuf<uint8_t> slot_, slotz_, fixz_;  // slots per (cell, basis) and per incidence; fixed-dof masks
  DBuf<T> K_, A_, diag_, delta_, rau_, rau_pc_, det_, invJ_, bco_, fixed_, fixed_div_, conv_table_, cconv_, fgeo_, p_, bz_, pz_;
  DBuf<T> h2_, supg_rule_;
  DBuf<T> u3_, b_[3], s_[3], v_[3];  // u3_: interleaved velocity; v_: staging of get/set fields
  static constexpr int kVelComponents = k::kVel;
  T* uc(int d) const { return u3_.p + d; }
  std::vector<int> color_off_;
  DBuf<int2> mspan_, gspan_;  // momentum rows' storage spans, by row / by colour position
  // pressure
  DBuf<int32_t> fcoff_, fine_crows_, sbase_, swidth_, scol_, fdslot_;
  DBuf<int16_t> sdcol_;
  k::Sell sell_{};
  long long sell_nnz_ = 0;
  std::vector<int> fine_coff_;
  // split form of the pressure operator
  bool split_ = false, half_on_ = false;
  k::SplitVerts svert_{};
  k::SplitCells scell_{};
  double bscale_ = 1.0;
  DBuf<int32_t> sp_off_, sp_cell_, sp_base_;
  DBuf<int4> sp_vid_, sp_nid_;
  DBuf<short4> sp_nd16_;
  DBuf<T> sp_g4_, sp_rv_, sp_tau_, sp_w_;
  DBuf<TA> sp_rvA_, sp_tauA_, sp_wA_;
  DBuf<double> sp_b_[3], sp_gd1_;
  DBuf<double2> sp_gd2_;
  DBuf<float4> sp_rec16_, sp_rec16h_, sp_gf4_;
  DBuf<float> sp_gf1_;
  DBuf<uint2> sp_rec8_, sp_h2_;
  DBuf<uint4> sp_h4_;
  DBuf<__half> sp_tauH_;
  DBuf<uint16_t> fcs_;
  DBuf<int> ctl_;

  DBuf<T> fval_, x_, r_, z_, pp_, q_, rhs_;
  DBuf<TA> fvalA_, fdiag_, fl1_, fr_, ftmp_, fcorr_, frhs_, fpong_, tinv_, rA_, zA_;
  std::vector<Level> L_;
  int dense_level_ = -1;  // the level applied as its V-cycle matrix dense_ (-1: none)
  DBuf<TA> dense_;
  std::vector<Xfer> X_;
  // mixed precision (NDS_MIXED): inner FP32 Krylov vectors, FGMRES basis
  // V (m+1 vectors) and preconditioned vectors Z (m), its FP64 work array,
  // and the stored corrections Y (and A Y) of the Galerkin guess
  bool mixed_ = false;
  int in_graph_ = 0;  // 1 while a loop body is being captured (its check kernel sets the graph condition)
  int fg_m_ = 0, nguess_ = 0, guess_head_ = 0, last_passes_ = 0;
  DBuf<float> xf_, rf_, zf_, pf_, qf_, fgV_, fgZ_, gYf_;
  DBuf<__half> fvalH_;  // FP16 copy of the fine operator for the V-cycle (amg_half)
  double hscale_ = 1.0;
  DBuf<double> fg_, fgpart_, gY_, gW_;
  DBuf<unsigned> fgtick_;  // of the FGMRES dots, one per basis vector
  LoopGraph g_loopf_, g_fgmres_;
  // learned stage: network state, face graph (neighbours, SELL offsets of
  // the edges, edge weights, Jacobi scaling), work vectors, counters
  MpnnPtr stage_;
  DBuf<int32_t> sg_nbr_, sg_off_;
  DBuf<uint8_t> sg_face_;
  DBuf<float> sg_ew_, sg_dscale_, st_z1_, st_t_;
  DBuf<unsigned long long> st_cnt_;
  bool resident_ = false;  // PCG as one kernel
  size_t res_smem_ = 0;
  int res_zmax_ = 0;
  bool res_copy_a_ = false, res_copy_s_ = false;
  DBuf<double> part_, sc_, tailpart_;
  DBuf<unsigned> ticket_;  // of the reduction tails (stream st_, one launch at a time)
  DBuf<int> flags_;
  double* hsc_ = nullptr;
  int* hflags_ = nullptr;  // [0] flags, [4..7] device-loop control words
};

}  // namespace nds

// ============================================================== C ABI
struct nds_solver {
  std::unique_ptr<nds::ISolver> impl;
};

namespace {
int fail(int code, const std::string& m) {
  nds::set_error(m);
  return code;
}
template <class F>
int guarded(F&& f) {
  try {
    f();
    return NDS_OK;
  } catch (const nds::SolveFailure& e) {
    return fail(e.code, e.what());
  } catch (const nds::CudaError& e) {
    return fail(NDS_E_CUDA, e.what());
  } catch (const std::exception& e) {
    return fail(NDS_E_SETUP, e.what());
  }
}
}  // namespace

extern "C" {

int nds_solver_create(const nds_problem* pp, nds_solver** out) {
  if (!pp || !out) return fail(NDS_E_INVALID, "null argument");
  const auto* P = reinterpret_cast<const nds::Problem*>(pp);
  return guarded([&] {
    int ndev = 0;
    const cudaError_t e = cudaGetDeviceCount(&ndev);
    if (e != cudaSuccess || ndev <= P->opt.device)
      throw nds::CudaError(std::string("no CUDA device available: ") + cudaGetErrorString(e));
    auto s = std::make_unique<nds_solver>();
    if (P->opt.precision == NDS_FP64) s->impl = std::make_unique<nds::Solver<double, double>>(*P);
    else if (P->opt.precision == NDS_FP32) s->impl = std::make_unique<nds::Solver<float, float>>(*P);
    else s->impl = std::make_unique<nds::Solver<double, float>>(*P);
    *out = s.release();
  });
}
int nds_solver_reset(nds_solver* s) {
  if (!s) return fail(NDS_E_INVALID, "null solver");
  return guarded([&] { s->impl->reset(); });
}
int nds_simple_step(nds_solver* s, nds_iter_report* r) {
  if (!s) return fail(NDS_E_INVALID, "null solver");
  return guarded([&] { s->impl->step(r); });
}
int nds_solve(nds_solver* s, nds_solve_report* r) {
  if (!s) return fail(NDS_E_INVALID, "null solver");
  return guarded([&] { s->impl->solve(r); });
}
int nds_get_fields(nds_solver* s, double* u0, double* u1, double* u2, double* p) {
  if (!s) return fail(NDS_E_INVALID, "null solver");
  return guarded([&] { s->impl->get_fields(u0, u1, u2, p); });
}
int nds_set_fields(nds_solver* s, const double* u0, const double* u1, const double* u2, const double* p) {
  if (!s) return fail(NDS_E_INVALID, "null solver");
  return guarded([&] { s->impl->set_fields(u0, u1, u2, p); });
}
int nds_simple_step_io(nds_solver* s, const double* u0_in, const double* u1_in, const double* u2_in,
                       const double* p_in, double* u0_out, double* u1_out, double* u2_out, double* p_out,
                       nds_iter_report* r) {
  if (!s) return fail(NDS_E_INVALID, "null solver");
  return guarded([&] {
    const double* in[4] = {u0_in, u1_in, u2_in, p_in};
    double* const out[4] = {u0_out, u1_out, u2_out, p_out};
    s->impl->step_io(in, out, r);
  });
}
void nds_solver_destroy(nds_solver* s) { delete s; }
int nds_solver_load_stage(nds_solver* s, const float* host_params, int count) {
  if (!s || !host_params || count != NDS_MPNN_NPARAM) return fail(NDS_E_INVALID, "nds_solver_load_stage: bad argument");
  return guarded([&] { s->impl->load_stage(host_params); });
}
int nds_solver_stage_graph(nds_solver* s, int32_t* nbr, float* ew, float* dscale) {
  if (!s) return fail(NDS_E_INVALID, "null solver");
  return guarded([&] { s->impl->stage_graph(nbr, ew, dscale); });
}
int nds_solver_pressure_pair(nds_solver* s, float* rhs, float* x) {
  if (!s) return fail(NDS_E_INVALID, "null solver");
  return guarded([&] { s->impl->pressure_pair(rhs, x); });
}
int nds_solver_apply_operator(nds_solver* s, const float* x, float* y) {
  if (!s || !x || !y) return fail(NDS_E_INVALID, "null argument");
  return guarded([&] { s->impl->apply_operator(x, y); });
}
int nds_solver_apply_operator_form(nds_solver* s, int form, const void* x, void* y) {
  if (!s || !x || !y) return fail(NDS_E_INVALID, "null argument");
  return guarded([&] { s->impl->apply_operator_form(form, x, y); });
}
int nds_solver_stage_counts(nds_solver* s, long long* applied, long long* fallbacks) {
  if (!s) return fail(NDS_E_INVALID, "null solver");
  return guarded([&] { s->impl->stage_counts(applied, fallbacks); });
}

unsigned long long nds_launch_count(void) { return nds::g_launches; }

}  // extern "C"

// ---------------------------------------------------------------------------
// Allocation-free continuity residual.
//
// Callers that may not allocate device memory -- code running between the
// steps of its own captured or real-time loop, or under an allocator that
// forbids cudaMalloc after start-up -- get the continuity residual of the
// solver's mesh for velocity vectors they own.  The partial sums of the
// continuity kernel go to a file-scope device array instead of a cudaMalloc'd
// buffer: at most kNoAllocBlocks blocks (the same 8 x 148 cap as the solver's
// own reductions), 16 KiB per device.  Every block overwrites its own slot
// and the reduction reads only the slots written by the same call, so
// nothing has to start at zero.  The array is shared by all calls on a
// device: calls that overlap in time (two host threads, or two streams
// without ordering between them) race on it.
//
// The array's device address is looked up (cudaGetSymbolAddress) on every
// call with the solver's device current: the lookup allocates nothing, and
// an address kept from an earlier call could be stale once the caller has
// torn the context down (cudaDeviceReset) and the module was loaded again.
// ---------------------------------------------------------------------------
namespace {
constexpr int kNoAllocBlocks = 1184;
constexpr int kNoAllocScratch = 2048;  // doubles; >= kNoAllocBlocks
static_assert(kNoAllocScratch >= kNoAllocBlocks, "scratch too small for the block cap");

__global__ void sqrt_in_place(double* x) { *x = sqrt(*x); }
}  // namespace

static __device__ __align__(256) double g_noalloc_part[kNoAllocScratch];

extern "C" {

int nds_continuity_noalloc(nds_solver* s, const double* u0, const double* u1, const double* u2, double* r,
                           double* norm, void* stream) {
  if (!s || !u0 || !u1 || !u2 || !r || !norm) return NDS_E_INVALID;
  const int32_t* ref = nullptr;
  const double *bco = nullptr, *fdiv = nullptr;
  int nc = 0, dev = 0;
  if (!s->impl->cell_arrays(&ref, &bco, &fdiv, &nc, &dev)) return NDS_E_INVALID;
  if (nc < 1 || dev < 0) return NDS_E_INVALID;
  const int grid = std::min(nds::grid_for(nc), kNoAllocBlocks);
  if (grid > kNoAllocScratch) return NDS_E_INVALID;
  int prev = -1;
  if (cudaGetDevice(&prev) != cudaSuccess) return NDS_E_CUDA;
  if (prev != dev && cudaSetDevice(dev) != cudaSuccess) return NDS_E_CUDA;
  int st = NDS_OK;
  double* part = nullptr;
  {
    void* a = nullptr;
    if (cudaGetSymbolAddress(&a, g_noalloc_part) == cudaSuccess) part = static_cast<double*>(a);
    else st = NDS_E_CUDA;
  }
  // every launch is checked with cudaPeekAtLastError, which leaves an error
  // pending from the caller's own earlier work in place for the caller
  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  if (st == NDS_OK) {
    nds::k::continuity<double, 1><<<grid, nds::kBlock, 0, cs>>>(nc, ref, bco, fdiv, u0, u1, u2, r, part);
    ++nds::g_launches;
    if (cudaPeekAtLastError() != cudaSuccess) st = NDS_E_CUDA;
  }
  if (st == NDS_OK) {
    nds::k::reduce_partials<1><<<1, nds::kBlock, 0, cs>>>(part, grid, norm);
    ++nds::g_launches;
    if (cudaPeekAtLastError() != cudaSuccess) st = NDS_E_CUDA;
  }
  if (st == NDS_OK) {
    sqrt_in_place<<<1, 1, 0, cs>>>(norm);
    ++nds::g_launches;
    if (cudaPeekAtLastError() != cudaSuccess) st = NDS_E_CUDA;
  }
  if (prev != dev) cudaSetDevice(prev);
  return st;
}

int nds_profile_enable(nds_solver* s, int on) {
  if (!s) return fail(NDS_E_INVALID, "null solver");
  return guarded([&] {
    s->impl->prof.collect();
    s->impl->prof.reset();
    s->impl->prof.on = on != 0;
  });
}
int nds_profile_read(nds_solver* s, nds_profile_entry* out, int max_entries, int* n_out) {
  if (!s || !out || !n_out) return fail(NDS_E_INVALID, "null argument");
  return guarded([&] {
    auto& P = s->impl->prof;
    P.collect();
    int n = 0;
    for (int c = 0; c < nds::P_NCAT && n < max_entries; ++c, ++n) {
      std::snprintf(out[n].name, sizeof(out[n].name), "%s", nds::kProfNames[c]);
      out[n].calls = P.calls[c];
      out[n].total_ms = P.total[c];
    }
    *n_out = n;
  });
}

}  // extern "C"
