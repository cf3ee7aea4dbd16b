// Internal declarations shared by the translation units of libsss.so.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <map>
#include <string>
#include <unordered_map>
#include <vector>

#include "sss.h"
#include "sss_lanes.h"
#include "sss_columns.h"
#include "sss_constant.h"
#include "sss_power.h"

namespace sss {

constexpr double kTau = 6.283185307179586;
constexpr int kMaxG = 8;      // generators per frame
constexpr int kMaxQ = 3;      // Gauss-Legendre nodes
constexpr int kMaxK = 6;      // exponentials per step
constexpr int kMaxCh = 4;     // coefficient channels
constexpr int kMaxSlots = kMaxQ * kMaxG;
constexpr int kMaxPhases = 6;  // lane counts of a prepared batch (8 .. 256)  // generator slots of a rotating plan (node, generator)
constexpr int kPlainMaxN = 52;  // dense shared-memory propagator path
// row-part kernels (forward and adjoint)
constexpr int kCloseMax = 8;    // close slots per lane
constexpr int kRing = 16;       // fine steps of coefficients per refill
// (C parts per lane, P entries per part) shapes instantiated
constexpr int kPartShapes[][2] = {{1, 4}, {2, 4}, {4, 4}, {2, 8}};
// slot-packed kernels: slots per lane (S <= kSlotsMax)
constexpr int kSlotsMax = 16;

void set_error(const std::string& msg);
int fail(int code, const std::string& msg);
int cuda_fail(cudaError_t e, const char* what);

#define SSS_CUDA(call)                                      \
    do {                                                    \
        cudaError_t e_ = (call);                            \
        if (e_ != cudaSuccess) return sss::cuda_fail(e_, #call); \
    } while (0)

// Lets `kern` be launched with as much dynamic shared memory as the device gives
// a block.  The limit belongs to the function and so to the whole process: every
// caller sets it to that maximum and none to its own launch's size, which would
// make a larger launch of another thread fail.
template <class Kern>
inline int allow_smem(Kern kern) {
    cudaFuncAttributes fa;
    int dev = 0, most = 0;
    SSS_CUDA(cudaFuncGetAttributes(&fa, kern));
    SSS_CUDA(cudaGetDevice(&dev));
    SSS_CUDA(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    most -= (int)fa.sharedSizeBytes;
    if (fa.maxDynamicSharedSizeBytes < most)
        SSS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    return 0;
}

// Device buffer that grows on demand and is owned by a plan.
struct DevBuf {
    void* p = nullptr;
    size_t bytes = 0;
    int ensure(size_t n);
    void release();
    template <class T> T* as() const { return static_cast<T*>(p); }
};

// Sparse form of the generators for the batched vector-action kernel:
// the union pattern of all generators, row-sorted.  For each pattern entry
// p: row, col, and the G generator values at (row, col).
struct SparseGenerators {
    int N = 0, G = 0, nnz = 0;
    std::vector<int> row_ptr;   // N+1
    std::vector<int> col;       // nnz
    std::vector<double> val;    // G*nnz, generator-major
};

// Host-side layout of the batched kernels: reachable rows, active
// generators, rows split across L lanes, per-lane entry lists.
struct BatchLayout {
    struct Ent { int col; int q; };   // compressed column, index into SparseGenerators
    int M = 0, Ga = 0, L = 0, E = 0, epl = 0, degree = 0, substeps = 0, threads = 0;
    bool use_reg = false;
    long nnz = 0;
    std::vector<int> active;                 // active generator indices
    std::vector<std::vector<Ent>> row_ents;  // per reachable row (reachable order)
    std::vector<std::vector<int>> lane_of;   // rows (reachable order) of each lane
    std::vector<int> newpos, row_orig;       // reachable -> lane order; lane order -> original
    std::vector<double> gv;                  // Ga*E*L generator values [g][e][l]
    std::vector<unsigned> words;             // E*L entry words [e][l]
    std::vector<int> entry_q;                // E*L index into SparseGenerators (-1: padding,
                                             // -2: partial add, -3: constant entry, value in cval)
    std::vector<double> cval;                // E*L constant entries' values (slot layouts)
    std::vector<int> cnt;                    // entries of each lane
    // row-part variant: C parts of P entries per lane, kc close slots
    bool parts = false;
    int C = 0, P = 0, kc = 0;
    std::vector<int> pcol;                   // C*P*L part entry columns [e][l]
    std::vector<unsigned> cw;                // kCloseMax*L close words [k][l]
    // slot-packed and phased row-part variants: S FMA slots per lane per
    // Horner term, kernel slot words in cw (load words [q][l], then store
    // words [S+q][l]), a barrier before slot bar_at, npart parked partial
    // sums per trajectory; phased: the shape index into kPhasedShapes
    bool slots = false, phased = false;
    int S = 0, bar_at = 0, npart = 0, shape = 0;
    std::vector<char> chan_const;            // per generator slot: its channel is batch-constant
    std::vector<double> chan_value;          // that constant
    std::vector<int> slot_chan;              // per generator slot: its program channel (-1: L0)
    // power-series variant: the series, its program, the varying generators
    // (active-generator indices), the power of two each coefficient is scaled
    // by, and the table of every exponential
    bool power = false;
    PowSeries ps;
    PowLayout pl;
    std::vector<int> pw_live;
    double pw_scale[kPowMaxLive] = {};
    std::vector<int> pw_tab;                 // [exponential << kMaxQ + code of the switched channel]
    // the switched channel of a forward pass of the adjoint, -1: none, and its
    // two values
    int pw_switch = -1;
    double pw_value[2] = {};
    // samples over which every live channel is constant (sss_constant.h): the
    // live program channels, the sets of their values, and the maps minus the
    // identity [set][hi, lo][column][row], rows in reachable order
    std::vector<int> cs_chan;
    std::vector<ConstSet> cs;
    std::vector<double> cs_map;
};

}  // namespace sss

struct sss_plan {
    sss_plan_desc d{};
    double W[sss::kMaxK * sss::kMaxQ] = {};
    double nodes[sss::kMaxQ] = {};
    bool rotating = false;
    int D = 0, S = 0;
    // host copies
    std::vector<double> gens;        // lab G*N*N, or rotating Q*G*N*N
    std::vector<double> dlast, slast, V, Vinv;
    sss::SparseGenerators sparse;    // lab frame, for sss_batch_run
    // device copies
    sss::DevBuf d_gens, d_dlast, d_slast, d_V, d_Vinv;
    sss::DevBuf d_sp_rowptr, d_sp_col;
    sss::DevBuf d_row_map;
    // workspace
    sss::DevBuf w_prop, w_in, w_out, w_prog, w_tab, w_aux, w_queue, w_ro,
        w_fin, w_samples, w_status;
    // health word of the prepared batch (see BatchArgs::health), reset by
    // sss_batch_prepare and by a check that found an error
    sss::DevBuf w_health;
    int last_launches = 0;
    int batch_lanes = 0;    // 0: chosen per run
    int batch_threads = 0;  // CTA size of the batched kernel, 0: 128
    int last_batch_lanes = 0, last_degree = 0, last_substeps = 0, last_rows = 0,
        last_nnz = 0, last_grid = 0, last_epl = 0, last_active = 0, last_variant = 0;
    // executed work of the last prepared batch (phase 0): generators assembled
    // per exponential, their non-zeros on the pruned pattern, FP64
    // instructions per Horner term per group; make_args records the first two
    int last_n_live = 0, last_live_nnz = 0, last_fp64_per_term = 0, mk_n_live = 0, mk_live_nnz = 0;
    // bank-aware renumbering of slot-programmed layouts: the modelled extra
    // shared-memory wavefronts of one Horner term (one group) before and
    // after, for the last layout built, and the numberings found so far
    // (keyed by a hash of the layout's kernel words)
    int last_bank_before = 0, last_bank_after = 0;
    // values of the constant entries of a slot layout being built: an entry
    // whose q is sparse.nnz + k has the fixed value slot_consts[k] and no
    // generator values (the G^T block of the adjoint's block series)
    std::vector<double> slot_consts;
    std::unordered_map<uint64_t, std::vector<int>> bank_cache;
    // row-kernel layouts found so far, by the pattern and configuration they
    // depend on (layout_key in sss_batch.cu): the cost at every lane count and
    // the layouts built, placed in their banks.  The search over lane counts
    // and packings takes 13 to 95 ms of host time and depends on nothing else,
    // so a sweep repeated on other programs of the same shape pays it once.
    struct LayoutMemo {
        double cost[sss::kLaneCounts] = {};
        bool costed = false;
        struct Built {
            sss::BatchLayout layout;
            int bank_before = 0, bank_after = 0;
        };
        std::map<int, Built> built;
    };
    std::map<std::vector<int>, LayoutMemo> layout_memo;
    // power series of large systems by the matrices they were made from: pattern,
    // constant parts, varying generators (1.6 ms of 16 cores at 171 rows and 5 ps;
    // new values of a laser or a drive's amplitude pay it)
    std::map<std::vector<double>, sss::PowSeries> series_memo;
    int big_resident[sss::kPowBigMaxCtas + 1] = {};   // clusters of so many CTAs the GPU holds (0: not asked yet)
    int batch_variant = 0;  // 0: register variant when it fits, 2: shared-memory variant,
                            // 3: one-chain register variant, 4: row-part variant
    int device = 0;
    int num_sms = 0;
    cudaEvent_t ev_begin = nullptr, ev_end = nullptr;  // around the last batched run's kernels
    bool ev_recorded = false;
    bool ev_keep_begin = false;  // a later phase of one run: keep the first launch's begin event
    int auto_lanes_ntraj = 0;    // trajectories the automatic lane rule counts (0: the batch)
    double auto_cost[sss::kLaneCounts] = {};  // last automatic layout: cost per lane count 8..256
    double auto_chain[sss::kLaneCounts] = {}; // and its chain figures (auto_lane_count)
    // a run by propagator columns being laid out or launched (sss_columns.cu):
    // its samples over all trajectories (0: not one) and its launches, which
    // record no timing events
    long cols_samples = 0;
    sss::ColumnsCut cols;
    // the inputs of the call on the host, where it has them (null: the layout
    // reads the device copies back)
    const double *host_rho0 = nullptr, *host_prog = nullptr;
    sss::DevBuf w_cols_tables, w_cols_queue;
    // the adjoint's forward pass being laid out on the power series: every
    // exponential's state is stored, and a channel of two values throughout the
    // programs (they cannot change before the launch) selects a table
    bool adj_forward = false;
    // constant samples of the batch being prepared, found for its first phase
    const sss::BatchLayout* phase_constants = nullptr;
    int launch_active = 0;       // trajectories with work in the next launch (0: the batch)
    // prepared batch (sss_batch_prepare -> sss_batch_launch): one kernel
    // layout per phase -- a single phase, or with uneven lengths and
    // automatic lanes one per widening lane count, phase k running from
    // output sample t_start on
    struct BatchPhase {
        alignas(16) unsigned char args[2048];
        size_t smem = 0;
        int L = 0, C = 0, P = 0, epl = 0, threads = 0, t_start = 0, S = 0, shape = 0;
        bool use_reg = false, one_chain = false, parts = false, shfl = false, slots = false,
             phased = false, power = false;
    };
    BatchPhase batch_phase[sss::kMaxPhases];
    sss::DevBuf batch_tables[sss::kMaxPhases];
    int batch_nphases = 0;
    std::vector<int> batch_longest;    // the prepared sample counts, longest first (or empty)
    const int* batch_order = nullptr;  // queue position -> trajectory, longest first (w_order)
    bool batch_ready = false, batch_empty = false, batch_has_rw = false, batch_table = false;
    int batch_ntraj = 0, batch_nch = 0, batch_nseg = 0, batch_F = 0;
    double batch_dt = 0.0;
    sss::DevBuf w_state;
    // adjoint (row-part path): forward and backward tables, stored states,
    // readouts, state buffer
    sss::DevBuf w_adjf, w_adjb, w_states, w_adjro, w_adjst, w_order;
    size_t adj_max_bytes = 0;  // stored-state memory of the adjoint, 0: half the free memory
    // equivalence-class (kernel) mode: states of n_full entries, image basis P
    // (n_full x N); unitary mode: operator generators of a u_n-level system
    // (N = 2 u_n), densities of u_nd entries (map u_map rows y, x, c, or all
    // 2 u_n^2 entries row-major)
    int n_full = 0;
    sss::DevBuf d_P;
    int u_n = 0, u_nd = 0;
    bool u_mapped = false;
    sss::DevBuf d_umap;
    // entries of one input state and of one output sample of sss_simulate
    int state_in() const { return n_full ? n_full : (u_n ? u_nd : d.N); }
};

namespace sss {
// sss_plain.cu
int plain_run(sss_plan* p, int ntraj, const double* d_rho0, int nch, int nseg,
              const double* d_prog, const double* d_tab, double t0, double dt,
              int T, int F, double* d_out, cudaStream_t st);
// sss_columns.cu: the same by propagator columns on the batched kernels
// (SSS_EINVAL: not for this plan, or no layout fits)
int columns_run(sss_plan* p, int ntraj, const double* h_rho0, const double* d_rho0, int nch, int nseg,
                const double* h_prog, const double* d_prog, const double* d_tab, double t0, double dt,
                int T, int F, double* d_out, cudaStream_t st);
// sss_batch.cu
int batch_run(sss_plan* p, int ntraj, const double* d_rho0, int nch, int nseg,
              const double* d_prog, const int* d_samples, const int* h_samples,
              double t0, double dt, int T_max, int F, const double* h_rw,
              double* d_readout, double* d_final, cudaStream_t st, double* d_trace = nullptr,
              const double* d_tab = nullptr);
int build_sparse(sss_plan* p);
// sss_adjoint.cu
// dch: the differentiated channel; npar: 2 (amplitude, phase) or 4 (also
// offset, frequency) gradient entries per segment
int adjoint_run(sss_plan* p, int ntraj, const double* d_rho0, int nch, int nseg,
                const double* d_prog, double t0, double dt, int T, int F, const double* h_rw,
                const double* h_tw, int dch, int npar, double* d_J, double* d_grad,
                cudaStream_t st);
// d_tab: a coefficient table (ntraj*(F*T_tab*Q)*G, rows (r*T_tab + t)*Q + k)
// in place of the programs; it runs on the row-part kernel
// h_samples: the trajectories' output-sample counts (host), or null; with
// them trajectories are handed out longest first and, with automatic lanes,
// the batch is prepared in phases
int batch_prepare(sss_plan* p, int ntraj, const double* d_rho0, int nch, int nseg,
                  const double* d_prog, double dt, int F, const double* h_rw, cudaStream_t st,
                  const double* d_tab = nullptr, int T_tab = 0, const int* h_samples = nullptr);
int batch_launch(sss_plan* p, double* d_state, const double* d_prog, const int* d_samples,
                 double t0, int t_begin, int n_samples, int T_max, double* d_readout,
                 cudaStream_t st, double* d_trace = nullptr, const double* d_tab = nullptr);
// Waits for the stream and reads the prepared batch's health word:
// SSS_ENONFINITE (and the word reset) if a launch since the last prepare or
// check wrote a NaN or infinite readout or final-state entry.
int batch_check(sss_plan* p, cudaStream_t st);
int build_layout(sss_plan* p, int ntraj, const double* d_rho0, int nch, int nseg,
                 const double* d_prog, double dt, int F, const std::vector<int>& force_active,
                 bool allow_register, BatchLayout* out, cudaStream_t st, bool force_parts = false,
                 const double* d_tab = nullptr, int T_tab = 0);
int slot_layout_host(int M, const int* row_ptr, const int* col, int L, int S_cap, int* S_out,
                     int* bar_out, int* npart_out, unsigned* words, int* entries);
// Slot-packed and phased row-part layouts of given rows (entries with q >=
// sparse.nnz are constant entries, see sss_plan::slot_consts), and the
// bank-aware placement of such a layout (varies[g]: generator slot g is
// assembled every exponential).
int slots_layout_rows(sss_plan* p, const std::vector<std::vector<BatchLayout::Ent>>& rows, int L,
                      int threads, int S_cap, const std::vector<int>& active,
                      const std::vector<int>& rows_reached, BatchLayout* out);
int phased_layout_rows(sss_plan* p, const std::vector<std::vector<BatchLayout::Ent>>& rows, int L,
                       int threads, int S_cap, const std::vector<int>& active,
                       const std::vector<int>& rows_reached, const std::vector<char>& varies,
                       BatchLayout* out);
int place_banks(sss_plan* p, BatchLayout& Ly, const std::vector<int>& active,
                const std::vector<char>& varies);
int parts_layout_rows(sss_plan* p, const std::vector<std::vector<BatchLayout::Ent>>& rows,
                      const std::vector<std::vector<char>>& prio, int L, int threads, int w_chain,
                      int w_close, const std::vector<int>& active,
                      const std::vector<int>& rows_reached, BatchLayout* out, int* nprio);
// Row-part forward kernel prepared outside the plan's batch state (for the
// adjoint): opaque kernel arguments and launch shape.
struct PartsForward {
    alignas(16) unsigned char args[2048];
    size_t smem = 0;
    int L = 0, C = 0, P = 0, threads = 0;
    bool power = false;   // the power-series kernels: E slots, RM merge slots, CTAs of a cluster
    int E = 0, RM = 0, ctas = 0;
};
// Build the device tables of a row-part layout into `tables` and the
// forward kernel's arguments.  Generators in `keep_live` are never folded
// into the constant part of Omega.
int parts_forward_prepare(sss_plan* p, const BatchLayout& Ly, int ntraj, int nch, int nseg,
                          double dt, int F, const double* h_rw, const std::vector<int>& keep_live,
                          DevBuf& tables, PartsForward* fw, cudaStream_t st);
// Launch it on `ntraj` trajectories (state in place, programs, readout
// (ntraj x T) or null, and optionally the state before every exponential:
// states[((b*T*F + n)*K + e)*M + row], rows in the layout's order).
int parts_forward_launch(sss_plan* p, const PartsForward& fw, int ntraj, double* d_state,
                         const double* d_prog, double t0, int T, double* d_readout,
                         double* d_states, cudaStream_t st);
}  // namespace sss
