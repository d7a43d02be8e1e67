// Kernel argument block, work schedule and per-state array layout shared by
// the evaluation kernels (pjg_wave.cuh, pjg_tile.cu), the schedule builder (pjg_sched.cu)
// and their host launcher (pjg_capi.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>
#include "pjg_tables.cuh"

enum { KIND_RATES = 0, KIND_JAC = 1, KIND_VJP = 2 };

// Two kernels: a thread per state (pjg_wave.cuh), for batches of several waves of
// resident blocks, and a block per tile of a few states (pjg_tile.cu).
#define PJG_BLOCK 128  // threads of a block of the former

// A block evaluates a tile of S = 2^slog states with W warps: lane % S is the
// state, and the 32 / S lane groups of a warp are workers (G = 32 W / S per
// block) that take different reactions, species and additions.
constexpr int kTileWarps = 8;
// Tile arrays (ns doubles per state, in shared memory; in the thread-per-state
// kernel's scratch before the vectors below):
enum {
    ARR_CONC = 0,  // concentrations c_k
    ARR_EP,        // exp(b_k), the reactant factor of 1 / Kc, where the state's
                   // |b| allow (StateVars::split); else the Gibbs function b_k
    ARR_EM,        // exp(-b_k), the product factor of 1 / Kc (split states)
    ARR_N_RATES,
    ARR_H = ARR_N_RATES,  // specific enthalpies (energies at constant volume)
    ARR_N_JAC,
    ARR_VT = ARR_N_JAC,   // J^T v: the weights vt_k
    ARR_N_VJP
};
__host__ __device__ constexpr int tile_arrays(int kind)
{
    return kind == KIND_RATES ? ARR_N_RATES : kind == KIND_JAC ? ARR_N_JAC : ARR_N_VJP;
}

// Per-state vectors of ns values in the block's slice of the scratch (L2):
// entry k of vector v at slice[(v ns + k) S + state]
enum {
    VEC_WDOT = 0,  // net molar production rates (sums over reactions)
    VEC_CP,        // specific heats
    VEC_H,         // specific enthalpies (energies at constant volume)
    VEC_N_RATES,
    VEC_DCP = VEC_N_RATES,  // d cp_k / dT
    VEC_NS,        // Jacobian: bath-gas terms of each species row, the same in every
                   // species column; J^T v: the species columns' sums
    VEC_N_VJP,
    VEC_RT = VEC_N_VJP,  // row T of the species columns, sum_k hw_k J_kj
    VEC_RE,        // row E of them, sum_k (1 - W_k / W_ns) J_kj
    VEC_CT,        // column T of the species rows
    VEC_CE,        // column E of them
    VEC_N_JAC      // then the third-body sums (Schedule)
};
__host__ __device__ constexpr int vec_arrays(int kind)
{
    return kind == KIND_RATES ? VEC_N_RATES : kind == KIND_VJP ? VEC_N_VJP : VEC_N_JAC;
}

// Targets of additions: a slot of the Jacobian, or with TGT_VEC an entry of
// the scratch slice (vector * ns + k); TGT_FIRST marks the first addition to
// the target, which stores.
constexpr unsigned TGT_FIRST = 1u << 31, TGT_VEC = 1u << 30, TGT_MASK = TGT_VEC - 1;
// A worker's additions of a batch come in runs of one kind, so that the loops
// over them test nothing per item: targets x (without flags) and source words
// y = byte offset of the term in the buffer (18 bits) | sign << 31; products
// hold the second term's distance (in terms, signed) in bits 20..30, the
// general run an integer factor there (signed) and the targets' flags.  Each
// run is a multiple of kItemUnroll items: stores repeat the last one, additions
// are padded with term 0, which is zero (to the last slot, or to the slice's
// last entry, which nothing reads).
enum { RUN_SLOT_FIRST = 0, RUN_VEC_FIRST, RUN_SLOT, RUN_VEC, RUN_PROD_FIRST, RUN_PROD, RUN_GENERAL, RUN_N };
constexpr int kItemUnroll = 4;
// items of a worker that are staged in shared memory at a time
__host__ __device__ constexpr int item_stage(int slog) { return slog >= 4 ? 64 : slog == 3 ? 48 : slog >= 1 ? 32 : 24; }
__host__ __device__ inline int item_q(unsigned y) { return (int)(y << 1) >> 21; }
constexpr unsigned kItemOff = 0x3ffff;

struct PostItem {  // target += coef * vec[src], after the reactions
    unsigned src, target;
    double coef;
};

struct Schedule {  // device tables of one (kind, output layout, S)
    // warps: read by the kernel, whose code for a constant ran the 500-species
    // Jacobian in 14.02 ms against 13.83
    int slog = 5, warps = kTileWarps, rounds = 1, n_batch = 0, buf_terms = 0;
    int n_vec = 0;                 // entries of the scratch slice per state
    const int4* tasks = nullptr;         // n_batch * rounds * W: class, first reaction, count
    const int* term_off = nullptr;       // per reaction: its terms in the batch's buffer
    const int* item_off = nullptr;       // the RUN_N runs of each worker of each batch
    const uint2* items = nullptr;
    const int* post_off = nullptr;       // G + 1
    const PostItem* post = nullptr;
};

// terms a reaction leaves in the batch's buffer, in this order
//   rates:    net
//   J^T v:    net, w g_j per participant, [w X]
//   Jacobian: w_T, net, d0, g_j per participant, [ns], [d1], [X], [w_E]
// ([..] where has_ns, has_d1, a third body, RX_WEREAL); X of a third-body list
// that several reactions share is summed over them, the list's coefficients
// multiply the sums; else one term per entry of the list, coefficient times X
template <class R>
__host__ __device__ inline int rxn_x_terms(const R& r)
{
    return RX_THD(r.flags) == THD_NONE ? 0 : r.list >= 0 ? 1 : r.thd_cnt;
}
__host__ __device__ inline bool rxn_has_d1(int flags) { return !(flags & RX_E22) || (flags & RX_HASNS); }

// The sums over species: this many workers take every parts-th species each,
// then their partial sums are added in order, in both kernels (so their order
// depends on the mechanism alone).  One for small mechanisms, where the eight
// additions would cost more than they spread (H2/O2 Jacobian 437 -> 420 us).
constexpr int kParts = 8;
__host__ __device__ constexpr int sum_parts(int ns) { return ns < 24 ? 1 : kParts; }

// tables of the thread-per-state kernel for one (kind, output layout)
struct WaveTables {
    const int* slot_off = nullptr;    // per reaction:
    const unsigned* slots = nullptr;  // per participant, its slots by participant and by entry of
                                      // an unshared third-body list (TGT_FIRST marked, TGT_MASK none)
    const int* tb_off = nullptr;      // per reaction with a shared third-body list:
    const int* tb = nullptr;          // its sums (Jacobian: per participant, rows T and E; J^T v: one)
    const PostItem* post = nullptr;
    const unsigned* zero = nullptr;   // species-block slots that nothing is added to
    int n_post = 0, n_zero = 0;
};

struct EvalArgs {
    // mechanism
    const RxnRec* rxn;
    const double* sp;
    const int* thd_spec;
    const double* thd_coef;
    const double* aux;
    int ns, nr;
    // 690 / (largest sum |nu| of a reversible reaction), at most 138: the bound
    // on every |b_k| of a state for the per-species factors of 1 / Kc
    double kc_split_max;
    int need_logP;
    int jac_approx;  // 'approximate' Jacobian type: no bath-gas terms in the species columns
    // third-body lists that several reactions share: offset and length in
    // thd_spec / thd_coef, default efficiency (0 or 1), whether ln [M] is needed
    const int4* m_lists;
    int n_m;
    int cls_off[16];  // the packed records' classes: [cls_off[c], cls_off[c + 1]), 15 of them
    Schedule sc;
    WaveTables wt;
    // states
    int64_t n;  // states in this launch
    int conp;
    const double* param;
    const double* phi;
    int64_t phi_ss, phi_sj;  // element (s, j) at phi[s * phi_ss + j * phi_sj]
    double* dphi;            // optional
    int64_t dphi_ss, dphi_sj;
    // tile: one slice of sc.n_vec * S doubles per block; thread per state: array
    // a, entry k, state s at scratch[(a * ns + k) * sc_ld + s], arrays then vectors
    double* scratch;
    int64_t sc_ld;
    // Jacobian: acc[slot * acc_ld + s * acc_ss]
    double* acc;
    int64_t acc_ld, acc_ss;
    const int* ns_rows;   // species rows with bath-gas terms
    const int* ns_slots;  // ns - 1 slots of each of them (-1 none)
    int n_ns;
    const int* sp_slots;  // 2 per species row: slot(k, T), slot(k, E)
    const int* cj_slots;  // 2 per species column: slot(T, j), slot(E, j)
    int s00, s01, s10, s11;
    // patterns that leave out a term of the species block (col_list null
    // otherwise): rows T and E are summed over the stored entries
    const int* col_off;    // ns
    const int2* col_list;  // (species row k, slot)
    // third-body lists' bath-gas coefficients, for J^T v: vNS += ns_coef * vec[ns_src]
    const PostItem* ns_post;
    int n_ns_post;
    // vector-Jacobian product
    const double* v;  // v[s * phi_ss + j * phi_sj]
    double* vjp;      // same layout
};

struct SchedInput {
    int kind = 0, ns = 0, jac_approx = 0;
    const std::vector<RxnRec>* rxn = nullptr;  // device records
    const std::vector<int>* cls = nullptr;     // class of each
    const std::vector<int>* thd_spec = nullptr;
    const std::vector<double>* thd_coef = nullptr;
    const std::vector<int>* slot = nullptr;    // (ns-1)^2 species-block slots, -1 none (Jacobian)
};
// The additions of one (kind, output layout), whatever the tile's shape, and
// the tables of the thread-per-state kernel (WaveTables).
struct SchedAdds {
    struct Item {
        unsigned target;
        int t, q;  // term of the reaction; factor, or the second term's distance
        bool prod;
    };
    int kind = 0, n_slot = 0, n_vec = 0;
    unsigned unread = 0;
    bool left_out = false;           // a term of the species block has no slot
    std::vector<int> cls, terms, item_off;  // per reaction: class, terms left in the buffer, items
    std::vector<Item> items;
    std::vector<unsigned> zeros;     // targets that nothing is added to
    std::vector<char> general;       // targets with a factor other than 1 and -1 (empty: none)
    std::vector<int> count, order;   // additions per target; targets, longest first
    std::vector<PostItem> post, ns_post;
    std::vector<int> wave_slot_off, wave_tb_off, wave_tb;
    std::vector<unsigned> wave_slots, wave_zero;
    int dense(unsigned t) const { return (int)(t & TGT_MASK) + ((t & TGT_VEC) ? n_slot : 0); }
};
struct SchedHost {  // one shape's tables before upload
    int n_batch = 0;
    std::vector<int4> tasks;
    std::vector<int> term_off, item_off, post_off;
    std::vector<uint2> items;
    std::vector<PostItem> post;
};
void sched_adds(const SchedInput& in, SchedAdds& out);
// false: a reaction's terms pass the buffer
bool sched_build(const SchedAdds& in, int slog, int rounds, int buf_terms, SchedHost& out);

// host launchers: pjg_tile.cu
constexpr size_t kTileStatic = 8192 + 256;  // exp table and flags, bytes
inline size_t stage_bytes(int slog) { return (size_t)kTileWarps * (32 >> slog) * item_stage(slog) * 8; }
constexpr int kTileSmemMax = 227 << 10;
size_t pjg_tile_smem(int kind, int ns, int n_m, int slog, int buf_terms);
int pjg_launch_tile(const EvalArgs& a, int kind, int grid, void* stream);
// resident blocks per SM of the kernels of `kind`
int pjg_tile_blocks_per_sm(int kind, size_t smem);
// pjg_eval.cu
int pjg_wave_blocks_per_sm(int kind, bool large);
// large: of a mechanism whose tiles are smaller than 32 states
int pjg_launch_wave(const EvalArgs& a, int kind, int sms, bool large, void* stream);
extern thread_local cudaError_t pjg_launch_err;  // of this thread's last evaluation launch
const char* pjg_launch_error_string();           // CUDA's description of it
int pjg_fp64_probe(int blocks, int threads, int iters, double* out, void* stream);
int pjg_launch_fexp(const double* x, double* y, int64_t n, void* stream);
int pjg_launch_chem_utils(const double* sp, int ns, int64_t n, int conp, const double* phi,
                          int64_t phi_ss, double* cp, double* h, double* b, int64_t out_ss,
                          int64_t out_sk, void* stream);
int pjg_launch_transpose(const double* src, int64_t ld, int64_t n, int nslot, double* dst,
                         void* stream);
