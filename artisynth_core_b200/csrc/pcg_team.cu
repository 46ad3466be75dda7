// pcg_team.cu -- block-Jacobi PCG with one team of CTAs per model.
//
// pcg.cu runs every model of the pack through one grid-wide loop: each
// iteration ends at a barrier of the whole grid, then reads the partial dot
// products and gathers the search direction, three dependent L2 round trips
// (5 us per iteration on the 40x10x10 hex beam whose arithmetic takes well
// under one).  Here a model's rows are dealt to a team of k CTAs, a compact
// set of rows each (recursive bisection of the node positions), and
//   * the CTA's blocks of S stay in registers and shared memory for the whole
//     solve (what exceeds them is streamed from a copy in the order the lanes
//     read it) and the PCG vectors in the registers of the lanes that own them;
//   * there is no grid barrier: every value that crosses CTAs travels in a
//     16-byte packet with a tag, written and read in one 128-bit access, so
//     the reader polls the datum itself and one L2 round trip carries both the
//     value and the synchronisation.  A reader waits for the rows next to its
//     own and for the team's k partial sums, nothing else;
//   * models run independently of one another: teams form from a queue of
//     slots (longest expected solves first), so a slow model occupies its own
//     CTAs instead of keeping the grid in its loop.
// Measured, grid-wide kernel -> this one, PCG per iteration: 40x10x10 hex beam
// 5.2 -> 2.7 us, 90-row beam 4.5 -> 1.3, 1,958-row quadratic beam 6.9 -> 2.2,
// 2,376-row NODAL block 9.4 -> 4.3, 60x30x30 NODAL block 43 -> 15 (FP64) and 36
// -> 14 (mixed); 256 uneven beams 11.5 -> 2.4 ms per solve.
// The recurrences, tests, restarts and results are those of pcg.cu's kernel
// (pipelined CG of Ghysels & Vanroose 2014, then classic PCG after a
// residual replacement); sums are formed in a fixed order, so results are
// bit-reproducible whatever the order in which teams form.  The size of a
// model's team goes by the pack's models: alone and packed it agrees to
// rounding.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <numeric>
#include <system_error>
#include <thread>
#include <type_traits>

#include "device_math.cuh"
#include "engine.h"

namespace b200fem {

namespace {

constexpr int kTeamThreads = 512;
constexpr int kTeamWarps = kTeamThreads / 32;
// the last warp collects the team's partial sums and forms the scalars while
// the others fetch the neighbouring rows and run the SpMV
constexpr int kRowWarps = kTeamWarps - 1;
constexpr int kRowThreads = kRowWarps * 32;
// Vector components: lanes 0..29 of a row warp own the three components of
// ten rows (a row never straddles a warp, so its w reaches m = Dinv w by
// shuffles), in up to kMaxSets sets of kSetRows rows.
constexpr int kSetRows = kRowWarps * 10;
constexpr int kMaxSets = 3;
// steps of a lane's first row group whose blocks stay in its registers
__host__ __device__ constexpr int reg_blocks(int sets, bool dil) { return sets == 1 ? (dil ? 1 : 2) : 0; }
constexpr int kWantRows = 46, kWantTeam = 80, kAloneRows = 96;  // see plan_team
constexpr double kExchangeRows = 165, kSetupRows = 3000, kFill = 0.95;  // see plan_team
constexpr int kRowWeight = 8;  // a row's vectors, in blocks
constexpr int kTeamMaxRestarts = 10;  // as in pcg.cu
constexpr int kTeamRoundCap = 400;    // as in pcg.cu

struct TeamArgs {
  const TeamSlot* slots;
  int n_slots;
  unsigned long long* ticket;
  const int* rows;         // slot-major: the global rows each slot owns (most blocks first)
  const unsigned char* pub;  // per owned row: some other CTA reads it
  const int* diag;         // per owned row: its diagonal block in S
  const int* halo;         // slot-major: the global rows of other slots that the slot reads
  const int4* group;       // slot-major: the row groups (RowGroup)
  const int* blk;          // per step and lane: the block of S (-1: none)
  const unsigned short* cl;  // per step and lane: its column as a local index (owned, then halo)
  const int* g1;           // factored NODAL, per step and lane: divBlk slots of d_row(col) and d_col(row) (-1 none)
  const int* g2;
  unsigned char* stream;   // steps beyond a slot's shared memory
  const void* S;
  const double* b;
  double* x;
  const double* step;
  double tol_override;
  double* model_out;
  int* flags;
  unsigned long long timeout_ns;
  int skip_cta;
  int max_iter, variant, update_state;
  int n_rows;
  unsigned* base;   // per model: packets tags used so far
  double* row_pk;   // [2][n_rows] two packets (32 bytes) each
  double* part_pk;  // [2][n_slots] two packets each
  double* t_pk;     // [2][n_rows] one packet each (factored NODAL)
  double *xpos, *vel, *vprev, *vprev2, *vprev3, *vprev4;
  const int* act_node;
  const int* model_active;
  const double* row_nrm;
  const double* row_off;
  const double* divblk;
  const double* node_kp;
};

// One packet: 96 bits of data and a 32-bit tag, moved as one 128-bit access
// (single-copy atomic for the .b128 type), so a reader that sees the tag sees
// the data.  Three doubles travel as two packets, one 32-byte sector: packet 0
// holds the first double and the high half of the third, packet 1 the second
// double and the low half of the third.
__device__ __forceinline__ void put_packet(double* slot, double v, unsigned half, unsigned tag) {
  const unsigned long long hi = ((unsigned long long)tag << 32) | half;
  asm volatile(
      "{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }"
      :
      : "l"(slot), "l"((unsigned long long)__double_as_longlong(v)), "l"(hi)
      : "memory");
}
__device__ __forceinline__ double get_packet(const double* slot, unsigned& half, unsigned& tag) {
  unsigned long long lo, hi;
  asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
               : "=l"(lo), "=l"(hi)
               : "l"(slot)
               : "memory");
  half = (unsigned)hi;
  tag = (unsigned)(hi >> 32);
  return __longlong_as_double((long long)lo);
}
__device__ __forceinline__ unsigned long long team_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// The bound of a poll: every 64 tries the wait ends when another CTA has
// recorded an error or the time limit has passed; the latter records
// B200FEM_ERR_TIMEOUT.  The limit is for waits between running CTAs, so it
// counts from the first check that finds the team complete: its first members
// may have to wait until other CTAs end whole solves of earlier models.  That
// wait ends with those solves, whose own waits are limited (teams form in
// ticket order, so only the last one is incomplete); kFormNs bounds it should
// a CTA be lost.
constexpr unsigned long long kFormNs = 60000000000ull;
struct PollBound {
  const TeamArgs& a;
  const TeamSlot& sl;
  const uint64_t& ticket0;  // the launch's first ticket
  unsigned long long t0 = 0;
  unsigned n = 0;
  bool formed = false;
  __device__ __forceinline__ PollBound(const TeamArgs& a, const TeamSlot& sl, const uint64_t& ticket0)
      : a(a), sl(sl), ticket0(ticket0) {}
  __device__ __forceinline__ bool give_up() {
    if ((++n & 63u) != 0) return false;
    if (*(volatile int*)a.flags != 0) return true;
    const unsigned long long now = team_ns();
    if (!formed && *(volatile unsigned long long*)a.ticket - ticket0 >= (unsigned long long)(sl.s0 + sl.k)) {
      formed = true;
      t0 = now;
    } else if (t0 == 0) {
      t0 = now;
    } else if (now - t0 > (formed ? a.timeout_ns : kFormNs)) {
      atomicExch(a.flags, B200FEM_ERR_TIMEOUT);
      return true;
    }
    return false;
  }
};

// Bytes of one step of a warp, value by value across the 32 lanes, so that its
// loads are contiguous and free of bank conflicts: the lanes' blocks of S
// (and, factored NODAL, d_row(col)), and d_col(row), which the product's second
// half reads.
__host__ __device__ constexpr int step_bytes(int mt_bytes, bool dil) { return 32 * (9 * mt_bytes + (dil ? 24 : 0)); }
constexpr int kStep2 = 32 * 24;
__host__ __device__ inline size_t team_align(size_t b) { return (b + 15) & ~(size_t)15; }
// shared memory of one slot; the steps of S kept there come last
struct TeamLayout {
  size_t xs, sn, ts, ckp, halo, group, cl, G2, S;
};
__host__ __device__ inline TeamLayout team_layout(int nloc, int nh, int steps, int groups, bool dil) {
  TeamLayout o;
  size_t p = 0;
  o.group = p;
  p += (size_t)groups * sizeof(int4);
  o.xs = p;
  p += team_align((size_t)(nloc + nh) * 3 * sizeof(double));
  o.sn = p;
  p += team_align((size_t)nloc * (dil ? 6 : 3) * sizeof(double));
  o.ts = p;
  if (dil) p += team_align((size_t)(nloc + nh) * sizeof(double));
  o.ckp = p;
  if (dil) p += team_align((size_t)nloc * sizeof(double));
  o.halo = p;
  p += team_align((size_t)nh * sizeof(int));
  o.cl = p;
  p += team_align((size_t)steps * 32 * sizeof(unsigned short));
  o.G2 = p;
  if (dil) p += (size_t)steps * kStep2;
  o.S = p;
  return o;
}
// A row group: the rows one warp walks together, 32 >> log lanes each of 1 << log
struct RowGroup {
  int shape;  // steps | log << 16 | (rows - 1) << 24
  int step;   // its first step
  int mem;    // its first step of S in memory (the register steps take none)
  int row;    // its first local row
  __device__ __forceinline__ int steps() const { return shape & 0xffff; }
  __device__ __forceinline__ int log() const { return (shape >> 16) & 255; }
  __device__ __forceinline__ int rows() const { return (shape >> 24) + 1; }
};

__device__ __forceinline__ void row_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kRowThreads) : "memory"); }

// Warp sums of three values in five levels: the first two levels also halve
// the number of values a lane carries (6 double shuffles instead of 15).
// Afterwards lanes 0-7 hold the sum of a, 8-15 of b, 16-23 of c.
__device__ __forceinline__ double team_sum3(double a, double b, double c, int lane) {
  const bool h16 = lane & 16, h8 = lane & 8;
  double k0 = h16 ? c : a, k1 = h16 ? 0.0 : b;
  k0 += __shfl_xor_sync(0xffffffffu, h16 ? a : c, 16);
  k1 += __shfl_xor_sync(0xffffffffu, h16 ? b : 0.0, 16);
  double v = (h8 ? k1 : k0) + __shfl_xor_sync(0xffffffffu, h8 ? k0 : k1, 8);
  v += __shfl_xor_sync(0xffffffffu, v, 4);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v;
}

enum { kRun = 0, kConverged = 1, kStop = 2 };

// The state update of a step for packs: one launch after every model's solve
// ended without an error (a single model updates its state in the PCG).
__global__ void team_state_kernel(int R, const int* __restrict__ act_node, const int* __restrict__ row_model,
                                  const double* __restrict__ step, const double* __restrict__ sol,
                                  double* __restrict__ x, double* __restrict__ vel, double* __restrict__ vprev,
                                  double* __restrict__ vprev2, double* __restrict__ vprev3,
                                  double* __restrict__ vprev4, const int* __restrict__ active,
                                  const double* __restrict__ row_nrm, const double* __restrict__ row_off,
                                  const int* __restrict__ flags) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= R || flags[0] != 0) return;
  const int m = row_model[row];
  if (active && !active[m]) return;
  const int n = act_node[row];
  const double h = step[(size_t)m * 8];
  double xn[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const size_t q = 3 * (size_t)n + c;
    const double vn = sol[3 * (size_t)row + c];
    vprev4[q] = vprev3[q];
    vprev3[q] = vprev2[q];
    vprev2[q] = vprev[q];
    vprev[q] = vel[q];
    vel[q] = vn;
    xn[c] = x[q] + h * vn;
  }
  if (row_nrm) {
    const double* q = row_nrm + 3 * (size_t)row;
    const double dist = q[0] * xn[0] + q[1] * xn[1] + q[2] * xn[2] - row_off[row];
#pragma unroll
    for (int c = 0; c < 3; c++) xn[c] -= q[c] * dist;
  }
#pragma unroll
  for (int c = 0; c < 3; c++) x[3 * (size_t)n + c] = xn[c];
}

// SETS: component sets (rows <= SETS * kSetRows); DIL: the factored NODAL
// matrix.
template <typename MT, int SETS, bool DIL>
__global__ void __launch_bounds__(kTeamThreads, 1) pcg_team_kernel(TeamArgs a) {
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ double s_part[kRowWarps][3];
  __shared__ double s_al, s_be;
  __shared__ int s_code, s_abort;
  __shared__ int s_ticket;
  __shared__ uint64_t s_ticket0;  // the launch's first ticket
  __shared__ TeamSlot s_slot;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const bool red = warp == kRowWarps;
  if (t == 0) s_abort = 0;

  for (bool start = true;; start = false) {
    // next slot; a launch draws n_slots + gridDim tickets in all (one past
    // the end per CTA), so the counter needs no reset between launches.
    // After an error of an earlier launch of the call nothing runs.  One
    // thread reads the error word and all go by its ticket: other CTAs write
    // the word while this one starts, and a CTA whose warps saw different
    // values would wait for those that have left.
    if (t == 0) {
      s_ticket = a.n_slots;
      if (!start || *(volatile int*)a.flags == 0) {
        const unsigned long long drawn = atomicAdd(a.ticket, 1ull);
        s_ticket = (int)(drawn % ((unsigned long long)a.n_slots + gridDim.x));
        s_ticket0 = drawn - s_ticket;
      }
    }
    __syncthreads();
    const int si = s_ticket;
    __syncthreads();
    if (si >= a.n_slots) return;
    // (in shared memory: the iterations need few of its fields, the registers
    // are for the vectors and the matrix)
    if (t == 0) s_slot = a.slots[si];
    __syncthreads();
    const TeamSlot& sl = s_slot;
    if (a.model_active && !a.model_active[sl.model]) {
      if (sl.rank == 0 && t == 0) {
        double* o = a.model_out + (size_t)sl.model * 4;
        o[0] = 0;
        o[1] = 0;
        o[2] = 1.0;
      }
      continue;
    }
    const int nloc = sl.nloc, nh = sl.nh, k = sl.k;
    // tags continue from the model's last solve: a packet left by it never
    // carries a tag of this one
    const unsigned tag0 = a.base[sl.model];
    const double* sp = a.step + (size_t)sl.model * 8;
    constexpr int kReg = reg_blocks(SETS, DIL), kStep = step_bytes((int)sizeof(MT), DIL);
    const int ng = sl.groups;
    const TeamLayout lay = team_layout(nloc, nh, sl.steps, ng, DIL);
    double* const xs = (double*)(dyn + lay.xs);
    double* const sn = (double*)(dyn + lay.sn);
    double* const ts = (double*)(dyn + lay.ts);
    double* const ckp = (double*)(dyn + lay.ckp);
    int* const hrow = (int*)(dyn + lay.halo);
    RowGroup* const grp = (RowGroup*)(dyn + lay.group);
    unsigned short* const cl = (unsigned short*)(dyn + lay.cl);
    unsigned char* const Ss = dyn + lay.S;
    double* const g2s = (double*)(dyn + lay.G2);
    unsigned char* const Sg = a.stream + (size_t)sl.stream0 * kStep;  // steps from sl.steps_smem on
    // the warp's row group of a pass (alternating direction: the groups get
    // shorter), -1 beyond the last
    auto group_of = [&](int pass) {
      const int g = pass * kRowWarps + ((pass & 1) ? kRowWarps - 1 - warp : warp);
      return g < ng ? g : -1;
    };
    const int passes = (ng + kRowWarps - 1) / kRowWarps;

    // ---- the slot's tables and starting vector to shared memory
    for (int i = t; i < nh; i += kTeamThreads) hrow[i] = a.halo[sl.h0 + i];
    for (int i = t; i < ng; i += kTeamThreads) ((int4*)grp)[i] = a.group[sl.g0 + i];
    for (int i = t; i < sl.steps * 16; i += kTeamThreads)
      ((unsigned*)cl)[i] = ((const unsigned*)(a.cl + (size_t)sl.w0 * 32))[i];
    for (int i = t; i < nloc + nh; i += kTeamThreads) {
      const int r = i < nloc ? a.rows[sl.r0 + i] : a.halo[sl.h0 + i - nloc];
#pragma unroll
      for (int c = 0; c < 3; c++) xs[3 * i + c] = a.x[3 * (size_t)r + c];
      if constexpr (DIL) {
        const double v = (sp[0] * sp[0] + sp[0] * sp[2]) * a.node_kp[a.act_node[r]];
        ts[i] = v;  // until the first product: kp of the neighbours for the block diagonal
        if (i < nloc) ckp[i] = v;
      }
    }
    __syncthreads();

    if ((int)blockIdx.x == a.skip_cta) {
      // failure-detection test: this CTA never publishes; it waits for
      // itself, bounded like every other wait, and the team's waits run out
      if (t == 0) {
        PollBound pb(a, sl, s_ticket0);
        while (!pb.give_up()) {
        }
      }
      return;
    }

    const double tol = a.tol_override > 0 ? a.tol_override : sp[6];
    // Two roles with the same sequence of CTA barriers per phase: B ends the
    // SpMV and makes the scalars known, C hands the per-warp dot products to
    // the reducing warp, D (classic PCG, true residual) makes a scalar known
    // that depends on C's.  E follows where a role would otherwise go on to
    // write what the other may not have read yet: the reducing warp s_code
    // of a restart's first iteration, a row warp s_abort in its next poll.
    if (red) {
      double sums[3] = {0, 0, 0};
      unsigned pe = 0;  // partial sums published
      const int nw = min(kRowWarps, (nloc + 9) / 10);
      // after C: the CTA's sums, published as the slot's partials
      auto publish = [&]() {
        double v0 = 0, v1 = 0, v2 = 0;
        if (lane < nw) {
          v0 = s_part[lane][0];
          v1 = s_part[lane][1];
          v2 = s_part[lane][2];
        }
        const double v = team_sum3(v0, v1, v2, lane);
        sums[0] = __shfl_sync(0xffffffffu, v, 0);
        sums[1] = __shfl_sync(0xffffffffu, v, 8);
        sums[2] = __shfl_sync(0xffffffffu, v, 16);
        if (k > 1 && lane < 2)
          put_packet(a.part_pk + ((size_t)(pe & 1) * a.n_slots + sl.s0 + sl.rank) * 4 + 2 * lane,
                     lane ? sums[1] : sums[0],
                     lane ? (unsigned)__double2loint(sums[2]) : (unsigned)__double2hiint(sums[2]), tag0 + pe + 1);
        pe++;
      };
      // the team's sums of the last publish (a team of one has them): lane
      // pairs take the two packets of a slot
      auto collect = [&]() {
        if (k == 1) return;
        const double* buf = a.part_pk + ((size_t)((pe - 1) & 1) * a.n_slots + sl.s0) * 4 + 2 * (lane & 1);
        const unsigned tag = tag0 + pe;
        PollBound pb(a, sl, s_ticket0);
        double m = 0, r = 0;
        auto round = [&](auto width, int qb) {
          constexpr int U = decltype(width)::value;
          double v[U];
          unsigned hf[U];
          for (;;) {
            bool all = true;
#pragma unroll
            for (int u = 0; u < U; u++) {
              const int q = qb + 16 * u + (lane >> 1);
              v[u] = 0;
              hf[u] = 0;
              if (q < k) {
                unsigned g;
                v[u] = get_packet(buf + (size_t)q * 4, hf[u], g);
                all &= g == tag;
              }
            }
            if (__all_sync(0xffffffffu, all)) break;
            if (__any_sync(0xffffffffu, pb.give_up())) {
              s_abort = 1;
              break;
            }
          }
#pragma unroll
          for (int u = 0; u < U; u++) {
            m += v[u];
            const unsigned o = __shfl_xor_sync(0xffffffffu, hf[u], 1);
            // (meaningful in the even lanes)
            r += __hiloint2double((int)hf[u], (int)o);
          }
        };
        if (k <= 16) round(std::integral_constant<int, 1>{}, 0);
        else if (k <= 48) round(std::integral_constant<int, 3>{}, 0);
        else
          for (int qb = 0; qb < k; qb += 160) round(std::integral_constant<int, 10>{}, qb);
        if (lane & 1) r = 0;
#pragma unroll
        for (int off = 16; off > 1; off >>= 1) {
          m += __shfl_xor_sync(0xffffffffu, m, off);
          r += __shfl_xor_sync(0xffffffffu, r, off);
        }
        sums[0] = __shfl_sync(0xffffffffu, m, 0);
        sums[1] = __shfl_sync(0xffffffffu, m, 1);
        sums[2] = __shfl_sync(0xffffffffu, r, 0);
      };
      double bb = 0, thr2 = 0, gold = 1, rga = 0, rg = 0, rho = 0, rel = 0;
      int iters = 0, total_it = 0;
      bool first = true, conv = false, have_bb = false, ok = false, classic = a.variant == 1;
      auto norms = [&]() {  // ||b|| of P0, once
        if (have_bb) return;
        collect();
        bb = sums[0];
        thr2 = tol * tol * bb;
        have_bb = true;
      };
      __syncthreads();  // C of P0
      publish();
      for (int restart = 0;; restart++) {
        if (classic) {
          norms();
          rho = sums[1];
          // (on a restart the residual has just missed the tolerance, though
          // its square may round to thr2: an iteration is due)
          conv = restart == 0 && (sums[2] <= thr2 || sums[2] == 0.0);
          first = true;
          for (int it = 0;; it++) {
            if (it > 0) {
              collect();
              gold = rho;
              rho = sums[0];
              iters++;
              conv = sums[1] <= thr2 || sums[1] == 0.0;
            }
            const int code = conv ? kConverged
                             : (total_it + it >= a.max_iter || (a.variant == 0 && it >= kTeamRoundCap)) ? kStop
                                                                                                       : kRun;
            if (lane == 0) {
              s_be = first ? 0.0 : rho / gold;
              s_code = code;
            }
            first = false;
            __syncthreads();  // B
            if (s_abort) return;
            if (code != kRun) {
              total_it += it;
              break;
            }
            __syncthreads();  // C: p.q
            publish();
            collect();
            if (lane == 0) s_al = rho / sums[0];
            __syncthreads();  // D
            if (s_abort) return;
            __syncthreads();  // C: r.z, r.r
            publish();
          }
        } else {
          norms();
          first = true;
          __syncthreads();  // B of P1
          if (s_abort) return;
          __syncthreads();  // C
          publish();
          for (int it = 0;; it++) {
            collect();
            const double gam = sums[0], del = sums[1], rr = sums[2];
            conv = (it > 0 || restart == 0) && (rr <= thr2 || rr == 0.0);
            const int code = conv ? kConverged
                             : (total_it + it >= a.max_iter || (a.variant == 0 && it >= kTeamRoundCap)) ? kStop
                                                                                                       : kRun;
            // beta = gam / gam_old, alpha = gam / (del - beta gam / alpha_old);
            // the reciprocals of the old values were formed while the rows
            // were updated, one division is left here
            const double alpha = first ? gam / del : gam / (del - gam * gam * rga);
            if (lane == 0) {
              s_be = first ? 0.0 : gam * rg;
              s_al = alpha;
              s_code = code;
            }
            __syncthreads();  // B
            if (s_abort) return;
            if (code != kRun) {
              total_it += it;
              break;
            }
            first = false;
            iters++;
            rg = 1.0 / gam;
            rga = rg / alpha;
            __syncthreads();  // C
            publish();
          }
        }
        __syncthreads();  // E
        __syncthreads();  // B of the true residual
        if (s_abort) return;
        __syncthreads();  // C
        publish();
        collect();
        rel = bb > 0 ? sqrt(sums[2] / bb) : sqrt(sums[2]);
        ok = rel <= tol || sums[2] == 0.0;
        // the true residual decides: a model that meets the tolerance is
        // done.  Otherwise residual replacement when the recurrence
        // converged; in auto mode also when the round hit its cap
        const bool capped = !conv && a.variant == 0;
        const bool again = !ok && (conv || capped) && restart < kTeamMaxRestarts && total_it < a.max_iter;
        if (lane == 0) s_code = again ? kRun : kStop;
        __syncthreads();  // D
        if (s_abort) return;
        if (!again) break;
        __syncthreads();  // E
        if (a.variant == 0) classic = true;
      }
      if (lane == 0 && sl.rank == 0) {
        double* o = a.model_out + (size_t)sl.model * 4;
        o[0] = iters;
        o[1] = rel;
        o[2] = ok ? 1.0 : 0.0;
        // row and dilational exchanges exceed the partial sums by at most two
        // per round: this bounds the tags of all three kinds
        a.base[sl.model] = tag0 + pe + 2 * (kTeamMaxRestarts + 2);
      }
    } else {
      unsigned e = 0;   // row exchanges published
      unsigned te = 0;  // dilational exchanges published
      // rows of other CTAs published in exchange e - 1, into xs: thread
      // pairs take the two packets of a row
      auto poll_rows = [&]() {
        const double* buf = a.row_pk + (size_t)((e - 1) & 1) * a.n_rows * 4 + 2 * (t & 1);
        const unsigned tag = tag0 + e;
        PollBound pb(a, sl, s_ticket0);
        for (int h = t >> 1; h < nh; h += kRowThreads / 2) {
          const double* src = buf + (size_t)hrow[h] * 4;
          unsigned g, hf;
          double v;
          for (;;) {
            v = get_packet(src, hf, g);
            if (g == tag) break;
            if (pb.give_up()) {
              s_abort = 1;
              return;
            }
          }
          double* o = xs + 3 * (nloc + h);
          o[t & 1] = v;
          // the third double's high (packet 0) or low half
          ((unsigned*)(o + 2))[1 - (t & 1)] = hf;
        }
      };
      // component ownership: set s holds component oc of row orow[s]
      const int oc = lane % 3, ob = lane - oc;
      int oi[SETS];       // local row (-1: none)
      int orow[SETS];     // global row
      bool opub[SETS];
#pragma unroll
      for (int j = 0; j < SETS; j++) {
        const int i = j * kSetRows + warp * 10 + lane / 3;
        oi[j] = lane < 30 && i < nloc ? i : -1;
        orow[j] = oi[j] >= 0 ? a.rows[sl.r0 + i] : 0;
        opub[j] = oi[j] >= 0 && k > 1 && oc < 2 && a.pub[sl.r0 + i];
      }
      // own rows' new values, to the neighbours and to xs (every lane calls)
      auto publish_rows = [&](const double* v) {
        double* buf = a.row_pk + (size_t)(e & 1) * a.n_rows * 4 + 2 * oc;
#pragma unroll
        for (int j = 0; j < SETS; j++) {
          const double third = __shfl_sync(0xffffffffu, v[j], ob + 2);
          if (opub[j])
            put_packet(buf + (size_t)orow[j] * 4, v[j],
                       oc ? (unsigned)__double2loint(third) : (unsigned)__double2hiint(third), tag0 + e + 1);
          if (oi[j] >= 0) xs[3 * oi[j] + oc] = v[j];
        }
        e++;
      };
      // The lane's blocks: the first kReg steps of its first row group in
      // registers (double in both forms: the conversion is paid once per
      // solve), the others in shared memory or in the slot's stream.
      double R[kReg > 0 ? kReg : 1][9];
      int rc[kReg > 0 ? kReg : 1];
      const int g_first = group_of(0);
      const int st_first = g_first >= 0 ? grp[g_first].steps() : 0;
#pragma unroll
      for (int b = 0; b < kReg; b++) {
        rc[b] = 0;
#pragma unroll
        for (int v = 0; v < 9; v++) R[b][v] = 0;
        if (b < st_first) {
          const int at = (grp[g_first].step + b) * 32 + lane;
          const int blk = a.blk[(size_t)sl.w0 * 32 + at];
          rc[b] = 3 * (int)cl[at];
          if (blk >= 0) {
            const MT* B = (const MT*)a.S + 9 * (size_t)blk;
#pragma unroll
            for (int v = 0; v < 9; v++) R[b][v] = (double)B[v];
          }
        }
      }
      for (int pass = 0; pass < passes; pass++) {
        const int g = group_of(pass);
        if (g < 0) continue;
        const RowGroup rg = grp[g];
        for (int b = 0; b < rg.steps(); b++) {
          const size_t at = ((size_t)sl.w0 + rg.step + b) * 32 + lane;
          if constexpr (DIL) {
            const int q2 = a.g2[at];
            double* gd = g2s + (size_t)(rg.step + b) * 96 + lane;
#pragma unroll
            for (int c = 0; c < 3; c++) gd[32 * c] = q2 >= 0 ? a.divblk[3 * (size_t)q2 + c] : 0.0;
          }
          // (register steps of the factored matrix keep d_row(col) in memory)
          if (!DIL && pass == 0 && b < kReg) continue;
          const int idx = rg.mem + b - (!DIL && pass == 0 ? kReg : 0);
          unsigned char* dst = idx < sl.steps_smem ? Ss + (size_t)idx * kStep : Sg + (size_t)(idx - sl.steps_smem) * kStep;
          const int blk = a.blk[at];
          const MT* B = (const MT*)a.S + 9 * (size_t)max(blk, 0);
#pragma unroll
          for (int v = 0; v < 9; v++) ((MT*)dst)[32 * v + lane] = blk >= 0 ? B[v] : MT(0);
          if constexpr (DIL) {
            double* gd = (double*)(dst + 32 * 9 * sizeof(MT));
            const int q1 = a.g1[at];
#pragma unroll
            for (int c = 0; c < 3; c++) gd[32 * c + lane] = q1 >= 0 ? a.divblk[3 * (size_t)q1 + c] : 0.0;
          }
        }
      }
      // one step of a row group from memory
      auto add_step = [&](const unsigned char* src, int c, bool with_S, double& a0, double& a1, double& a2, double& tt) {
        const double* xv = xs + 3 * c;
        const double x0 = xv[0], x1 = xv[1], x2 = xv[2];
        const MT* B = (const MT*)src + lane;
        if (with_S) {
          a0 += (double)B[0] * x0 + (double)B[32] * x1 + (double)B[64] * x2;
          a1 += (double)B[96] * x0 + (double)B[128] * x1 + (double)B[160] * x2;
          a2 += (double)B[192] * x0 + (double)B[224] * x1 + (double)B[256] * x2;
        }
        if constexpr (DIL) {
          const double* gd = (const double*)(src + 32 * 9 * sizeof(MT)) + lane;
          tt += gd[0] * x0 + gd[32] * x1 + gd[64] * x2;
        }
      };
      // steps in flight at once: memory-bound slots want more, the small ones
      // their registers for the matrix
      constexpr int kFlight = SETS == 1 ? 1 : 2;
      // sn = S xs for the slot's rows (xs complete behind the row barrier)
      auto product = [&]() {
        row_barrier();
#pragma unroll 1
        for (int pass = 0; pass < passes; pass++) {
          const int g = group_of(pass);
          if (g < 0) continue;
          const RowGroup rg = grp[g];
          const int st = rg.steps();
          const unsigned short* cp = cl + rg.step * 32 + lane;
          int idx = rg.mem, b = 0;
          double a0 = 0, a1 = 0, a2 = 0, tt = 0;
          if (kReg > 0 && pass == 0) {
#pragma unroll
            for (int q = 0; q < kReg; q++) {
              const double* xv = xs + rc[q];
              const double x0 = xv[0], x1 = xv[1], x2 = xv[2];
              a0 += R[q][0] * x0 + R[q][1] * x1 + R[q][2] * x2;
              a1 += R[q][3] * x0 + R[q][4] * x1 + R[q][5] * x2;
              a2 += R[q][6] * x0 + R[q][7] * x1 + R[q][8] * x2;
              if constexpr (DIL) {
                if (q < st) {
                  const unsigned char* src = idx + q < sl.steps_smem ? Ss + (size_t)(idx + q) * kStep
                                                                    : Sg + (size_t)(idx + q - sl.steps_smem) * kStep;
                  const double* gd = (const double*)(src + 32 * 9 * sizeof(MT)) + lane;
                  tt += gd[0] * x0 + gd[32] * x1 + gd[64] * x2;
                }
              }
            }
            b = kReg;
            if (DIL) idx += kReg;
          }
          const int in_smem = min(st - b, sl.steps_smem - idx);
#pragma unroll kFlight
          for (int q = 0; q < in_smem; q++) add_step(Ss + (size_t)(idx + q) * kStep, cp[32 * (b + q)], true, a0, a1, a2, tt);
          const int done = max(in_smem, 0);
          const unsigned char* sg = Sg + (ptrdiff_t)(idx + done - sl.steps_smem) * kStep;
#pragma unroll kFlight
          for (int q = done; q < st - b; q++) {
            add_step(sg, cp[32 * (b + q)], true, a0, a1, a2, tt);
            sg += kStep;
          }
          for (int off = (1 << rg.log()) >> 1; off > 0; off >>= 1) {
            a0 += __shfl_xor_sync(0xffffffffu, a0, off);
            a1 += __shfl_xor_sync(0xffffffffu, a1, off);
            a2 += __shfl_xor_sync(0xffffffffu, a2, off);
            if constexpr (DIL) tt += __shfl_xor_sync(0xffffffffu, tt, off);
          }
          const int sub = lane >> rg.log();
          if ((lane & ((1 << rg.log()) - 1)) == 0 && sub < rg.rows()) {
            const int i = rg.row + sub;
            sn[3 * i] = a0;
            sn[3 * i + 1] = a1;
            sn[3 * i + 2] = a2;
            if constexpr (DIL) {
              const double tv = ckp[i] * tt;
              ts[i] = tv;
              if (k > 1)
                put_packet(a.t_pk + ((size_t)(te & 1) * a.n_rows + a.rows[sl.r0 + i]) * 2, tv, 0u, tag0 + te + 1);
            }
          }
        }
        if constexpr (DIL) {
          // t of the neighbours, then each row adds sum_j t_j d_j(row)
          const double* buf = a.t_pk + (size_t)(te & 1) * a.n_rows * 2;
          const unsigned tag = tag0 + te + 1;
          PollBound pb(a, sl, s_ticket0);
          for (int h = t; h < nh; h += kRowThreads) {
            const double* src = buf + (size_t)hrow[h] * 2;
            unsigned g, hf;
            double v;
            for (;;) {
              v = get_packet(src, hf, g);
              if (g == tag) break;
              if (pb.give_up()) {
                s_abort = 1;
                break;
              }
            }
            if (g != tag) break;
            ts[nloc + h] = v;
          }
          te++;
          row_barrier();
#pragma unroll 1
          for (int pass = 0; pass < passes; pass++) {
            const int g = group_of(pass);
            if (g < 0) continue;
            const RowGroup rg = grp[g];
            const int st = rg.steps();
            const unsigned short* cp = cl + rg.step * 32 + lane;
            const double* gd = g2s + (size_t)rg.step * 96 + lane;
            double a0 = 0, a1 = 0, a2 = 0;
#pragma unroll 2
            for (int b = 0; b < st; b++) {
              const double tv = ts[cp[32 * b]];
              a0 += tv * gd[96 * b];
              a1 += tv * gd[96 * b + 32];
              a2 += tv * gd[96 * b + 64];
            }
            for (int off = (1 << rg.log()) >> 1; off > 0; off >>= 1) {
              a0 += __shfl_xor_sync(0xffffffffu, a0, off);
              a1 += __shfl_xor_sync(0xffffffffu, a1, off);
              a2 += __shfl_xor_sync(0xffffffffu, a2, off);
            }
            const int sub = lane >> rg.log();
            if ((lane & ((1 << rg.log()) - 1)) == 0 && sub < rg.rows()) {
              const int i = rg.row + sub;
              sn[3 * i] += a0;
              sn[3 * i + 1] += a1;
              sn[3 * i + 2] += a2;
            }
          }
        }
      };
      // the warp's sums of the rows' dot-product terms, ahead of C
      auto hand_sums = [&](double d0, double d1, double d2) {
        const double v = team_sum3(d0, d1, d2, lane);
        if ((lane & 7) == 0 && lane < 24) s_part[warp][lane >> 3] = v;
      };
      double x[SETS], r[SETS], u[SETS], w[SETS], z[SETS], q[SETS], s[SETS], p[SETS], D[SETS][3];
      // y = Dinv v of the row whose component this lane holds
      auto apply_inverse = [&](const double* v, double* y) {
#pragma unroll
        for (int j = 0; j < SETS; j++) {
          const double v0 = __shfl_sync(0xffffffffu, v[j], ob), v1 = __shfl_sync(0xffffffffu, v[j], ob + 1),
                       v2 = __shfl_sync(0xffffffffu, v[j], ob + 2);
          y[j] = D[j][0] * v0 + D[j][1] * v1 + D[j][2] * v2;
        }
      };
      // plane constraints: y -= n (n . y), the lane's component
      auto project = [&](double* y) {
        if (!a.row_nrm) return;
#pragma unroll
        for (int j = 0; j < SETS; j++) {
          const double v0 = __shfl_sync(0xffffffffu, y[j], ob), v1 = __shfl_sync(0xffffffffu, y[j], ob + 1),
                       v2 = __shfl_sync(0xffffffffu, y[j], ob + 2);
          const double* nq = a.row_nrm + 3 * (size_t)orow[j];
          if (oi[j] >= 0) y[j] -= nq[oc] * (nq[0] * v0 + nq[1] * v1 + nq[2] * v2);
        }
      };
#pragma unroll
      for (int j = 0; j < SETS; j++) {
        x[j] = r[j] = u[j] = w[j] = z[j] = q[j] = s[j] = p[j] = 0;
        D[j][0] = D[j][1] = D[j][2] = 0;
      }

      if constexpr (DIL) {
        // the dilational term's diagonal blocks, sum_n c kp_n d_n(row) d_n(row)^T
        // (their six different entries), into sn
        for (int pass = 0; pass < passes; pass++) {
          const int g = group_of(pass);
          if (g < 0) continue;
          const RowGroup rg = grp[g];
          const unsigned short* cp = cl + rg.step * 32 + lane;
          const double* gd = g2s + (size_t)rg.step * 96 + lane;
          double q6[6] = {0, 0, 0, 0, 0, 0};
          for (int b = 0; b < rg.steps(); b++) {
            const double ck = ts[cp[32 * b]], y0 = gd[96 * b], y1 = gd[96 * b + 32], y2 = gd[96 * b + 64];
            q6[0] += ck * y0 * y0;
            q6[1] += ck * y0 * y1;
            q6[2] += ck * y0 * y2;
            q6[3] += ck * y1 * y1;
            q6[4] += ck * y1 * y2;
            q6[5] += ck * y2 * y2;
          }
          for (int off = (1 << rg.log()) >> 1; off > 0; off >>= 1)
#pragma unroll
            for (int c = 0; c < 6; c++) q6[c] += __shfl_xor_sync(0xffffffffu, q6[c], off);
          const int sub = lane >> rg.log();
          if ((lane & ((1 << rg.log()) - 1)) == 0 && sub < rg.rows())
#pragma unroll
            for (int c = 0; c < 6; c++) sn[6 * (rg.row + sub) + c] = q6[c];
        }
        row_barrier();
      }
      // ---- P0: block-Jacobi inverse, r = b - S x0, u = Dinv r; ||b||^2,
      // r.u, r.r
#pragma unroll
      for (int j = 0; j < SETS; j++) {
        if (oi[j] < 0) continue;
        const int i = oi[j];
        const MT* B = (const MT*)a.S + 9 * (size_t)a.diag[sl.r0 + i];
        double dg[9], inv[9];
#pragma unroll
        for (int c = 0; c < 9; c++) {
          dg[c] = (double)B[c];
          inv[c] = 0;
        }
        if constexpr (DIL) {
          const double* q6 = sn + 6 * i;
          dg[0] += q6[0];
          dg[1] += q6[1];
          dg[2] += q6[2];
          dg[3] += q6[1];
          dg[4] += q6[3];
          dg[5] += q6[4];
          dg[6] += q6[2];
          dg[7] += q6[4];
          dg[8] += q6[5];
        }
        if (invert3(inv, dg) == 0.0) {
          // a singular diagonal block: the solve ends at the next barrier B
          atomicExch(a.flags, B200FEM_ERR_INVALID_ARG);
          s_abort = 1;
        }
        if (a.row_nrm) {
          // P D^-1 P with P = I - n n^T
          const double* nq = a.row_nrm + 3 * (size_t)orow[j];
          double tm[9];
#pragma unroll
          for (int m = 0; m < 3; m++)
#pragma unroll
            for (int l = 0; l < 3; l++)
              tm[3 * m + l] = inv[3 * m + l] - nq[m] * (nq[0] * inv[l] + nq[1] * inv[3 + l] + nq[2] * inv[6 + l]);
#pragma unroll
          for (int m = 0; m < 3; m++)
#pragma unroll
            for (int l = 0; l < 3; l++)
              inv[3 * m + l] = tm[3 * m + l] - (tm[3 * m] * nq[0] + tm[3 * m + 1] * nq[1] + tm[3 * m + 2] * nq[2]) * nq[l];
        }
#pragma unroll
        for (int c = 0; c < 3; c++) D[j][c] = oc == 0 ? inv[c] : oc == 1 ? inv[3 + c] : inv[6 + c];
      }
      product();      // (its first barrier also ends the reads of kp in ts and of sn)
      row_barrier();  // sn
      double d0 = 0, d1 = 0, d2 = 0;
      {
        double bv[SETS];
#pragma unroll
        for (int j = 0; j < SETS; j++) {
          bv[j] = 0;
          if (oi[j] < 0) continue;
          bv[j] = a.b[3 * (size_t)orow[j] + oc];
          x[j] = xs[3 * oi[j] + oc];
          r[j] = bv[j] - sn[3 * oi[j] + oc];
        }
        project(r);
        project(bv);
        apply_inverse(r, u);
#pragma unroll
        for (int j = 0; j < SETS; j++) {
          d0 += bv[j] * bv[j];
          d1 += r[j] * u[j];
          d2 += r[j] * r[j];
        }
      }
      publish_rows(u);
      hand_sums(d0, d1, d2);
      __syncthreads();  // C
      bool classic = a.variant == 1;
      for (;;) {
        if (classic) {
          // ---- classic PCG: two exchanges per iteration, from r and
          // z = u = Dinv r of P0 or of the true-residual pass
#pragma unroll
          for (int j = 0; j < SETS; j++) p[j] = q[j] = 0;
          for (;;) {
            poll_rows();
            product();
            __syncthreads();  // B
            if (s_abort) return;
            if (s_code != kRun) break;
            {
              const double be = s_be;
              double az[SETS];
#pragma unroll
              for (int j = 0; j < SETS; j++) az[j] = oi[j] >= 0 ? sn[3 * oi[j] + oc] : 0.0;
              project(az);
              d0 = 0;
#pragma unroll
              for (int j = 0; j < SETS; j++) {
                p[j] = u[j] + be * p[j];
                q[j] = az[j] + be * q[j];
                d0 += p[j] * q[j];
              }
            }
            hand_sums(d0, 0.0, 0.0);
            __syncthreads();  // C
            __syncthreads();  // D
            if (s_abort) return;
            const double al = s_al;
#pragma unroll
            for (int j = 0; j < SETS; j++) {
              x[j] += al * p[j];
              r[j] -= al * q[j];
            }
            apply_inverse(r, u);
            publish_rows(u);
            d0 = d1 = 0;
#pragma unroll
            for (int j = 0; j < SETS; j++) {
              d0 += r[j] * u[j];
              d1 += r[j] * r[j];
            }
            hand_sums(d0, d1, 0.0);
            __syncthreads();  // C
          }
        } else {
          // ---- P1: w = S u, m = Dinv w; r.u, w.u, r.r
          poll_rows();
          product();
          __syncthreads();  // B
          if (s_abort) return;
          double m[SETS];
#pragma unroll
          for (int j = 0; j < SETS; j++) {
            w[j] = oi[j] >= 0 ? sn[3 * oi[j] + oc] : 0.0;
            z[j] = q[j] = s[j] = p[j] = 0;
          }
          project(w);
          apply_inverse(w, m);
          publish_rows(m);
          d0 = d1 = d2 = 0;
#pragma unroll
          for (int j = 0; j < SETS; j++) {
            d0 += r[j] * u[j];
            d1 += w[j] * u[j];
            d2 += r[j] * r[j];
          }
          hand_sums(d0, d1, d2);
          __syncthreads();  // C
          for (;;) {
            // n = S m beside the scalars of this iteration, then
            // z = n + beta z; q = m + beta q; s = w + beta s; p = u + beta p;
            // x += alpha p; r -= alpha s; u -= alpha q; w -= alpha z; m = Dinv w
            poll_rows();
            product();
            __syncthreads();  // B
            if (s_abort) return;
            if (s_code != kRun) break;
            const double al = s_al, be = s_be;
            {
              double nn[SETS];
#pragma unroll
              for (int j = 0; j < SETS; j++) nn[j] = oi[j] >= 0 ? sn[3 * oi[j] + oc] : 0.0;
              project(nn);
#pragma unroll
              for (int j = 0; j < SETS; j++) {
                z[j] = nn[j] + be * z[j];
                q[j] = m[j] + be * q[j];
                s[j] = w[j] + be * s[j];
                p[j] = u[j] + be * p[j];
                x[j] += al * p[j];
                r[j] -= al * s[j];
                u[j] -= al * q[j];
                w[j] -= al * z[j];
              }
            }
            apply_inverse(w, m);
            publish_rows(m);
            d0 = d1 = d2 = 0;
#pragma unroll
            for (int j = 0; j < SETS; j++) {
              d0 += r[j] * u[j];
              d1 += w[j] * u[j];
              d2 += r[j] * r[j];
            }
            hand_sums(d0, d1, d2);
            __syncthreads();  // C
          }
        }
        // ---- the true residual decides; on a miss the recurrences restart
        // from it
        __syncthreads();  // E
        publish_rows(x);
        poll_rows();
        product();
        __syncthreads();  // B
        if (s_abort) return;
#pragma unroll
        for (int j = 0; j < SETS; j++)
          r[j] = oi[j] >= 0 ? a.b[3 * (size_t)orow[j] + oc] - sn[3 * oi[j] + oc] : 0.0;
        project(r);
        apply_inverse(r, u);
        publish_rows(u);
        d1 = d2 = 0;
#pragma unroll
        for (int j = 0; j < SETS; j++) {
          d1 += r[j] * u[j];
          d2 += r[j] * r[j];
        }
        hand_sums(0.0, d1, d2);
        __syncthreads();  // C
        __syncthreads();  // D
        if (s_abort) return;
        if (s_code != kRun) break;
        __syncthreads();  // E
        if (a.variant == 0) classic = true;
      }
#pragma unroll
      for (int j = 0; j < SETS; j++) {
        double xn = 0, off = 0;
        const bool own = oi[j] >= 0;
        const size_t n3 = own ? 3 * (size_t)a.act_node[orow[j]] + oc : 0;
        if (own) a.x[3 * (size_t)orow[j] + oc] = x[j];
        if (!a.update_state) continue;
        if (own) {
          a.vprev4[n3] = a.vprev3[n3];
          a.vprev3[n3] = a.vprev2[n3];
          a.vprev2[n3] = a.vprev[n3];
          a.vprev[n3] = a.vel[n3];
          a.vel[n3] = x[j];
          xn = a.xpos[n3] + sp[0] * x[j];
        }
        if (a.row_nrm) {
          // GlobalMass position correction of a single-particle plane
          // constraint: the node moves onto its plane along the normal
          const double v0 = __shfl_sync(0xffffffffu, xn, ob), v1 = __shfl_sync(0xffffffffu, xn, ob + 1),
                       v2 = __shfl_sync(0xffffffffu, xn, ob + 2);
          if (own) {
            const double* nq = a.row_nrm + 3 * (size_t)orow[j];
            off = nq[oc] * (nq[0] * v0 + nq[1] * v1 + nq[2] * v2 - a.row_off[orow[j]]);
          }
        }
        if (own) a.xpos[n3] = xn - off;
      }
    }
  }
}

using TeamKernel = void (*)(TeamArgs);
template <typename MT, bool DIL>
TeamKernel team_kernel_of(int sets) {
  return sets == 3 ? pcg_team_kernel<MT, 3, DIL> : sets == 2 ? pcg_team_kernel<MT, 2, DIL> : pcg_team_kernel<MT, 1, DIL>;
}
TeamKernel team_kernel(const Engine& eng) {
  const bool dil = eng.factored && eng.d.n_dil_nodes > 0;
  if (eng.precision == B200FEM_PREC_MIXED)
    return dil ? team_kernel_of<float, true>(eng.team_sets) : team_kernel_of<float, false>(eng.team_sets);
  return dil ? team_kernel_of<double, true>(eng.team_sets) : team_kernel_of<double, false>(eng.team_sets);
}

// f(thread, i) for i in [0, n) on up to `threads` host threads.
template <typename F>
void parallel_for(int n, int threads, F&& f) {
  std::atomic<int> next(0);
  auto work = [&](int th) {
    for (int i; (i = next++) < n;) f(th, i);
  };
  std::vector<std::thread> pool;
  try {
    for (int th = 1; th < std::min(threads, n); th++) pool.emplace_back(work, th);
  } catch (const std::system_error&) {  // the system has no more threads: those there are do it
  }
  work(0);
  for (auto& t : pool) t.join();
}
int host_threads() { return (int)std::min(16u, std::max(1u, std::thread::hardware_concurrency())); }

// Recursive bisection of rows [a, b) into k parts of nearly equal weight along
// the longest axis of their nodes' rest positions.
// The cuts go to cut[0 .. k - 1]; the two halves of a large range are cut in
// parallel.
void bisect(std::vector<int>& rows, int a, int b, int k, const double* pos, const int* node,
            const std::vector<int>& weight, int* cut) {
  if (k <= 1) {
    cut[0] = b;
    return;
  }
  double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
  long long total = 0;
  for (int i = a; i < b; i++) {
    total += weight[rows[i]];
    for (int c = 0; c < 3; c++) {
      const double v = pos[3 * (size_t)node[rows[i]] + c];
      lo[c] = std::min(lo[c], v);
      hi[c] = std::max(hi[c], v);
    }
  }
  int ax = 0;
  for (int c = 1; c < 3; c++)
    if (hi[c] - lo[c] > (hi[ax] - lo[ax]) * (1 + 1e-9)) ax = c;
  std::vector<std::pair<double, int>> key(b - a);
  for (int i = a; i < b; i++) key[i - a] = {pos[3 * (size_t)node[rows[i]] + ax], rows[i]};
  std::sort(key.begin(), key.end());
  for (int i = a; i < b; i++) rows[i] = key[i - a].second;
  const int kl = k / 2;
  long long sum = 0;
  int mid = a;
  // (every part keeps at least one row)
  while (mid < b - (k - kl) && (mid < a + kl || (2 * sum + weight[rows[mid]]) * k <= 2 * total * kl))
    sum += weight[rows[mid++]];
  auto left = [&]() { bisect(rows, a, mid, kl, pos, node, weight, cut); };
  std::thread other;
  if (b - a >= 8192) {
    try {
      other = std::thread(left);
    } catch (const std::system_error&) {
    }
  }
  if (!other.joinable()) left();
  bisect(rows, mid, b, k - kl, pos, node, weight, cut + kl);
  if (other.joinable()) other.join();
}

}  // namespace

namespace {
// One model's split over k CTAs (slot offsets relative to it)
struct TeamSplit {
  std::vector<TeamSlot> slots;
  std::vector<int> rows, halo, blk;
  std::vector<int4> group;
  std::vector<unsigned short> cl;
  std::vector<unsigned char> pub;  // per row of the model
  size_t smem = 0;
  int stream = 0;
};
}  // namespace

// Largest dynamic shared memory of one CTA of the team kernel.
static size_t team_smem_budget(int device) {
  int optin = 0;
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  return (size_t)std::max(0, optin - 2048);
}

// Adds the slots of `p` behind those of `out`.
template <typename Dst>
static void append_split(Dst& out, const TeamSplit& p) {
  for (TeamSlot s : p.slots) {
    s.r0 += (int)out.rows.size();
    s.h0 += (int)out.halo.size();
    s.g0 += (int)out.group.size();
    s.w0 += (int)(out.cl.size() / 32);
    s.stream0 += out.stream;
    out.slots.push_back(s);
  }
  out.stream += p.stream;
  out.smem = std::max(out.smem, p.smem);
  out.rows.insert(out.rows.end(), p.rows.begin(), p.rows.end());
  out.halo.insert(out.halo.end(), p.halo.begin(), p.halo.end());
  out.group.insert(out.group.end(), p.group.begin(), p.group.end());
  out.cl.insert(out.cl.end(), p.cl.begin(), p.cl.end());
  out.blk.insert(out.blk.end(), p.blk.begin(), p.blk.end());
}

// Lanes (as a power of two) that walk a row of n blocks in at most T steps.
static int lanes_log(int n, int T) {
  int l = 1;
  while (l < 5 && (T << l) < n) l++;
  return l;
}

// Splits one model's n rows from row0 on (rowptr/col: the pattern with global
// rows) over k CTAs of nearly equal weight.  pos: node positions, node: row -
// row0 -> node.  A CTA's rows are ordered by their number of blocks, most
// first, and a warp's row group holds rows with the same number of lanes,
// chosen so that every row takes at most T steps; T is the smallest number
// for which the groups are walked in one pass of the row warps (a latency:
// the longest rows, 27 blocks in a tet mesh and over 60 in a quadratic one,
// would otherwise hold up all others), or kManySteps where one pass cannot
// do, which wastes few lanes.  A row's blocks are dealt to its steps and
// lanes so that the sixteen lanes of a half-warp read x from different banks
// where that can be had.  Steps of S that do not fit the shared memory are
// streamed when `stream` allows it, else the split fails.
constexpr int kManySteps = 6;
static bool team_split_model(int row0, int n, int k, int sets, const std::vector<int>& rowptr,
                             const std::vector<int>& col, const double* pos, const int* node, int mt_bytes, bool dil,
                             size_t budget, bool stream, int threads, TeamSplit& result) {
  std::vector<int> rows(n), cut(k), weight(n);
  std::iota(rows.begin(), rows.end(), 0);
  auto len = [&](int r) { return rowptr[row0 + r + 1] - rowptr[row0 + r]; };
  for (int r = 0; r < n; r++) weight[r] = len(r) + kRowWeight;
  bisect(rows, 0, n, k, pos, node, weight, cut.data());
  int nmax = 0;
  for (int c = 0; c < k; c++) nmax = std::max(nmax, cut[c] - (c ? cut[c - 1] : 0));
  if (nmax > sets * kSetRows) return false;
  // register steps take no memory (the factored matrix keeps d_row(col) of
  // all its steps there)
  const int reg = dil ? 0 : reg_blocks(sets, false);
  struct Scratch {
    std::vector<int> stamp, loc, rem;
  };
  std::vector<Scratch> scratch(threads);
  std::vector<TeamSplit> piece(k);
  std::atomic<bool> fits(true);
  // one CTA's slot; false when it does not fit
  auto split_slot = [&](int th, int c) -> bool {
    TeamSplit& out = piece[c];
    std::vector<int>&stamp = scratch[th].stamp, &loc = scratch[th].loc, &rem = scratch[th].rem;
    if (stamp.empty()) {
      stamp.assign(n, -1);
      loc.assign(n, 0);
    }
    const int a = c ? cut[c - 1] : 0, b = cut[c], nloc = b - a;
    if (nloc <= 0) return false;
    std::sort(rows.begin() + a, rows.begin() + b, [&](int x, int y) {
      return len(x) != len(y) ? len(x) > len(y) : x < y;
    });
    for (int i = a; i < b; i++) {
      stamp[rows[i]] = c;
      loc[rows[i]] = i - a;
    }
    const int h0 = 0;
    for (int i = a; i < b; i++)
      for (int p = rowptr[row0 + rows[i]]; p < rowptr[row0 + rows[i] + 1]; p++) {
        const int j = col[p] - row0;
        if (stamp[j] != c) {
          stamp[j] = c;
          out.halo.push_back(j);
        }
      }
    std::sort(out.halo.begin() + h0, out.halo.end());
    const int nh = (int)out.halo.size() - h0;
    if (nloc + nh > 65535) return false;
    for (int h = 0; h < nh; h++) {
      loc[out.halo[h0 + h]] = nloc + h;
      out.halo[h0 + h] += row0;
    }
    TeamSlot s{};
    s.rank = c;
    s.k = k;
    s.nloc = nloc;
    s.nh = nh;
    for (int i = a; i < b; i++) out.rows.push_back(row0 + rows[i]);
    auto count_groups = [&](int T) {
      int g = 0;
      for (int i = a; i < b; g++) i += 32 >> lanes_log(len(rows[i]), T);
      return g;
    };
    int T = 1;
    while (T <= 64 && count_groups(T) > kRowWarps) T++;
    if (T > kManySteps && count_groups(kManySteps) > kRowWarps) T = std::min(T, kManySteps);
    int mem = 0;  // steps of S kept in memory
    for (int i1 = a; i1 < b;) {
      const int lg = lanes_log(len(rows[i1]), T), L = 1 << lg;
      const int g0 = i1, g1 = std::min(b, i1 + (32 >> lg));
      const int steps = (len(rows[g0]) + L - 1) / L;
      if (steps > 0xffff) return false;
      out.group.push_back(int4{steps | lg << 16 | (g1 - g0 - 1) << 24, s.steps, mem, g0 - a});
      mem += s.groups < kRowWarps ? std::max(0, steps - reg) : steps;
      s.groups++;
      const size_t at = out.cl.size();
      out.cl.resize(at + 32 * (size_t)steps, 0);
      out.blk.resize(at + 32 * (size_t)steps, -1);
      const int half = std::max(1, 16 >> lg);
      for (int i0 = g0; i0 < g1; i0 += half) {
        const int nr = std::min(half, g1 - i0);
        // the rows' blocks not placed yet, one list after the other
        int start[16], left[16];
        rem.clear();
        for (int q = 0; q < nr; q++) {
          start[q] = (int)rem.size();
          const int r = row0 + rows[i0 + q];
          for (int p = rowptr[r]; p < rowptr[r + 1]; p++) rem.push_back(p);
          left[q] = (int)rem.size() - start[q];
        }
        for (int st = 0; st < steps; st++) {
          unsigned char used[16] = {0};
          int pad = 0;
          for (int q = 0; q < nr; q++) {
            for (int l = 0; l < L && left[q] > 0; l++) {
              int best = 0, bu = 255;
              for (int z = 0; z < left[q]; z++) {
                const int u = used[loc[col[rem[start[q] + z]] - row0] & 15];
                if (u < bu) {
                  bu = u;
                  best = z;
                  if (u == 0) break;
                }
              }
              const int p = rem[start[q] + best];
              rem[start[q] + best] = rem[start[q] + --left[q]];
              const int lc = loc[col[p] - row0];
              used[lc & 15]++;
              pad = lc;
              const size_t w = at + 32 * (size_t)st + (size_t)(i0 - g0 + q) * L + l;
              out.cl[w] = (unsigned short)lc;
              out.blk[w] = p;
            }
          }
          // lanes without a block read an address the half-warp reads anyway
          for (int q = 0; q < nr * L; q++) {
            const size_t w = at + 32 * (size_t)st + (size_t)(i0 - g0) * L + q;
            if (out.blk[w] < 0) out.cl[w] = (unsigned short)pad;
          }
        }
      }
      s.steps += steps;
      i1 = g1;
    }
    const size_t fixed = team_layout(nloc, nh, s.steps, s.groups, dil).S;
    if (fixed > budget) return false;
    const size_t sb = step_bytes(mt_bytes, dil);
    s.steps_smem = (int)std::min<size_t>(mem, (budget - fixed) / sb);
    out.stream = mem - s.steps_smem;
    if (!stream && s.steps_smem < mem) return false;
    out.smem = fixed + sb * s.steps_smem;
    out.slots.push_back(s);
    return true;
  };
  parallel_for(k, threads, [&](int th, int c) {
    if (fits && !split_slot(th, c)) fits = false;
  });
  if (!fits) return false;
  result = TeamSplit();
  result.pub.assign(n, 0);
  size_t lanes = 0;
  for (const TeamSplit& p : piece) lanes += p.cl.size();
  result.cl.reserve(lanes);
  result.blk.reserve(lanes);
  for (TeamSplit& p : piece) {
    for (int h : p.halo) result.pub[h - row0] = 1;
    append_split(result, p);
  }
  return true;
}

// A model's PCG iterations relative to other models', for the queue order
// only: block-Jacobi PCG takes about sqrt(1 + h^2 w^2) of them, w = sqrt(M /
// rho) / dx the highest frequency of the mesh (M the P-wave modulus).  The
// step size is not known when the pack is built; h = 0.01 weighs stiff models
// against soft ones.  Fitted to 700 uneven NeoHookean beams (5 to 590
// iterations, correlation 0.97).
static double expected_iterations(const ModelDesc& m, const ModelHost& h) {
  const double* p = m.mat_params;
  double modulus = 0;
  if (m.mat_kind == B200FEM_MAT_MOONEYRIVLIN) modulus = p[5] + 8.0 / 3.0 * (p[0] + p[1]);
  else modulus = p[0] * (1 - p[1]) / ((1 + p[1]) * (1 - 2 * p[1]));
  double vol = 0;
  for (double v : h.rest_vol) vol += v;
  const double dx = std::cbrt(std::max(vol, 1e-300) / std::max(m.n_nodes, 1));
  const double w = std::sqrt(std::max(modulus, 0.0) / std::max(m.density, 1e-300)) / dx;
  const double it = 4 + 24 * 0.01 * w;
  return std::isfinite(it) ? std::min(it, 1e6) : 4;
}

// The team layout of a pack: per model the number of CTAs, its split, and the
// slots of all models in queue order.
bool plan_team(const Engine& eng, int grid_max, const std::vector<int>& rowptr, const std::vector<int>& col,
               const std::vector<int>& diag, bool dil, TeamHost& out) {
  const int M = (int)eng.hosts.size();
  const int mt = eng.precision == B200FEM_PREC_MIXED ? 4 : 8;
  const size_t budget = team_smem_budget(eng.device);
  const int R = eng.row_off[M];
  if (R <= 0 || grid_max <= 0) return false;
  for (int r = 0; r < R; r++)  // a row without blocks (an active node in no element) has no diagonal
    if (diag[r] < rowptr[r] || diag[r] >= rowptr[r + 1]) return false;
  // Rows per CTA wanted: all CTAs busy from the start, at least kWantRows.
  // Fewer rows shorten the product and put more CTAs into every exchange (us
  // per iteration: 40x10x10 hex beam 4.2 at 30 rows, 3.2 at 44, 3.3 at 60, 3.9
  // at 90; 1,958-row quadratic beam 2.7, 2.2, 2.4, 3.5; 2,376-row NODAL block,
  // whose two exchanges bound it, 4.3 at 12 to 60).  Up to kAloneRows one CTA
  // needs no exchange at all: a 90-row beam 1.36 against 1.44 in two CTAs.
  struct Range {
    int lo, hi;   // fewest CTAs that hold the model's rows, most that help it
    double it;
  };
  std::vector<int> order, team(M, 0);
  for (int m = 0; m < M; m++)
    if (eng.row_off[m + 1] > eng.row_off[m]) order.push_back(m);
  // duration of one solve in the time of a row: the iterations' exchange and
  // rows, and the slot's set-up (measured: 1.4 us per iteration and 8.5 ns per
  // row of it, 26 us per slot)
  auto cost = [&](const Range& r, int n, int k) { return r.it * (kExchangeRows + (double)n / k) + kSetupRows; };
  auto plan = [&](int sets, std::vector<int>& teams) {
    std::vector<Range> range(M);
    double lo = 0, hi = 0;
    for (int m : order) {
      const int a = eng.row_off[m], n = eng.row_off[m + 1] - a;
      const size_t need = (size_t)(rowptr[a + n] - rowptr[a]) * (9 * mt + 2 + (dil ? 48 : 0)) + (size_t)n * 48;
      const int rows = sets * kSetRows * 8 / 9;  // parts of equal weight differ in their rows
      Range& r = range[m];
      r.lo = std::max({1, (int)((need + budget - 1) / budget), (n + rows - 1) / rows});
      // beyond kWantTeam CTAs only rows count (the hex beam above)
      r.hi = n <= kAloneRows ? 1
                             : std::max(std::min((n + kWantRows - 1) / kWantRows, kWantTeam), n / (2 * kWantRows));
      r.lo = std::min({r.lo, grid_max, n});
      r.hi = std::max(r.lo, std::min(r.hi, grid_max));
      r.it = expected_iterations(eng.models[m], eng.hosts[m]);
      lo = std::max(lo, cost(r, n, r.hi));
      hi += cost(r, n, r.lo) * r.lo;
    }
    // the shortest makespan that the CTAs' time allows: every model takes the
    // fewest CTAs that end it in time (48 uneven beams, whose slowest holds
    // three CTAs for 1.75 ms at their fewest, then end at 0.72 ms)
    auto teams_for = [&](double T) {
      double area = 0;
      for (int m : order) {
        const int n = eng.row_off[m + 1] - eng.row_off[m];
        const Range& r = range[m];
        int k = r.lo;
        while (k < r.hi && cost(r, n, k) > T) k++;
        teams[m] = k;
        area += k * cost(r, n, k);
      }
      return area;
    };
    hi = std::max(hi, lo);
    if (teams_for(lo) > kFill * grid_max * lo) {
      for (int i = 0; i < 40; i++) {
        const double T = 0.5 * (lo + hi);
        if (teams_for(T) > kFill * grid_max * T) lo = T;
        else hi = T;
      }
      teams_for(hi);
      return hi;
    }
    return lo;
  };
  // Two component sets (300 rows) a CTA: enough rows to spread an iteration's
  // exchange over (256 uneven beams, mixed: 2.36 ms at up to 300 rows, 3.06 at
  // 150, 2.52 at 450), few enough to keep a slow model's iterations short;
  // three only where a model needs them.
  int sets = 2;
  for (int m : order)
    if ((eng.row_off[m + 1] - eng.row_off[m]) > (long long)grid_max * (sets * kSetRows * 8 / 9)) sets = kMaxSets;
  plan(sets, team);
  // queue order: the longest expected solve first, so that no long one starts
  // last and the short ones fill the CTAs that the others free
  std::vector<double> expect(M, 0.0);
  int nloc_max = 0;
  for (int m : order) {
    const int n = eng.row_off[m + 1] - eng.row_off[m];
    expect[m] = cost(Range{0, 0, expected_iterations(eng.models[m], eng.hosts[m])}, n, team[m]);
    nloc_max = std::max(nloc_max, (n + team[m] - 1) / team[m]);
  }
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return expect[x] > expect[y]; });
  // component sets of the launch (the kernel's register steps go by them);
  // parts of equal weight differ in their rows
  sets = std::min(kMaxSets, (nloc_max + nloc_max / 8 + kSetRows - 1) / kSetRows);
  std::vector<TeamSplit> split(M);
  std::atomic<bool> good(true);
  // few models: threads within each split, else one model per thread
  const int threads = host_threads(), across = (int)order.size() >= threads ? threads : 1;
  parallel_for((int)order.size(), across, [&](int, int i) {
    const int m = order[i], a = eng.row_off[m], n = eng.row_off[m + 1] - a;
    for (int k = team[m]; good; k = std::min({grid_max, n, k + std::max(1, k / 10)})) {
      // the largest team streams what does not fit
      const bool last = k >= std::min(grid_max, n);
      if (team_split_model(a, n, k, sets, rowptr, col, eng.models[m].rest.data(), eng.hosts[m].act_node.data(), mt,
                           dil, budget, last, across > 1 ? 1 : std::min(threads, 1 + n / 512), split[m]))
        break;
      if (last) good = false;
    }
  });
  if (!good) return false;
  out = TeamHost();
  out.pub.resize(R);
  std::vector<unsigned char> rpub(R, 0);
  for (int m : order) {
    TeamSplit& sp = split[m];
    const int s0 = (int)out.slots.size();
    std::copy(sp.pub.begin(), sp.pub.end(), rpub.begin() + eng.row_off[m]);
    for (TeamSlot& s : sp.slots) {
      s.model = m;
      s.s0 = s0;
    }
    if (order.size() == 1) {
      // (one model: nothing to shift)
      out.slots.swap(sp.slots);
      out.rows.swap(sp.rows);
      out.halo.swap(sp.halo);
      out.blk.swap(sp.blk);
      out.group.swap(sp.group);
      out.cl.swap(sp.cl);
      out.smem = sp.smem;
      out.stream = sp.stream;
    } else {
      append_split(out, sp);
    }
    sp = TeamSplit();
  }
  out.diag.resize(out.rows.size());
  for (size_t i = 0; i < out.rows.size(); i++) {
    out.diag[i] = diag[out.rows[i]];
    out.pub[i] = rpub[out.rows[i]];
  }
  out.grid = std::min(grid_max, (int)out.slots.size());
  out.sets = sets;
  out.step_bytes = step_bytes(mt, dil);
  return true;
}

void team_parallel(int n, const std::function<void(int)>& f) {
  parallel_for(n, host_threads(), [&](int, int i) { f(i); });
}

static std::mutex g_team_mu;

cudaError_t prepare_team(Engine& eng) {
  std::lock_guard<std::mutex> lk(g_team_mu);
  // the opt-in is process-wide per function: always the device's largest, so
  // no engine lowers what another needs
  return cudaFuncSetAttribute(team_kernel(eng), cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)team_smem_budget(eng.device));
}

// After a solve that ended with an error its tickets are incomplete and its
// packets are of no use: start both over (the stream is idle).
cudaError_t team_recover(Engine& eng) {
  if (!eng.team) return cudaSuccess;
  DevPack& d = eng.d;
  cudaError_t e = cudaMemsetAsync(d.team_ticket, 0, sizeof(unsigned long long), eng.stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(d.team_row_pk, 0, sizeof(double) * 8 * (size_t)d.n_rows, eng.stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(d.team_part_pk, 0, sizeof(double) * 8 * (size_t)d.team_slots, eng.stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(d.team_base, 0, sizeof(unsigned) * (size_t)d.n_models, eng.stream);
  if (e == cudaSuccess && d.team_t_pk)
    e = cudaMemsetAsync(d.team_t_pk, 0, sizeof(double) * 4 * (size_t)d.n_rows, eng.stream);
  return e == cudaSuccess ? cudaStreamSynchronize(eng.stream) : e;
}

cudaError_t launch_pcg_team(Engine& eng, int max_iter, bool update_state, const double* rhs, double* xsol,
                            double tol_override, double* model_out) {
  DevPack& d = eng.d;
  const bool fp32 = eng.precision == B200FEM_PREC_MIXED;
  TeamArgs a{};
  a.slots = d.team_slot;
  a.n_slots = d.team_slots;
  a.ticket = d.team_ticket;
  a.rows = d.team_rows;
  a.pub = d.team_pub;
  a.halo = d.team_halo;
  a.diag = d.team_diag;
  a.group = d.team_group;
  a.blk = d.team_blk;
  a.stream = d.team_stream;
  a.cl = d.team_cl;
  a.g1 = d.team_g1;
  a.g2 = d.team_g2;
  a.S = eng.factored ? (fp32 ? (const void*)d.S1_f : (const void*)d.S1) : (fp32 ? (const void*)d.S_f : (const void*)d.S);
  a.b = rhs;
  a.x = xsol;
  a.step = d.step;
  a.tol_override = tol_override;
  a.model_out = model_out;
  a.flags = d.flags;
  a.timeout_ns = 1000000ull * (unsigned long long)eng.barrier_timeout_ms;
  a.skip_cta = eng.test_skip_arrival - 1;
  a.max_iter = max_iter;
  a.variant = eng.pcg_variant;
  // a pack's state is updated after every model's solve, and only when none
  // ended with an error; a single model's in the solve itself
  a.update_state = update_state && d.n_models == 1 ? 1 : 0;
  a.n_rows = d.n_rows;
  a.base = d.team_base;
  a.row_pk = d.team_row_pk;
  a.part_pk = d.team_part_pk;
  a.t_pk = d.team_t_pk;
  a.xpos = d.x;
  a.vel = d.v;
  a.vprev = d.vprev;
  a.vprev2 = d.vprev2;
  a.vprev3 = d.vprev3;
  a.vprev4 = d.vprev4;
  a.act_node = d.act_node;
  a.model_active = eng.any_inactive ? d.model_active : nullptr;
  a.row_nrm = (update_state && eng.integrator == B200FEM_INTEGRATOR_CONSTRAINED_BACKWARD_EULER && d.row_nrm)
                  ? d.row_nrm
                  : nullptr;
  a.row_off = a.row_nrm ? d.row_off : nullptr;
  a.divblk = d.divblk;
  a.node_kp = d.node_kp;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(eng.team_grid);
  cfg.blockDim = dim3(kTeamThreads);
  cfg.dynamicSmemBytes = eng.team_smem;
  cfg.stream = eng.stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, team_kernel(eng), a);
  if (e != cudaSuccess || !update_state || d.n_models == 1) return e;
  team_state_kernel<<<(d.n_rows + 127) / 128, 128, 0, eng.stream>>>(
      d.n_rows, d.act_node, d.row_model, d.step, xsol, d.x, d.v, d.vprev, d.vprev2, d.vprev3, d.vprev4,
      a.model_active, a.row_nrm, a.row_off, d.flags);
  return cudaGetLastError();
}

}  // namespace b200fem
