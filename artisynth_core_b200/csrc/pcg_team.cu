// pcg_team.cu -- block-Jacobi PCG with one team of CTAs per model.
//
// pcg.cu runs every model of the pack through one grid-wide loop: each
// iteration ends at a barrier of the whole grid, then reads the partial dot
// products and gathers the search direction, three dependent L2 round trips
// (5 us per iteration on the 40x10x10 hex beam whose arithmetic takes well
// under one).  Here a model's rows are dealt to a team of k CTAs, a compact
// set of rows each (recursive bisection of the node positions), and
//   * the CTA's blocks of S stay in shared memory for the whole solve and the
//     PCG vectors of a row in the registers of the thread that owns it;
//   * there is no barrier: every value that crosses CTAs travels as a 16-byte
//     packet {double, tag} written and read in one 128-bit access, so the
//     reader polls the datum itself and one L2 round trip carries both the
//     value and the synchronisation.  A reader waits for the rows next to its
//     own and for the team's k partial sums, nothing else;
//   * models run independently of one another: teams form from a queue of
//     slots (largest models first), so a slow model occupies its own CTAs
//     instead of keeping the grid in its loop.
// The recurrences, tests, restarts and results are those of pcg.cu's kernel
// (pipelined CG of Ghysels & Vanroose 2014, then classic PCG after a
// residual replacement); sums are formed in a fixed order, so results are
// bit-reproducible and a model's result does not depend on the rest of the
// pack.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <numeric>

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
constexpr int kMaxSets = 2;
constexpr int kTeamMaxRows = kSetRows * kMaxSets;
// blocks of a lane's first row that stay in its registers for the solve
__host__ __device__ constexpr int reg_blocks(int sets) { return sets == 1 ? 3 : 1; }
constexpr int kWantRows = 60, kAloneRows = 96;  // see plan_team
constexpr int kTeamMaxRestarts = 10;  // as in pcg.cu
constexpr int kTeamRoundCap = 400;    // as in pcg.cu

struct TeamArgs {
  const TeamSlot* slots;
  int n_slots;
  unsigned long long* ticket;
  const int* rows;         // slot-major: the global rows each slot owns (ascending)
  const unsigned char* pub;  // per owned row (slot-major): some other CTA reads it
  const int* halo;         // slot-major: the global rows of other slots that the slot reads
  const int* ro;           // slot-major, nloc + 1 per slot: block offsets within the slot
  const int* src;          // per owned row: first block of the row in S
  const unsigned short* dloc;  // per owned row: its diagonal block within the row
  const unsigned short* cl;  // slot-major: per block its column as a local index (owned, then halo)
  const int* g1;           // factored NODAL: per block the divBlk slots of d_row(col) and d_col(row) (-1 none)
  const int* g2;
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
// recorded an error or the time limit (counted from the first such check)
// has passed; the latter records B200FEM_ERR_TIMEOUT.
struct PollBound {
  int* flags;
  unsigned long long limit, t0 = 0;
  unsigned n = 0;
  __device__ __forceinline__ PollBound(int* f, unsigned long long l) : flags(f), limit(l) {}
  __device__ __forceinline__ bool give_up() {
    if ((++n & 63u) != 0) return false;
    if (*(volatile int*)flags != 0) return true;
    const unsigned long long now = team_ns();
    if (t0 == 0) t0 = now;
    else if (now - t0 > limit) {
      atomicExch(flags, B200FEM_ERR_TIMEOUT);
      return true;
    }
    return false;
  }
};

__host__ __device__ inline size_t team_align(size_t b) { return (b + 15) & ~(size_t)15; }
struct TeamLayout {
  size_t S, g, xs, sn, ts, ckp, ro, halo, cl, total;
};
__host__ __device__ inline TeamLayout team_layout(int nloc, int nb, int nh, int mt_bytes, bool dil) {
  TeamLayout o;
  size_t p = 0;
  o.S = p;
  p += team_align((size_t)nb * 9 * mt_bytes);
  o.g = p;
  if (dil) p += team_align((size_t)nb * 6 * sizeof(double));
  o.xs = p;
  p += team_align((size_t)(nloc + nh) * 3 * sizeof(double));
  o.sn = p;
  p += team_align((size_t)nloc * 3 * sizeof(double));
  o.ts = p;
  if (dil) p += team_align((size_t)(nloc + nh) * sizeof(double));
  o.ckp = p;
  if (dil) p += team_align((size_t)nloc * sizeof(double));
  o.ro = p;
  p += team_align((size_t)(nloc + 1) * sizeof(int));
  o.halo = p;
  p += team_align((size_t)nh * sizeof(int));
  o.cl = p;
  p += team_align((size_t)nb * sizeof(unsigned short));
  o.total = p;
  return o;
}

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

// L: lanes per block row in the SpMV; SETS: component sets (rows <= SETS *
// kSetRows); DIL: the factored NODAL matrix.
template <typename MT, int L, int SETS, bool DIL>
__global__ void __launch_bounds__(kTeamThreads, 1) pcg_team_kernel(TeamArgs a) {
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ double s_part[kRowWarps][3];
  __shared__ double s_al, s_be;
  __shared__ int s_code, s_abort;
  __shared__ int s_ticket;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, gl = lane & (L - 1);
  const bool red = warp == kRowWarps;
  // an error of an earlier launch of the call: nothing runs
  if (*(volatile int*)a.flags != 0) return;
  if (t == 0) s_abort = 0;

  for (;;) {
    // next slot; a launch draws n_slots + gridDim tickets in all (one past
    // the end per CTA), so the counter needs no reset between launches
    if (t == 0) s_ticket = (int)(atomicAdd(a.ticket, 1ull) % ((unsigned long long)a.n_slots + gridDim.x));
    __syncthreads();
    const int si = s_ticket;
    __syncthreads();
    if (si >= a.n_slots) return;
    const TeamSlot sl = a.slots[si];
    if (a.model_active && !a.model_active[sl.model]) {
      if (sl.rank == 0 && t == 0) {
        double* o = a.model_out + (size_t)sl.model * 4;
        o[0] = 0;
        o[1] = 0;
        o[2] = 1.0;
      }
      continue;
    }
    const int nloc = sl.nloc, nh = sl.nh, nb = sl.nb, k = sl.k;
    // tags continue from the model's last solve: a packet left by it never
    // carries a tag of this one
    const unsigned tag0 = a.base[sl.model];
    const double* sp = a.step + (size_t)sl.model * 8;
    const TeamLayout lay = team_layout(nloc, nb, nh, (int)sizeof(MT), DIL);
    MT* const S = (MT*)(dyn + lay.S);
    double* const gs = (double*)(dyn + lay.g);  // per block d_row(col), d_col(row)
    double* const xs = (double*)(dyn + lay.xs);
    double* const sn = (double*)(dyn + lay.sn);
    double* const ts = (double*)(dyn + lay.ts);
    double* const ckp = (double*)(dyn + lay.ckp);
    int* const ro = (int*)(dyn + lay.ro);
    int* const hrow = (int*)(dyn + lay.halo);
    unsigned short* const cl = (unsigned short*)(dyn + lay.cl);

    // ---- the slot's matrix, columns and starting vector to shared memory
    for (int i = t; i <= nloc; i += kTeamThreads) ro[i] = a.ro[sl.ro0 + i];
    for (int i = t; i < nh; i += kTeamThreads) hrow[i] = a.halo[sl.h0 + i];
    for (int i = t; i < nb; i += kTeamThreads) cl[i] = a.cl[sl.b0 + i];
    __syncthreads();
    {
      // a warp per row: the row's blocks are contiguous in S
      const MT* Sg = (const MT*)a.S;
      for (int i = warp; i < nloc; i += kTeamWarps) {
        const int o = ro[i] * 9, n = ro[i + 1] * 9 - o;
        const MT* sv = Sg + (size_t)a.src[sl.r0 + i] * 9;
        for (int q = lane; q < n; q += 32) {
          const unsigned d = (unsigned)__cvta_generic_to_shared(S + o + q);
          asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(sv + q), "n"((int)sizeof(MT)));
        }
      }
      asm volatile("cp.async.commit_group;");
    }
    for (int i = t; i < nloc + nh; i += kTeamThreads) {
      const int r = i < nloc ? a.rows[sl.r0 + i] : hrow[i - nloc];
#pragma unroll
      for (int c = 0; c < 3; c++) xs[3 * i + c] = a.x[3 * (size_t)r + c];
    }
    if constexpr (DIL) {
      for (int i = t; i < nb; i += kTeamThreads) {
        const int q1 = a.g1[sl.b0 + i], q2 = a.g2[sl.b0 + i];
#pragma unroll
        for (int c = 0; c < 3; c++) {
          gs[6 * i + c] = q1 >= 0 ? a.divblk[3 * (size_t)q1 + c] : 0.0;
          gs[6 * i + 3 + c] = q2 >= 0 ? a.divblk[3 * (size_t)q2 + c] : 0.0;
        }
      }
      const double cm = sp[0] * sp[0] + sp[0] * sp[2];
      for (int i = t; i < nloc + nh; i += kTeamThreads) {
        const int r = i < nloc ? a.rows[sl.r0 + i] : hrow[i - nloc];
        const double v = cm * a.node_kp[a.act_node[r]];
        ts[i] = v;  // until the first product: kp of the neighbours for the block diagonal
        if (i < nloc) ckp[i] = v;
      }
    }
    asm volatile("cp.async.wait_group 0;");
    __syncthreads();

    if ((int)blockIdx.x == a.skip_cta) {
      // failure-detection test: this CTA never publishes; it waits for
      // itself, bounded like every other wait, and the team's waits run out
      if (t == 0) {
        PollBound pb(a.flags, a.timeout_ns);
        while (!pb.give_up()) {
        }
      }
      return;
    }

    const double tol = a.tol_override > 0 ? a.tol_override : sp[6];
    // Two roles with the same sequence of CTA barriers per phase: B ends the
    // SpMV and makes the scalars known, C hands the per-warp dot products to
    // the reducing warp, D (classic PCG, true residual) makes a scalar known
    // that depends on C's.
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
          put_packet(a.part_pk + ((size_t)(pe & 1) * a.n_slots + si) * 4 + 2 * lane, lane ? sums[1] : sums[0],
                     lane ? (unsigned)__double2loint(sums[2]) : (unsigned)__double2hiint(sums[2]), tag0 + pe + 1);
        pe++;
      };
      // the team's sums of the last publish (a team of one has them): lane
      // pairs take the two packets of a slot
      auto collect = [&]() {
        if (k == 1) return;
        const double* buf = a.part_pk + (size_t)((pe - 1) & 1) * a.n_slots * 4 + 2 * (lane & 1);
        const unsigned tag = tag0 + pe;
        const int qe = sl.s0 + k;
        PollBound pb(a.flags, a.timeout_ns);
        double m = 0, r = 0;
        constexpr int U = 5;
        for (int qb = sl.s0; qb < qe; qb += 16 * U) {
          double v[U];
          unsigned hf[U];
          for (;;) {
            bool all = true;
#pragma unroll
            for (int u = 0; u < U; u++) {
              const int q = qb + 16 * u + (lane >> 1);
              v[u] = 0;
              hf[u] = 0;
              if (q < qe) {
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
        }
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
          conv = sums[2] <= thr2 || sums[2] == 0.0;
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
            conv = rr <= thr2 || rr == 0.0;
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
        PollBound pb(a.flags, a.timeout_ns);
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
      // the lane's blocks of its first row in registers (double in both
      // forms: the conversion is paid once per solve)
      constexpr int kRegBlocks = reg_blocks(SETS);
      double R[kRegBlocks][9];
      int rc[kRegBlocks];
      const int i0 = warp * (32 / L) + lane / L;  // first row of the lane's group
      const int pr0 = i0 < nloc ? ro[i0] + gl : 0, pr1 = i0 < nloc ? ro[i0 + 1] : 0;
#pragma unroll
      for (int b = 0; b < kRegBlocks; b++) {
        const int p = pr0 + L * b;
        const bool in = p < pr1;
        rc[b] = in ? 3 * (int)cl[p] : 0;
#pragma unroll
        for (int q = 0; q < 9; q++) R[b][q] = in ? (double)S[9 * p + q] : 0.0;
      }
      // sn = S xs for the slot's rows (xs complete behind the row barrier)
      auto product = [&]() {
        row_barrier();
        constexpr int G = 32 / L;
        for (int base = warp * G, pass = 0; base < nloc; base += kRowWarps * G, pass++) {
          const int i = base + lane / L;
          const bool valid = i < nloc;
          double a0 = 0, a1 = 0, a2 = 0, tt = 0;
          int p = 0, p1 = 0;
          if (pass == 0) {
#pragma unroll
            for (int b = 0; b < kRegBlocks; b++) {
              const double* xv = xs + rc[b];
              const double x0 = xv[0], x1 = xv[1], x2 = xv[2];
              a0 += R[b][0] * x0 + R[b][1] * x1 + R[b][2] * x2;
              a1 += R[b][3] * x0 + R[b][4] * x1 + R[b][5] * x2;
              a2 += R[b][6] * x0 + R[b][7] * x1 + R[b][8] * x2;
              if constexpr (DIL) {
                const int pp = pr0 + L * b;
                if (pp < pr1) tt += gs[6 * pp] * x0 + gs[6 * pp + 1] * x1 + gs[6 * pp + 2] * x2;
              }
            }
            p = pr0 + L * kRegBlocks;
            p1 = pr1;
          } else if (valid) {
            p = ro[i] + gl;
            p1 = ro[i + 1];
          }
#pragma unroll 1
          for (; p < p1; p += L) {
            const double* xv = xs + 3 * (int)cl[p];
            const MT* B = S + 9 * p;
            const double x0 = xv[0], x1 = xv[1], x2 = xv[2];
            a0 += (double)B[0] * x0 + (double)B[1] * x1 + (double)B[2] * x2;
            a1 += (double)B[3] * x0 + (double)B[4] * x1 + (double)B[5] * x2;
            a2 += (double)B[6] * x0 + (double)B[7] * x1 + (double)B[8] * x2;
            if constexpr (DIL) tt += gs[6 * p] * x0 + gs[6 * p + 1] * x1 + gs[6 * p + 2] * x2;
          }
#pragma unroll
          for (int off = L / 2; off > 0; off >>= 1) {
            a0 += __shfl_xor_sync(0xffffffffu, a0, off);
            a1 += __shfl_xor_sync(0xffffffffu, a1, off);
            a2 += __shfl_xor_sync(0xffffffffu, a2, off);
            if constexpr (DIL) tt += __shfl_xor_sync(0xffffffffu, tt, off);
          }
          if (valid && gl == 0) {
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
          PollBound pb(a.flags, a.timeout_ns);
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
          for (int base = warp * G; base < nloc; base += kRowWarps * G) {
            const int i = base + lane / L;
            const bool valid = i < nloc;
            int p = 0, p1 = 0;
            if (valid) {
              p = ro[i] + gl;
              p1 = ro[i + 1];
            }
            double a0 = 0, a1 = 0, a2 = 0;
#pragma unroll 2
            for (; p < p1; p += L) {
              const double tv = ts[cl[p]];
              a0 += tv * gs[6 * p + 3];
              a1 += tv * gs[6 * p + 4];
              a2 += tv * gs[6 * p + 5];
            }
#pragma unroll
            for (int off = L / 2; off > 0; off >>= 1) {
              a0 += __shfl_xor_sync(0xffffffffu, a0, off);
              a1 += __shfl_xor_sync(0xffffffffu, a1, off);
              a2 += __shfl_xor_sync(0xffffffffu, a2, off);
            }
            if (valid && gl == 0) {
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

      // ---- P0: block-Jacobi inverse, r = b - S x0, u = Dinv r; ||b||^2,
      // r.u, r.r
#pragma unroll
      for (int j = 0; j < SETS; j++) {
        if (oi[j] < 0) continue;
        const int i = oi[j];
        const MT* B = S + 9 * (ro[i] + a.dloc[sl.r0 + i]);
        double dg[9], inv[9];
#pragma unroll
        for (int c = 0; c < 9; c++) {
          dg[c] = (double)B[c];
          inv[c] = 0;
        }
        if constexpr (DIL) {
          // the dilational term's diagonal block: sum_n c kp_n d_n(row) d_n(row)^T
          for (int pb = ro[i]; pb < ro[i + 1]; pb++) {
            const double* g = gs + 6 * pb + 3;
            const double ck = ts[cl[pb]];
#pragma unroll
            for (int m = 0; m < 3; m++)
#pragma unroll
              for (int l = 0; l < 3; l++) dg[3 * m + l] += ck * g[m] * g[l];
          }
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
      product();      // (its first barrier also ends the reads of kp in ts)
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
TeamKernel team_kernel_of(int lanes, int sets) {
  if (sets > 1) return lanes == 4 ? pcg_team_kernel<MT, 4, 2, DIL> : pcg_team_kernel<MT, 8, 2, DIL>;
  return lanes == 4 ? pcg_team_kernel<MT, 4, 1, DIL> : lanes == 8 ? pcg_team_kernel<MT, 8, 1, DIL>
                                                                   : pcg_team_kernel<MT, 16, 1, DIL>;
}
TeamKernel team_kernel(const Engine& eng) {
  const bool dil = eng.factored && eng.d.n_dil_nodes > 0;
  if (eng.precision == B200FEM_PREC_MIXED)
    return dil ? team_kernel_of<float, true>(eng.team_lanes, eng.team_sets)
               : team_kernel_of<float, false>(eng.team_lanes, eng.team_sets);
  return dil ? team_kernel_of<double, true>(eng.team_lanes, eng.team_sets)
             : team_kernel_of<double, false>(eng.team_lanes, eng.team_sets);
}

// Recursive bisection of `rows` into k parts of nearly equal size along the
// longest axis of their nodes' rest positions; part[i] of the i-th row.
void bisect(std::vector<int>& rows, int a, int b, int k, const double* pos, const int* node, std::vector<int>& cut) {
  if (k <= 1) {
    cut.push_back(b);
    return;
  }
  double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
  for (int i = a; i < b; i++)
    for (int c = 0; c < 3; c++) {
      const double v = pos[3 * (size_t)node[rows[i]] + c];
      lo[c] = std::min(lo[c], v);
      hi[c] = std::max(hi[c], v);
    }
  int ax = 0;
  for (int c = 1; c < 3; c++)
    if (hi[c] - lo[c] > (hi[ax] - lo[ax]) * (1 + 1e-9)) ax = c;
  const int kl = k / 2;
  const int mid = a + (int)((long long)(b - a) * kl / k);
  std::nth_element(rows.begin() + a, rows.begin() + mid, rows.begin() + b, [&](int x, int y) {
    const double px = pos[3 * (size_t)node[x] + ax], py = pos[3 * (size_t)node[y] + ax];
    return px != py ? px < py : x < y;
  });
  bisect(rows, a, mid, kl, pos, node, cut);
  bisect(rows, mid, b, k - kl, pos, node, cut);
}

}  // namespace

namespace {
// One model's split over k CTAs (slot offsets relative to it)
struct TeamSplit {
  std::vector<TeamSlot> slots;
  std::vector<int> rows, ro, halo, blk;
  std::vector<unsigned short> cl;
  std::vector<unsigned char> pub;  // per row of the model
  int nloc_max = 0;
  size_t smem = 0;
};
}  // namespace

// Largest dynamic shared memory of one CTA of the team kernel.
static size_t team_smem_budget(int device) {
  int optin = 0;
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  return (size_t)std::max(0, optin - 2048);
}

// Splits one model's rows (rowptr/col: its pattern with global rows, blocks
// counted from the pack's first) over k CTAs.  pos: node positions, node:
// row - row0 -> node.  Returns false when a CTA would not fit.
static bool team_split_model(int row0, int n, int k, const std::vector<int>& rowptr, const std::vector<int>& col,
                      const double* pos, const int* node, int mt_bytes, bool dil, size_t budget, TeamSplit& out) {
  std::vector<int> rows(n);
  std::iota(rows.begin(), rows.end(), 0);
  std::vector<int> cut;
  bisect(rows, 0, n, k, pos, node, cut);
  out = TeamSplit();
  std::vector<int> stamp(n, -1), loc(n, 0);
  out.pub.assign(n, 0);
  int a = 0;
  for (int c = 0; c < k; c++) {
    const int b = cut[c];
    if (b <= a || b - a > kTeamMaxRows) return false;
    std::sort(rows.begin() + a, rows.begin() + b);
    for (int i = a; i < b; i++) {
      stamp[rows[i]] = c;
      loc[rows[i]] = i - a;
    }
    std::vector<int> halo;
    int nb = 0;
    for (int i = a; i < b; i++) {
      const int r = row0 + rows[i];
      nb += rowptr[r + 1] - rowptr[r];
      for (int p = rowptr[r]; p < rowptr[r + 1]; p++) {
        const int j = col[p] - row0;
        if (stamp[j] != c) {
          stamp[j] = c;
          halo.push_back(j);
        }
      }
    }
    std::sort(halo.begin(), halo.end());
    const int nloc = b - a, nh = (int)halo.size();
    if (nloc + nh > 65535 || team_layout(nloc, nb, nh, mt_bytes, dil).total > budget) return false;
    for (int h = 0; h < nh; h++) {
      loc[halo[h]] = nloc + h;
      out.pub[halo[h]] = 1;
    }
    TeamSlot s{};
    s.rank = c;
    s.k = k;
    s.nloc = nloc;
    s.nh = nh;
    s.nb = nb;
    s.r0 = (int)out.rows.size();
    s.ro0 = (int)out.ro.size();
    s.h0 = (int)out.halo.size();
    s.b0 = (int)out.cl.size();
    int o = 0;
    for (int i = a; i < b; i++) {
      const int r = row0 + rows[i];
      out.rows.push_back(r);
      out.ro.push_back(o);
      for (int p = rowptr[r]; p < rowptr[r + 1]; p++) {
        out.cl.push_back((unsigned short)loc[col[p] - row0]);
        out.blk.push_back(p);
      }
      o += rowptr[r + 1] - rowptr[r];
    }
    out.ro.push_back(o);
    for (int h : halo) out.halo.push_back(row0 + h);
    out.slots.push_back(s);
    out.nloc_max = std::max(out.nloc_max, nloc);
    out.smem = std::max(out.smem, team_layout(nloc, nb, nh, mt_bytes, dil).total);
    a = b;
  }
  return true;
}

// The team layout of a pack: per model the number of CTAs, its split, and the
// slots of all models in queue order (most rows first, so that the longest
// solves start first and the short ones fill the CTAs they free).
bool plan_team(Engine& eng, int grid_max, const std::vector<int>& rowptr, const std::vector<int>& col,
               const std::vector<int>& diag, bool dil, TeamHost& out) {
  const int M = (int)eng.hosts.size();
  const int mt = eng.precision == B200FEM_PREC_MIXED ? 4 : 8;
  const size_t budget = team_smem_budget(eng.device);
  const int R = eng.row_off[M];
  if (R <= 0 || grid_max <= 0) return false;
  // Rows per CTA wanted: all CTAs busy from the start, at least kWantRows.
  // 60 rows give each row eight of the 480 row lanes; fewer rows per CTA put
  // more CTAs into every sum (40x10x10 hex beam, us per iteration: 3.4 at 32
  // rows in 148 CTAs, 2.8 at 64 rows in 76, 3.1 at 96; 1,958-row quadratic
  // beam 2.9 at 32 rows, 3.0 at 48, 4.7 at 64, where four lanes walk its
  // 23-block rows).  Up to kAloneRows one CTA needs no exchange at all: a
  // 72-row beam 1.36 us per iteration against 1.6 in two CTAs.
  const int want = std::max(kWantRows, (R + grid_max - 1) / grid_max);
  std::vector<int> order;
  for (int m = 0; m < M; m++)
    if (eng.row_off[m + 1] > eng.row_off[m]) order.push_back(m);
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) {
    return eng.row_off[x + 1] - eng.row_off[x] > eng.row_off[y + 1] - eng.row_off[y];
  });
  out = TeamHost();
  out.pub.assign(R, 0);
  std::vector<unsigned char> rpub(R, 0);
  for (int m : order) {
    const int a = eng.row_off[m], n = eng.row_off[m + 1] - a;
    const long long nb = rowptr[a + n] - rowptr[a];
    const size_t need = team_layout(n, (int)std::min<long long>(nb, 1 << 28), 0, mt, dil).total;
    int k = std::max({1, n <= kAloneRows ? 1 : (n + want - 1) / want, (int)((need + budget - 1) / budget), (n + kTeamMaxRows - 1) / kTeamMaxRows});
    TeamSplit sp;
    for (;; k += std::max(1, k / 10)) {
      if (k > std::min(grid_max, n)) return false;
      if (team_split_model(a, n, k, rowptr, col, eng.models[m].rest.data(), eng.hosts[m].act_node.data(), mt, dil,
                           budget, sp))
        break;
    }
    const int s0 = (int)out.slots.size();
    const int r0 = (int)out.rows.size(), ro0 = (int)out.ro.size(), h0 = (int)out.halo.size(), b0 = (int)out.cl.size();
    for (TeamSlot s : sp.slots) {
      s.model = m;
      s.s0 = s0;
      s.r0 += r0;
      s.ro0 += ro0;
      s.h0 += h0;
      s.b0 += b0;
      out.slots.push_back(s);
    }
    for (int i = 0; i < n; i++) rpub[a + i] = sp.pub[i];
    out.rows.insert(out.rows.end(), sp.rows.begin(), sp.rows.end());
    out.ro.insert(out.ro.end(), sp.ro.begin(), sp.ro.end());
    out.halo.insert(out.halo.end(), sp.halo.begin(), sp.halo.end());
    out.cl.insert(out.cl.end(), sp.cl.begin(), sp.cl.end());
    out.blk.insert(out.blk.end(), sp.blk.begin(), sp.blk.end());
    out.nloc = std::max(out.nloc, sp.nloc_max);
    out.smem = std::max(out.smem, sp.smem);
  }
  out.src.resize(out.rows.size());
  out.dloc.resize(out.rows.size());
  for (size_t i = 0; i < out.rows.size(); i++) {
    const int r = out.rows[i];
    out.src[i] = rowptr[r];
    // a row without blocks (an active node in no element) cannot be owned:
    // its diagonal has no place in the slot
    if (diag[r] < rowptr[r] || diag[r] >= rowptr[r + 1] || rowptr[r + 1] - rowptr[r] > 65535) return false;
    out.dloc[i] = (unsigned short)(diag[r] - rowptr[r]);
    out.pub[i] = rpub[r];
  }
  out.grid = std::min(grid_max, (int)out.slots.size());
  // lanes per row of the SpMV: as many as the row warps hold at once
  out.lanes = out.nloc * 16 <= kRowThreads ? 16 : out.nloc * 8 <= kRowThreads ? 8 : 4;
  out.sets = out.nloc > kSetRows ? 2 : 1;
  return true;
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
  a.ro = d.team_ro;
  a.src = d.team_src;
  a.dloc = d.team_dloc;
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
