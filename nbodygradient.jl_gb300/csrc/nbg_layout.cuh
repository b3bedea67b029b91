// nbg_layout.cuh -- data layout shared by the host orchestration and the
// kernels of libnbg_cuda: operator-record sizes, the per-group argument block
// and the launcher declarations (definitions live in nbg_kernels_impl.cuh and
// are instantiated once per body count by nbg_inst.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace nbg {

// Pair record: K[36] (row-major r*6+l), mi = m_i/(m_i+m_j), mj likewise, and
// Psi[6] = G k d(delxv/k)/dk, B[6] = delxv/(m_i+m_j).  With D = J_i - J_j and
// u = K D, plus Psi in the columns of m_i and m_j, the pair adds mj u to body i
// and -mi u to body j; the column of m_i takes B off body j's rows and that of
// m_j adds it to body i's (d(mj)/dm_i = -mj/(m_i+m_j) and so on).
constexpr int PREC = 50;
constexpr int PREC_MI = 36, PREC_MJ = 37, PREC_PSI = 38, PREC_B = 44;

__host__ __device__ constexpr int op_size(int N) { return 12 * N * N; }
__host__ __device__ inline int pair_bit(int i, int j, int N) { return i * N - i * (i + 1) / 2 + (j - i - 1); }

// Record size of one step for N bodies with npk Kepler pairs; kick operators
// only when the group has kick pairs.
__host__ __device__ inline int step_record_size(int N, int npk, bool kick) {
  return (kick ? 2 * op_size(N) : 0) + 2 * npk * PREC + op_size(N);
}

// Captured Kepler-pair parameters (producer -> operator kernel), see
// put_capture: x0[3], v0[3], eight values of the solve and the four
// coefficients of its result.  1/r = 0 in its place marks a pair without mass.
constexpr int PCAP = 18;
constexpr int PCAP_RINV = 11;
// Doubles of scratch a search needs: in kick groups its final step's record,
// else that step's captures, snapshots and pair records with d(delxv)/dh.
__host__ __device__ inline int search_scratch(int N, int npk, bool kick) {
  return kick ? step_record_size(N, npk, true) : 2 * npk * (PCAP + PREC + 6) + 6 * N;
}

constexpr int PROD_BS = 32;     // orbit producer: threads per warp-sized unit of work
constexpr int PROD_MAX_WARPS = 4;  // orbit producer: up to 4 independent warps per block
__host__ __device__ constexpr int team_lanes(int N) { return N / 2 > 1 ? N / 2 : 1; }  // lanes of a system's team
// Jacobian consumer: columns per block.  96 N bytes of shared memory a column:
// four warps a block, two from nine bodies on, so that six or more warps fit an
// SM (227 KB) at every N; every block holds 24 KB or more.
__host__ __device__ constexpr int cons_bs(int N) { return N >= 9 ? 64 : 128; }
constexpr int TRANSIT_BS = 32;  // transit searches: one warp per block
constexpr int OPS_BS = 128;     // operator kernels

// Doubles per transit of the adjoint record: the row u^T = w^T S(dt0) of
// the transit time and gdot (7N + 1); TransitParameters add the rows of
// v_sky and b_sky^2, v_sky and d v_sky / dt (21N + 3).
__host__ __device__ inline int trec_size(int N, int tbv) { return tbv ? 21 * N + 3 : 7 * N + 1; }

// Snapshots per step, 3N doubles each: positions at the correctors, then
// phisalpha!'s accelerations there, or in kick groups the positions at the
// first and at the second kick.
__host__ __device__ inline int snap_count(bool kick) { return kick ? 3 : 2; }


// Up to how many running systems of a group the latency-bound forms are taken.
//
// Rows consumer: six lanes a column are level with one at 64 columns an SM (96
// up to four bodies).  us a step: N = 8 96 systems 417 -> 387, 192 484 -> 510;
// N = 10 96 systems 627 -> 549, 192 747 -> 792.
__host__ inline int rows_limit(int N, int sms) { return (N <= 4 ? 96 : 64) * sms / (7 * N); }

// Systems whose producer blocks fit on half of the SMs, one block each (two
// systems of up to three bodies to a block, lanes_systems): as many get SMs of
// their own.
__host__ inline int tail_limit(int N, int sms) { return (N <= 3 ? 2 : 1) * (sms / 2 > 32 ? sms / 2 : 32); }

// Lanes producer: a level costs a warp per pair where the one-lane and team
// forms carry 32 or 32 / (N/2) systems, so the line is where the levels, 2N - 3
// per system, fill the FP64 pipes, alone or beside the consumer.  us a step, one
// lane or team -> lanes:
//   with derivatives    N = 2 512 systems 63 -> 39, 1024 65 -> 63;
//                       N = 3 152 182 -> 100 on SMs of its own, 200 172 -> 210;
//                       N = 4 512 423 -> 306, 1024 460 -> 586;
//                       N = 5 1024 1307 -> 1140, 2048 1383 -> 1638;
//                       N = 6 512 1434 -> 1055, 1024 1626 -> 1724;
//                       N = 8 384 2118 -> 1600, 768 2360 -> 2629;
//                       N = 10 256 2735 -> 1896, 512 3450 -> 3972
//   without             N = 2 768 59 -> 46, 1024 59 -> 64; N = 3 768 172 -> 170, 1024 174 -> 186;
//                       N = 4 768 379 -> 323, 1024 381 -> 450; N = 5 512 498 -> 459, 768 630 -> 705;
//                       N = 8 384 1112 -> 1079, 576 1140 -> 1305; N = 10 256 1380 -> 1288, 384 2273 -> 2426
__host__ inline int lanes_limit(int N, bool grad, int sms) {
  if (!grad) return N <= 4 ? 5 * sms : 24 * sms / (2 * N - 3);
  if (N == 3) return tail_limit(N, sms);
  return N <= 4 ? rows_limit(N, sms) : 48 * sms / (2 * N - 3);
}

struct GroupArgs {
  int N, S, nsys, grad, K, R, npk;
  int spw;   // orbit producer: systems per warp (lanes >= spw idle)
  int team;  // orbit producer: 1 = a team of lanes per system (orbit_team_kernel), 0 = one lane
  // transit searches of this chunk on a block's lanes each (transit_lanes_kernel):
  // set by the host per chunk when few systems of the group are still running,
  // so that the searches are latency-bound; a full group keeps one lane per
  // search, which uses every lane of every warp
  int search_lanes;
  // forms for latency-bound chunks (few systems running), set by the host per
  // chunk: the orbit producer's lanes form
  // (orbit_lanes_kernel) and the Jacobian consumer's rows form
  // (jacobian_rows_kernel)
  int wide, rows;
  // Block layout of the orbit producer: pwarps independent warps per block
  // (0: by the group's size, launch_orbit) and prod_smem bytes of dynamic shared memory per block (at
  // least what the team form needs).  A large allocation keeps the
  // shared-memory-hungry consumer blocks, and the operator / search blocks
  // that ask for guard_smem bytes, off the SMs that run producer blocks.
  int pwarps, prod_smem, guard_smem;
  unsigned long long kick;
  // per-system state, structure of arrays: element e of system s at [e * S + s]
  double *x, *v, *xe, *ve, *m, *dqdt, *gsave;
  long long* count;  // [N][S]
  double *t0, *h, *hI;
  long long* nsteps;
  // first chunk of each slot, in steps (null: every system starts at chunk 0);
  // the request server admits systems into running groups this way
  const long long* kbase;
  // length of each system's last step (null: h); the plain integration
  // drivers end on a fractional step (Integrator.jl:187-194)
  const double* hlast;
  int notransit;  // 1: no transit detection (the plain integration drivers)
  int tbv;        // 1: TransitParameters outputs (t, v_sky, b_sky^2 per transit)
  // CartesianOutput recording (null: off): the state at the start of every
  // step of the chunk, x and v as [slot][step][x (3N), v (3N)], jac_step as
  // [slot][step][7N x 7N column-major]
  double* trajxv;
  double* trajJ;
  int *ntt, *ti, *sysidx;
  unsigned int* status;
  // packed outputs in the caller's layout, indexed by global system
  double* tt;
  const long long* off_tt;
  double* dtdq0;
  const long long* off_dq;
  // records
  double* steprec;  // [K][R][S]
  double* trec;     // [K][N-1][7N+1][S]
  int* tflag;       // [K][N-1][S]
  // consumer state: non-mass rows of jac_step / jac_error, [S][6N][7N]
  double *Jint, *Eint;
  // transit searches queued by the orbit producer for the transit kernel
  double* task_f;   // [task_cap][12N + 2]: x, v, xerror, verror, first dt0, t
  int* task_i;      // [task_cap][3]: system, slot kk*(N-1)+o, transit index
  int* task_count;  // tasks queued in this chunk
  int task_cap;
  double* tscratch;  // [search_scratch][tgrid]: captures and records of a search's final partial step
  int tgrid;         // threads of the transit kernel
  // producer captures for the operator kernels
  double* pcap;   // [K][2 npk][18][S]: Kepler-pair parameters
  double* xsnap;  // [K][snaps][3N][S]: see snap_count
  // d(delxv)/dh of a system's last step, for its dq/dt: [2 npk][6][S]
  double* dh;
  double* vsnap;  // [2][3N][S]: v at the two drifts of a system's last step, for its dq/dt
};

// Length of step istep of the system in slot s (nst steps in all).
__device__ __forceinline__ double step_length(const GroupArgs& g, int s, long long istep, long long nst, double h) {
  return (g.hlast && istep == nst - 1) ? g.hlast[s] : h;
}

// Index of the first step of chunk `chunk` for the system in slot s (negative
// while the slot's system is admitted for a later chunk: the request server
// writes a slot's settings while the previous chunk's kernels may still run).
__device__ __forceinline__ long long chunk_first_step(const GroupArgs& g, int chunk, int s) {
  return (long long)chunk * g.K - (g.kbase ? g.kbase[s] : 0);
}

template <int N> int launch_orbit(const GroupArgs& g, int chunk, cudaStream_t st);
template <int N> int launch_jac(const GroupArgs& g, int chunk, cudaStream_t st);
template <int N> int launch_seed(const GroupArgs& g, cudaStream_t st);
template <int N> int launch_transit(const GroupArgs& g, int chunk, cudaStream_t st);
template <int N> int launch_operators(const GroupArgs& g, int chunk, cudaStream_t st);

}  // namespace nbg
