// sm_100a kernels and the level loop of the gate-count search.
//
// Reference semantics (src/cheese.cu): per level, every parent of the frontier is expanded by every candidate
// gate in parent-major, gate-minor order (levels 1249-1377); a child is cut by the W2/W3 window rules (613-632),
// its residual S g^-1 is normalised (145-174), compared with the goal (184-203), pruned by the lower bounds
// (combine of H / structure / support / CX / T, 257-607) and, when alive, keyed by its symmetry class
// (224-241). Survivors are deduplicated by exact class equality keeping the smallest index (1335-1343).
//
// B200 design:
// * one warp per parent (dynamic work counter), parent residual staged in shared memory, all G children walked by
//   the warp; each lane owns entries lane, lane + 32 of the residual;
// * frontier residuals are kept in HBM (1 KB per 3-qubit node with int32 limbs) instead of being replayed from
//   the prefix, so there is no per-level replay pass;
// * each frontier node carries its T bound and CX bound. The T bound (the sde of the Pauli transfer matrix) is
//   unchanged by right multiplication with a Clifford gate (the PTM of a Clifford is a signed permutation), and
//   the F_p operator-Schmidt ranks behind the CX bound are unchanged by one-qubit gates (an invertible local map
//   of the reshaped matrix). So only non-Clifford children (t, tdg) run the 64-point Walsh-Hadamard T bound and
//   only multi-qubit children (cx) run the rank eliminations; the values are identical, not estimates;
// * the T bound accumulates the 2-adic valuations of all transform outputs with two OR words: v = 2 m + d with
//   m = ctz(OR of all coefficients) and d read from bit m of OR((a^c)|(b^d)), the same minimum valuation the
//   reference reads off entry by entry (cheese.cu:419-449);
// * dedupe = stable LSD radix sort of survivor keys, run detection, exact class comparison inside runs (warp per
//   run), then a radix sort of the kept indices restores lexicographic order and a gather builds the next level.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <chrono>
#include <climits>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <stdexcept>
#include <type_traits>

#include "cz_engine.h"
#include "cz_sort.cuh"

namespace cz {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int RC_STOP = -3;        // levels(): stopped after the requested level
constexpr int EXP_WARPS = 8;       // warps per expand block
constexpr int EXP_MINB = 4;        // expand blocks per SM: 32 warps (64 registers; latency-bound code, measured
                                   // 6 % faster than 2 blocks of 128 registers despite a spill of two registers)
constexpr int EXPB_MINB = 3;       // batched: 3 blocks of 80 registers as fast as 4 of 64 with more spills, or 2
constexpr int INHERIT_KMAX = 60;   // the T bound is computed exactly (mod 2^32 / 2^64) only while 2(n + k) <= 128
enum GateKind : uint8_t { GK_GENERAL = 0, GK_ONEQ = 1, GK_PERM = 2 };

constexpr uint8_t QC_NONE = 0xff;
// gcol: kind in the low 3 bits, qubit a in bits 3-4, qubit b in bits 5-6
enum ColKind : uint8_t { COL_UNKNOWN = 0, COL_SAME = 1, COL_S = 2, COL_H = 3, COL_CX = 4 };

// ---------------- device-side spec ----------------
struct DevSpec {
  int n, G, depth, standard, lite, tdiv, ncuts, have_table, nsym, nogoal, gk, ncx;
  int cutmask[CUTMAX], cutsize[CUTMAX], rad[CUTMAX];
  uint64_t w1, w2, w3;                 // w, w^2, w^3 mod p with w = 3^((p-1)/8)
  uint32_t wm[3];                      // w, w^2, w^3 times 2^32 mod p (the CX bound's Montgomery form)
  uint8_t symperm[SYMMAX][8];
  uint8_t symconj[SYMMAX];
  uint8_t gflags[GMAX];
  uint8_t gmask[GMAX];                 // qubits a gate acts on
  uint8_t gkind[GMAX];                 // GK_*: how the child update multiplies by the gate
  uint8_t gph[GMAX][4];                // one-qubit unit gates: w-power of ginv[m][lc] at [2 m + lc] (8: zero)
  uint8_t gmono[GMAX][8];              // GF_UNITMON gates: column c of S g^-1 is column src of S times w^p: src | p << 4
  uint8_t gcol[GMAX];                  // how a Clifford gate permutes the transfer matrix's columns: COL_* | qubit(s)
  int cuts3;                           // 3 qubits and exactly the three one-qubit cuts
  uint8_t qcut[3];                     // per qubit: bit offset in NodeMeta.needs of the cut around it, QC_NONE if none
  uint8_t gperm[GMAX][8];              // permutation gates: local column lc takes local row gperm[lc]
  int goal_id;                         // the goal is the identity with exponent 0 (unitary targets)
  int8_t gnq[GMAX], gik[GMAX];
  int8_t gq[GMAX][3];
  const uint8_t *bad2;
  const uint32_t *bad3;
  const int *cxtable;
  const int4 *ginv;                    // GMAX x 64 local inverse matrices (a, b, c, d as int32)
  const longlong2 *goal;               // N*N entries as (a, b), (c, d) pairs
  int unit;                            // target and gates unitary: every residual is sqrt2^k times a unitary matrix
  int states, m;                       // state targets: m rows (images of the inputs) are searched for the goal rows
  const int *ginfo;                    // state targets: per row the goal's sde, nullity and Schmidt rank per cut
};

// per frontier node: exponent, bounds carried to the children, last two gates (0xff: none), H structure (bit 0:
// hs = 2) with the mask of qubits acted on non-trivially (bits 1..3), per-cut CX needs (2 bits per cut), and the columns
// of the Pauli transfer matrix with an entry of sde T (see cols_t_least; 0: not known)
struct NodeMeta { int16_t k; uint8_t T, c2, g1, g2, hsn, needs; uint64_t cols; };
static_assert(sizeof(NodeMeta) == 16, "node record");

struct DevStats {
  unsigned long long w2, w3, dead, alive, found, first_found, n_surv, t_evals, children, work, full;
  unsigned int ovf, surv_overflow;
  unsigned long long n_work, n_kept;
  unsigned long long n_tq, n_left;    // deferred T evaluations queued; those the packed form left to the general one
  unsigned int sort_err, pad;         // a dedupe sort's look-back gave up (its result is not used)
  unsigned long long work2;           // parent counter of the level kernel's second part (multi-qubit gates)
};

// A T-bound evaluation deferred from the level kernel to k_tbound: the parent, up to two children that share one
// T bound (odd diagonals on one qubit: P T_q = (P Tdg_q) S_q with S_q Clifford), and the bounds already known
// (k, the CX bound, its per-cut needs and the H structure are the parent's for these one-qubit diagonal gates).
struct TQEntry {
  unsigned long long p;
  int16_t k;
  uint8_t n, g[2], c2, needs, hs, ntriv[2];
  uint8_t pad[4];
};
static_assert(sizeof(TQEntry) == 24, "T queue entry layout");

template <typename ST> struct ExpandArgs {
  long long m;
  int t, rem, keep;
  int split;                       // warps that share a parent's candidates
  const Z4<ST> *R;
  const NodeMeta *meta;
  DevStats *st;
  unsigned long long cap;
  uint64_t *sh1, *sh2, *sidx;
  NodeMeta *smeta;
  TQEntry *tq;                     // deferred T evaluations (nullptr: in place)
  unsigned long long tqcap;
  const struct GoalShort *gshort = nullptr;   // the level's goal pass (nullptr: none); a complete hit skips it
};

// The goal pass of a level: the parents whose stored lower bound is <= 1 (no other parent has a child equal to the
// goal: its bounds are sound), listed with their children tested for the goal before the level runs. When it finds
// the goal, the level is the found level: it prints no statistics line, so the bounds of its other children are
// never needed.
struct GoalShort {
  unsigned long long count, found, first;   // candidates (all, even past the list's room), goal children, first one
  unsigned int ovf, pad;
};
constexpr unsigned GOAL_LIST = 1u << 16;

// ---------------- asynchronous copies (cp.async: global -> shared, 16 bytes, bypassing registers) ----------------
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int K> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(K) : "memory");
}

// ---------------- arithmetic helpers ----------------
template <typename ST> __device__ __forceinline__ bool zz(const Z4<ST> &x) { return !(x.a | x.b | x.c | x.d); }
template <typename ST> __device__ __forceinline__ bool zq(const Z4<ST> &x, const Z4<ST> &y) {
  return x.a == y.a && x.b == y.b && x.c == y.c && x.d == y.d;
}
template <typename ST> __device__ __forceinline__ Z4<ST> zcj(const Z4<ST> &x) { return {x.a, (ST)-x.d, (ST)-x.c, (ST)-x.b}; }
template <typename U, typename ST> __device__ __forceinline__ Z4<U> toU(const Z4<ST> &x) {
  return {(U)(int64_t)x.a, (U)(int64_t)x.b, (U)(int64_t)x.c, (U)(int64_t)x.d};
}
template <typename U> __device__ __forceinline__ Z4<U> umul(const Z4<U> &x, const Z4<U> &y) {
  return {(U)(x.a * y.a - x.b * y.d - x.c * y.c - x.d * y.b), (U)(x.a * y.b + x.b * y.a - x.c * y.d - x.d * y.c),
          (U)(x.a * y.c + x.b * y.b + x.c * y.a - x.d * y.d), (U)(x.a * y.d + x.b * y.c + x.c * y.b + x.d * y.a)};
}
template <typename U> __device__ __forceinline__ Z4<U> uadd(const Z4<U> &x, const Z4<U> &y) {
  return {(U)(x.a + y.a), (U)(x.b + y.b), (U)(x.c + y.c), (U)(x.d + y.d)};
}
template <typename U> __device__ __forceinline__ Z4<U> usub(const Z4<U> &x, const Z4<U> &y) {
  return {(U)(x.a - y.a), (U)(x.b - y.b), (U)(x.c - y.c), (U)(x.d - y.d)};
}
template <typename U> __device__ __forceinline__ Z4<U> ushfl(const Z4<U> &x, int m) {
  return {__shfl_xor_sync(FULL, x.a, m), __shfl_xor_sync(FULL, x.b, m), __shfl_xor_sync(FULL, x.c, m),
          __shfl_xor_sync(FULL, x.d, m)};
}
__device__ __forceinline__ uint64_t fmix64(uint64_t h) {
  h ^= h >> 33; h *= 0xff51afd7ed558ccdULL; h ^= h >> 33; h *= 0xc4ceb9fe1a85ec53ULL; h ^= h >> 33;
  return h;
}
// ---------------- per-warp bound evaluations (child residual S in shared memory) ----------------

// ---- T bound: max(0, max over the nonzero PTM entries of their sde) (cheese.cu:397-449) ----
// PTM entry (f, z) up to a unit: X_f(z) = sum_e (-1)^{e.z} Q_f[e], Q_f[e] = S[e ^ f] conj(S[e]), e and f running over
// the E = N^2 (row, column) index pairs. Computed in Z[w] mod 2^b (b = 32 while 2 (n + k) <= 64, else 64): the
// valuations are read off the low bits, as the reference does.
//
// One lane per pair f != 0, its transforms in registers. For f != 0, Q_f[e ^ f] = conj Q_f[e], so over a subgroup H
// of index 2 that misses f, X_f(z) = sum_{e in H} (-1)^{e.z} (Q + (-1)^{f.z} conj Q)[e]: with Q = a + b w + c w^2 +
// d w^3, Q + conj Q = 2a + (b - d) sqrt2 and Q - conj Q = i (2c + (b + d) sqrt2), so four real transforms over the
// E/2 points of H (of a, c, b - d, b + d) give every output, and an output 2A + X sqrt2 has valuation
// min(2 v2(A) + 2, 2 v2(X) + 1). H is {e < E/2} when f has its top bit, else {e : bit j of e is 0} with j the lowest
// set bit of f; point i of H is e(i) = i with a 0 bit inserted at j (a linear map, so the transform over i is the
// transform over H). With 32 lanes a round takes 32 pairs (f = lane + 32 r); f = 0 (Q = |S|^2 = alpha + beta sqrt2,
// one 64-point transform each) is done by the whole warp, each lane holding points lane + 32 t.
// Valuations fold into OR words: m = ctz(OR of 2A, X, alpha, beta over all outputs) is the least 2-adic valuation,
// and v = 2 m + 1 unless bit m is set in the OR of the 2A and alpha outputs (then v = 2 m).
// PASSES splits the four components into passes (fewer live registers, the products recomputed per pass).
template <typename U> __device__ __forceinline__ U pair_component(int comp, const Z4<U> &x, const Z4<U> &y) {
  switch (comp) {   // the coordinates of x conj(y): a, c, b - d, b + d
    case 0: return y.a * x.a + y.b * x.b + y.c * x.c + y.d * x.d;
    case 1: return y.a * x.c + y.b * x.d - y.c * x.a - y.d * x.b;
    case 2: return (y.b - y.d) * x.a + (y.a + y.c) * x.b + (y.b + y.d) * x.c - (y.a - y.c) * x.d;
    default: return (y.a - y.c) * x.b + (y.b - y.d) * x.c + (y.a + y.c) * x.d - (y.b + y.d) * x.a;
  }
}
// the pairs of one round: f (f = 0 skipped) with point map e(i) = insert a 0 at bit j of i
template <int NQ, typename U, int PASSES, typename ST>
__device__ __forceinline__ void tbound_round(const Z4<ST> *S, int f, U &P, U &Q) {
  constexpr int E = 1 << (2 * NQ), HP = E / 2, CPP = 4 / PASSES;
  static_assert(4 % PASSES == 0, "passes split the four components evenly");
  if (f == 0) return;
  const int lomask = (f & HP) ? E - 1 : (f & -f) - 1;   // bits below the inserted 0
#pragma unroll 1
  for (int pass = 0; pass < PASSES; pass++) {
    U v[CPP][HP];
#pragma unroll
    for (int i = 0; i < HP; i++) {
      const int e = (i & lomask) | ((i & ~lomask) << 1);
      const Z4<U> y = toU<U>(S[e]), x = toU<U>(S[e ^ f]);
#pragma unroll
      for (int c = 0; c < CPP; c++) v[c][i] = pair_component<U>(pass * CPP + c, x, y);
    }
#pragma unroll
    for (int h = 1; h < HP; h <<= 1)
#pragma unroll
      for (int i = 0; i < HP; i++)
        if (!(i & h)) {
#pragma unroll
          for (int c = 0; c < CPP; c++) {
            const U u = v[c][i], w = v[c][i | h];
            v[c][i] = u + w;
            v[c][i | h] = u - w;
          }
        }
#pragma unroll
    for (int c = 0; c < CPP; c++) {
      U o = 0;
#pragma unroll
      for (int i = 0; i < HP; i++) o |= v[c][i];
      if (pass * CPP + c < 2) P |= o;
      else Q |= o;
    }
  }
}
template <int NQ, typename U, int PASSES, typename ST>
__device__ __forceinline__ int tbound_lanes(const Z4<ST> *S, int k, int lane) {
  constexpr int E = 1 << (2 * NQ);
  U P = 0, Q = 0;
#pragma unroll 1
  for (int f = lane; f < E; f += 32) tbound_round<NQ, U, PASSES>(S, f, P, Q);
  // f = 0: alpha = |y|^2 real part, beta its sqrt2 part, transformed over all E points across the warp
  constexpr int PL = E > 32 ? E / 32 : 1;   // points per lane
  U al[PL], be[PL];
#pragma unroll
  for (int t = 0; t < PL; t++) {
    const int e = lane + 32 * t;
    const Z4<U> y = e < E ? toU<U>(S[e]) : Z4<U>{0, 0, 0, 0};
    al[t] = y.a * y.a + y.b * y.b + y.c * y.c + y.d * y.d;
    be[t] = y.a * y.b + y.b * y.c + y.c * y.d - y.d * y.a;
  }
#pragma unroll
  for (int h = 1; h < PL; h <<= 1)
#pragma unroll
    for (int t = 0; t < PL; t++)
      if (!(t & h)) {
        U u = al[t], w = al[t | h]; al[t] = u + w; al[t | h] = u - w;
        u = be[t]; w = be[t | h]; be[t] = u + w; be[t | h] = u - w;
      }
  U R1 = 0, R2 = 0;
#pragma unroll
  for (int t = 0; t < PL; t++) {
#pragma unroll
    for (int h = 1; h < 32 && h < E; h <<= 1) {
      const U oa = __shfl_xor_sync(FULL, al[t], h), ob = __shfl_xor_sync(FULL, be[t], h);
      al[t] = (lane & h) ? oa - al[t] : al[t] + oa;
      be[t] = (lane & h) ? ob - be[t] : be[t] + ob;
    }
    R1 |= al[t] | be[t];
    R2 |= al[t];
  }
#pragma unroll
  for (int m = 16; m; m >>= 1) {
    P |= __shfl_xor_sync(FULL, P, m); Q |= __shfl_xor_sync(FULL, Q, m);
    R1 |= __shfl_xor_sync(FULL, R1, m); R2 |= __shfl_xor_sync(FULL, R2, m);
  }
  const U O1 = (U)(P << 1) | Q | R1, O2 = (U)(P << 1) | R2;
  if (!O1) return 0;
  const int mv = sizeof(U) == 8 ? __ffsll((long long)O1) - 1 : __ffs((int)O1) - 1;
  const int v = 2 * mv + (((O2 >> mv) & 1) ? 0 : 1);
  const int top = 2 * (NQ + k);
  return top - v > 0 ? top - v : 0;
}
// ---- columns of the transfer matrix that reach the T bound (3 qubits) ----
// (Of the T evaluations of the budget 12 proofs 86 % are decided from these 64 bits before they are queued.)
// Column (zc, fc) belongs to the input Pauli with X part fc and Z part zc and is bit 8 zc + fc of a 64-bit mask. M holds the
// columns with an entry of sde T. Right multiplication by a Clifford permutes columns, so M follows along. A T on qubit q
// leaves the columns with fc_q = 0 and turns a pair (zc, zc ^ 1 << q) with fc_q = 1 into (u +- w) / sqrt2: where one of
// the pair has an entry of sde T and the other none, u +- w has one of sde T and the child's bound is T + 1; and an entry
// of sde T in an unchanged column keeps the child's bound at T or more.
__device__ __forceinline__ uint64_t cols_x0(int q) {   // fc_q = 0
  return q == 0 ? 0x5555555555555555ULL : (q == 1 ? 0x3333333333333333ULL : 0x0f0f0f0f0f0f0f0fULL);
}
__device__ __forceinline__ uint64_t cols_z0(int q) {   // zc_q = 0
  return q == 0 ? 0x00ff00ff00ff00ffULL : (q == 1 ? 0x0000ffff0000ffffULL : 0x00000000ffffffffULL);
}
__device__ __forceinline__ uint64_t cols_flip_z(uint64_t M, int q) {   // zc -> zc ^ 1 << q
  const uint64_t m = cols_z0(q);
  return ((M & m) << (8 << q)) | ((M >> (8 << q)) & m);
}
// the least T bound of the child of an odd diagonal on qubit q
__device__ __forceinline__ int cols_t_least(uint64_t M, int T, int q) {
  if (!M) return T - 1;
  const uint64_t x0 = cols_x0(q);
  if ((M ^ cols_flip_z(M, q)) & ~x0) return T + 1;
  return (M & x0) ? T : T - 1;
}
// the columns after right multiplication with a Clifford gate (gcol code)
__device__ __forceinline__ uint64_t cols_after(uint64_t M, int code) {
  const int a = (code >> 3) & 3, b = (code >> 5) & 3;
  switch (code & 7) {
    case COL_SAME: return M;
    case COL_S: {                                        // X <-> Y on a
      const uint64_t x0 = cols_x0(a);
      return (M & x0) | (cols_flip_z(M, a) & ~x0);
    }
    case COL_H: {                                        // X <-> Z on a: bits a and 3 + a of the index exchanged
      const int d = 7 << a;
      const uint64_t x = ((M >> d) ^ M) & ~cols_x0(a) & cols_z0(a);
      return M ^ x ^ (x << d);
    }
    case COL_CX: {                                       // control a, target b: fc_b ^= fc_a, zc_a ^= zc_b
      const uint64_t fa = ~cols_x0(a), fb = cols_x0(b);
      M = (M & ~fa) | ((M & fa & fb) << (1 << b)) | ((M & fa & ~fb) >> (1 << b));
      const uint64_t zb = ~cols_z0(b), za = cols_z0(a);
      return (M & ~zb) | ((M & zb & za) << (8 << a)) | ((M & zb & ~za) >> (8 << a));
    }
    default: return 0;
  }
}

// ---- the same T bound for unitary residuals of small exponent, four components to a register ----
// In a unitary residual (entries sqrt2^k U) sum |entry|^2 per row is 2^k in both embeddings of Z[sqrt2], so an entry's
// coefficients satisfy a^2 + b^2 + c^2 + d^2 <= 2^k, and a transform output X_f(z) = 2^k N PTM(f, z) has |A| <= 2^(n +
// k - 1) and |X| <= 2^(n + k - 1/2). While n + k <= 7 the coefficients and their sums and differences fit in 8 bits
// and so does every output, so the four components of a product are four dp4a of 8-bit words and travel through the
// transform as the base-256 digits of one 32-bit integer (additions are linear in the digits; intermediate digits may
// leave the range, the outputs do not). A digit bias of 128 at point 0 reaches every output, so the output bytes are
// digit + 128: their low 7 bits are the digit's, all that a valuation needs. One lane per pair f as above: 32 x (2
// shared loads, 4 dp4a, 3 shifts) + 80 butterflies, where 32-bit components took 32 x (2 wide loads, 28 multiply-adds)
// + 320 butterflies and four times the registers.
constexpr int PACK_MAX = 7;              // n + k up to which the packed form is exact
__device__ __forceinline__ int pack4(int a, int b, int c, int d) {
  return (int)__byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}
// an entry y as four words of 8-bit coefficients: dot products with x's first word are the components a, c, b - d and
// b + d of x conj(y)
template <typename ST> __device__ __forceinline__ int4 pack_entry(const Z4<ST> &v) {
  const int a = (int)v.a, b = (int)v.b, c = (int)v.c, d = (int)v.d;
  return make_int4(pack4(a, b, c, d), pack4(-c, -d, a, b), pack4(b - d, a + c, b + d, c - a),
                   pack4(-b - d, a - c, b - d, a + c));
}
// The transform of pair f into v (0 for f = 0). Point map as in tbound_round, the inserted 0 at the lowest row bit of f if
// it has one (then the column bits of e, and of the output index, are bits 0 to NQ - 1), else at its lowest column bit.
template <int NQ, bool IDENT>
__device__ __forceinline__ void packed_round(const int4 *Y, const int *X, int f, int (&v)[1 << (2 * NQ - 1)]) {
  constexpr int E = 1 << (2 * NQ), HP = E / 2, ROWS = E - (1 << NQ);
  const int fl = (f & ROWS) ? f & ROWS : f, lomask = IDENT ? E - 1 : ((f & HP) ? E - 1 : (fl & -fl) - 1);
#pragma unroll
  for (int i = 0; i < HP; i++) {
    const int e = IDENT ? i : (i & lomask) | ((i & ~lomask) << 1);
    const int4 y = Y[e];
    const int x = X[e ^ f];              // the first words again, one per bank
    int s = __dp4a(x, y.w, 0);
    s = __dp4a(x, y.z, s << 8);
    s = __dp4a(x, y.y, s << 8);
    v[i] = __dp4a(x, y.x, s << 8);
  }
  v[0] += (int)0x80808080u;
#pragma unroll
  for (int h = 1; h < HP; h <<= 1)
#pragma unroll
    for (int i = 0; i < HP; i++)
      if (!(i & h)) {
        const int u = v[i], w = v[i | h];
        v[i] = u + w;
        v[i | h] = u - w;
      }
}
// the bound from the OR words of the transform outputs: O1 = OR of 2A, X, alpha, beta, O2 = OR of 2A, alpha
template <int NQ> __device__ __forceinline__ int bound_of(unsigned O1, unsigned O2, int k) {
  if (!O1) return 0;
  const int mv = __ffs((int)O1) - 1;
  return max(0, 2 * (NQ + k) - (2 * mv + (((O2 >> mv) & 1) ? 0 : 1)));
}
// bytes (A, C, X, Y) of an OR word to (O1, O2)
__device__ __forceinline__ void unpack_or(unsigned o, unsigned &O1, unsigned &O2) {
  O2 = ((o | (o >> 8)) & 0x7fu) << 1;
  O1 = O2 | (((o >> 16) | (o >> 24)) & 0x7fu);
}
// T bound of the residual packed in Y and X (E words). At 3 qubits the 32 pairs f >= 32 come first: a bound above thr
// already decides the entry (bounds only grow with further pairs); then the rest is left out and the result is a
// lower bound above thr. On the deep proofs 92 % of the entries are dead and these 32 pairs show it for every one.
// cols (3 qubits, when asked for): the columns with an entry of that sde. A lane's outputs of pair (fr, fc) belong to the
// columns (zc, fc); their ORs by zc are joined over fr, and the bit that decides the bound is tested in each.
template <int NQ>
__device__ __forceinline__ int packed_tbound(const int4 *Y, const int *X, int k, int lane, int thr, bool want_cols,
                                             uint64_t &cols) {
  constexpr int E = 1 << (2 * NQ), HP = E / 2, PL = E > 32 ? E / 32 : 1, ZC = 1 << NQ;
  unsigned o = 0, O1, O2, oc[ZC];
  int v[HP];
  cols = 0;
#pragma unroll
  for (int z = 0; z < ZC; z++) oc[z] = 0;
  if constexpr (E == 64) {
    packed_round<NQ, true>(Y, X, 32 + lane, v);
#pragma unroll
    for (int i = 0; i < HP; i++) oc[i & 7] |= (unsigned)v[i];
#pragma unroll
    for (int z = 0; z < 8; z++) o |= oc[z];
    o = __reduce_or_sync(FULL, o);
    unpack_or(o, O1, O2);
    const int T = bound_of<NQ>(O1, O2, k);
    if (T > thr) return T;
  }
  const int f = lane < E ? lane : 0;
  packed_round<NQ, false>(Y, X, f, v);
  unsigned o2 = 0;
#pragma unroll
  for (int i = 0; i < HP; i++) o2 |= (unsigned)v[i];
  if (f) o |= o2;
  if constexpr (E == 64) {
    if (want_cols) {
      if (lane >= 8) {                         // fr != 0: the output index keeps the column bits
#pragma unroll
        for (int i = 0; i < HP; i++) oc[i & 7] |= (unsigned)v[i];
      } else if (lane) {
        // fr = 0: the index lacks column bit j; of the two columns it stands for, the real components (bytes 0 and 2)
        // belong to the one with even fc & zc, the imaginary ones to the other
        const int j = __ffs(lane) - 1, lo = (1 << j) - 1;
        unsigned w[4] = {0, 0, 0, 0};
#pragma unroll
        for (int i = 0; i < HP; i++) w[i & 3] |= (unsigned)v[i];
#pragma unroll
        for (int z = 0; z < 8; z++) {
          const int t = ((z >> (j + 1)) << j) | (z & lo);
          const unsigned wt = (t & 2) ? ((t & 1) ? w[3] : w[2]) : ((t & 1) ? w[1] : w[0]);
          oc[z] |= wt & ((__popc(lane & z) & 1) ? 0xff00ff00u : 0x00ff00ffu);
        }
      }
    }
  }
  // f = 0: alpha + 2^16 beta over all E points across the warp (|alpha| <= 2^7, |beta| < 2^7)
  int q[PL];
#pragma unroll
  for (int t = 0; t < PL; t++) {
    const int4 y = lane + 32 * t < E ? Y[lane + 32 * t] : make_int4(0, 0, 0, 0);
    // beta = ab + bc + cd - da: half of (a, b, c, d) . (b - d, a + c, b + d, c - a)
    q[t] = __dp4a(y.x, y.x, 0) + ((__dp4a(y.x, y.z, 0) >> 1) << 16);
  }
#pragma unroll
  for (int h = 1; h < PL; h <<= 1)
#pragma unroll
    for (int t = 0; t < PL; t++)
      if (!(t & h)) { const int u = q[t], w = q[t | h]; q[t] = u + w; q[t | h] = u - w; }
  unsigned R = 0;
#pragma unroll
  for (int t = 0; t < PL; t++) {
#pragma unroll
    for (int h = 1; h < 32 && h < E; h <<= 1) {
      const int u = __shfl_xor_sync(FULL, q[t], h);
      q[t] = (lane & h) ? u - q[t] : u + q[t];
    }
    R |= (unsigned)(q[t] + 0x8000) ^ 0x8000u;
  }
  o = __reduce_or_sync(FULL, o);
  const unsigned Ra = __reduce_or_sync(FULL, R);
  unpack_or(o, O1, O2);
  O1 |= (Ra & 0xffffu) | (Ra >> 16);
  O2 |= Ra & 0xffffu;
  if constexpr (E == 64) {
    if (want_cols && O1) {
      const int mv = __ffs((int)O1) - 1;
      const bool even = (O2 >> mv) & 1;        // the least valuation is even: 2 A or alpha reaches it, else X or beta
      const unsigned tm = even ? (mv ? 0x0101u << (mv - 1) : 0u) : 0x01010000u << mv;
      R |= __shfl_xor_sync(FULL, R, 8);        // output z of f = 0 is in lane z mod 32: joined over the row bits
      R |= __shfl_xor_sync(FULL, R, 16);
      const unsigned z0 = __ballot_sync(FULL, ((even ? R : R >> 16) >> mv) & 1);
      unsigned half[2] = {0, 0};
#pragma unroll
      for (int z = 0; z < 8; z++) {
        const unsigned has = __ballot_sync(FULL, (oc[z] & tm) != 0);
        half[z >> 2] |= (((has | has >> 8 | has >> 16 | has >> 24) & 0xffu) | ((z0 >> z) & 1u)) << (8 * (z & 3));
      }
      cols = half[0] | (uint64_t)half[1] << 32;
    }
  }
  return bound_of<NQ>(O1, O2, k);
}
// 32-bit residues in one pass (3 qubits: 128 transform values per lane); 64-bit residues (k > 29, rare) one
// component per pass
template <int NQ, typename ST> __device__ __noinline__ int warp_tbound32(const Z4<ST> *S, int k, int lane) {
  return tbound_lanes<NQ, uint32_t, 1>(S, k, lane);
}
template <int NQ, typename ST> __device__ __noinline__ int warp_tbound64(const Z4<ST> *S, int k, int lane) {
  return tbound_lanes<NQ, uint64_t, 4>(S, k, lane);
}
template <int NQ, typename ST> __device__ __forceinline__ int ptm_bound(const Z4<ST> *S, int k, int lane) {
  return 2 * (NQ + k) > 64 ? warp_tbound64<NQ, ST>(S, k, lane) : warp_tbound32<NQ, ST>(S, k, lane);
}

// ---- CX bound (cheese.cu:257-303, 585-597): F_p ranks of the operator-Schmidt matrices across the cuts ----
// F_p arithmetic in Montgomery form with R = 2^32: mont(x, y) = x y / R mod p. A rank only depends on which
// elimination results are zero, and every Montgomery product carries the same factor 1 / R, so the elimination
// v2 <- mont(a, v2) - mont(b, v1) = (a v2 - b v1) / R keeps every rank of the reference's a v2 - b v1.
constexpr uint32_t inv_mod_2_32(uint32_t p) {      // p^-1 mod 2^32 by Newton's iteration (p odd)
  uint32_t x = p;
  for (int i = 0; i < 5; i++) x *= 2u - p * x;
  return x;
}
constexpr uint32_t PRIME_NINV = 0u - inv_mod_2_32(PRIME);
static_assert(PRIME * inv_mod_2_32(PRIME) == 1u, "Montgomery inverse");
__device__ __forceinline__ uint32_t mont(uint32_t x, uint32_t y) {   // x, y < p
  const uint64_t t = (uint64_t)x * y;
  const uint32_t m = (uint32_t)t * PRIME_NINV;
  const uint32_t u = (uint32_t)((t + (uint64_t)m * PRIME) >> 32);
  return u >= PRIME ? u - PRIME : u;
}
__device__ __forceinline__ uint32_t addp(uint32_t x, uint32_t y) { const uint32_t s = x + y; return s >= PRIME ? s - PRIME : s; }
__device__ __forceinline__ uint32_t subp(uint32_t x, uint32_t y) { return x >= y ? x - y : x + PRIME - y; }
template <typename ST> __device__ __forceinline__ uint32_t limb_modp(ST a) {
  const ST r = a % (ST)PRIME;
  return (uint32_t)(r < 0 ? r + (ST)PRIME : r);
}
// x = a + b w + c w^2 + d w^3 mapped to F_p (w -> a primitive 8th root of unity mod p), in normal form:
// mont(b mod p, w R mod p) = b w mod p
template <typename ST> __device__ __forceinline__ uint32_t to_fp(const Z4<ST> &x, const DevSpec &sp) {
  return addp(addp(limb_modp(x.a), mont(limb_modp(x.b), sp.wm[0])),
              addp(mont(limb_modp(x.c), sp.wm[1]), mont(limb_modp(x.d), sp.wm[2])));
}
// The bound from the per-cut needs ceil(log2 rank) through the CX table. Cuts a gate does not cross keep their
// parent's need (a gate inside one side is a local map); needs_in = the parent's packed needs, gmask = the gate's
// qubits (0: every cut recomputed). Every cut has one qubit (at most 3 qubits), so its matrix is 4 x E/4: rows
// (output bit, input bit) of the cut qubit, columns those of the other qubits. The matrices of 32 / (E/4) cuts are
// eliminated side by side, one column per lane: per row a ballot finds the group's pivot column, and the rows
// below are reduced by it. Returns the bound and packs the child's needs (2 bits per cut) into needs_out.
// elem(o, i): the F_p image of the residual's entry in row o, column i.
template <int NQ, typename Elem>
__device__ __forceinline__ int warp_cx_elems(Elem elem, const DevSpec &sp, int lane, int gmask, int needs_in,
                                             int &needs_out) {
  constexpr int N = 1 << NQ, CC = N * N / 4 > 0 ? N * N / 4 : 1, SLOTS = 32 / CC, ALLQ = N - 1;
  static_assert(NQ <= 3, "cuts of one qubit: 4 x E/4 matrices within a warp");
  const bool inherit = sp.ncuts <= 4 && gmask;
  unsigned todo = 0;
  for (int i = 0; i < sp.ncuts; i++) {
    const int A = sp.cutmask[i];
    if (!(inherit && (!(gmask & A) || !(gmask & ~A & ALLQ)))) todo |= 1u << i;
  }
  uint64_t fresh = 0;                        // 3 bits per recomputed cut: its need
  const int slot = lane / CC, col = lane % CC;
  while (todo) {
    int mycut = -1;
    for (int s2 = 0; s2 < SLOTS; s2++) {      // the group's cuts: the lowest SLOTS cuts still to do
      const int c = todo ? __ffs(todo) - 1 : -1;
      if (s2 == slot) mycut = c;
      todo &= todo - 1;
    }
    const int A = mycut >= 0 ? sp.cutmask[mycut] : 0;
    uint32_t v[4];
#pragma unroll
    for (int rr = 0; rr < 4; rr++) {
      int o = 0, i = 0, nb = 0;
#pragma unroll
      for (int q = 0; q < NQ; q++) {
        if ((A >> q) & 1) { o |= ((rr >> 1) & 1) << q; i |= (rr & 1) << q; }
        else { o |= ((col >> (NQ - 1 + nb)) & 1) << q; i |= ((col >> nb) & 1) << q; nb++; }
      }
      v[rr] = mycut >= 0 ? elem(o, i) : 0u;
    }
    const unsigned group = (CC >= 32 ? FULL : ((1u << CC) - 1u)) << (slot * CC);
    int rank = 0;
#pragma unroll
    for (int rr = 0; rr < 4; rr++) {
      const unsigned bal = __ballot_sync(FULL, v[rr] != 0) & group;
      const int piv = bal ? __ffs(bal) - 1 : lane;
      const uint32_t a = __shfl_sync(FULL, v[rr], piv);
#pragma unroll
      for (int r2 = rr + 1; r2 < 4; r2++) {
        const uint32_t b = __shfl_sync(FULL, v[r2], piv);
        if (bal) v[r2] = subp(mont(a, v[r2]), mont(b, v[rr]));
      }
      rank += bal != 0;
    }
    const int need = rank <= 1 ? 0 : (rank == 2 ? 1 : 2);
    for (int s2 = 0; s2 < SLOTS; s2++) {
      const int c = __shfl_sync(FULL, mycut, s2 * CC), nd = __shfl_sync(FULL, need, s2 * CC);
      if (c >= 0) fresh |= (uint64_t)nd << (3 * c);
    }
  }
  int idx = 0, mult = 1, mx = 0, packed = 0;
  for (int i = 0; i < sp.ncuts; i++) {
    const int A = sp.cutmask[i];
    int need;
    if (inherit && (!(gmask & A) || !(gmask & ~A & ALLQ))) need = (needs_in >> (2 * i)) & 3;
    else need = min((int)((fresh >> (3 * i)) & 7), sp.rad[i] - 1);
    if (i < 4) packed |= (need & 3) << (2 * i);
    idx += need * mult;
    mult *= sp.rad[i];
    mx = max(mx, need);
  }
  needs_out = packed;
  return sp.have_table && idx < sp.ncx ? __ldg(&sp.cxtable[idx]) : mx;
}

template <int NQ, typename ST>
__device__ __forceinline__ int warp_cx_bound(const Z4<ST> *S, const DevSpec &sp, int lane, int gmask, int needs_in,
                                             int &needs_out) {
  return warp_cx_elems<NQ>([&](int o, int i) { return to_fp(S[(o << NQ) + i], sp); }, sp, lane, gmask, needs_in, needs_out);
}

// The same for a two-qubit column permutation of a 3-qubit residual with one cut around each qubit (sp.cuts3): the two
// crossed cuts side by side, one per half warp, from the parent's F_p image F with its columns permuted (mono: source column
// per column). A need only tells ranks 1, 2 and 3 or more apart, so three of the four rows are eliminated first and the last
// one only where they left a rank below 3 (rarely): 54 instead of 132 instructions.
__device__ __forceinline__ int warp_cx_pair(const uint32_t *F, const uint8_t *mono, const DevSpec &sp, int lane, int q0, int q1,
                                            int needs_in, int &needs_out) {
  const int q = lane < 16 ? q0 : q1, col = lane & 15, lo = (1 << q) - 1;
  auto wide = [&](int x) { return ((x & ~lo) << 1) | (x & lo); };      // a 0 inserted at bit q
  const int i0 = wide(col & 3), o0 = wide(col >> 2) << 3, s0 = mono[i0] & 15, s1 = mono[i0 | (1 << q)] & 15, o1 = o0 | (8 << q);
  uint32_t v[3] = {F[o0 + s0], F[o0 + s1], F[o1 + s0]}, w = F[o1 + s1];
  const unsigned half = lane < 16 ? 0xffffu : 0xffff0000u;
  uint32_t pa[3];
  int pl[3], rank = 0;
  bool used[3];
#pragma unroll
  for (int r = 0; r < 3; r++) {
    const unsigned bal = __ballot_sync(FULL, v[r] != 0) & half;
    used[r] = bal != 0;
    pl[r] = bal ? __ffs(bal) - 1 : lane;
    rank += used[r];
    pa[r] = __shfl_sync(FULL, v[r], pl[r]);
#pragma unroll
    for (int r2 = r + 1; r2 < 3; r2++) {
      const uint32_t b = __shfl_sync(FULL, v[r2], pl[r]);
      if (used[r]) v[r2] = subp(mont(pa[r], v[r2]), mont(b, v[r]));
    }
  }
  if (!__all_sync(FULL, rank == 3)) {
#pragma unroll
    for (int r = 0; r < 3; r++) {
      const uint32_t b = __shfl_sync(FULL, w, pl[r]);
      if (used[r]) w = subp(mont(pa[r], w), mont(b, v[r]));
    }
    rank += (__ballot_sync(FULL, w != 0) & half) != 0;
  }
  const int need = rank <= 1 ? 0 : (rank == 2 ? 1 : 2);
  const int n0 = __shfl_sync(FULL, need, 0), n1 = __shfl_sync(FULL, need, 16), b0 = sp.qcut[q0], b1 = sp.qcut[q1];
  const int needs = (needs_in & ~(3 << b0) & ~(3 << b1)) | n0 << b0 | n1 << b1;
  needs_out = needs;
  const int c0 = needs & 3, c1 = (needs >> 2) & 3, c2 = (needs >> 4) & 3, idx = c0 + 3 * c1 + 9 * c2;
  return sp.have_table && idx < sp.ncx ? __ldg(&sp.cxtable[idx]) : max(c0, max(c1, c2));
}

// the least c + max(h + t, supp - 2 c) over c >= c2 (cheese.cu:599-607): the second term falls by 2 per step of c until
// it meets h + t, so the least c with supp - 2 c <= h + t is best, or c2 if that is larger
__device__ __forceinline__ int combine(int h, int t, int c2, int supp) {
  return max(c2, (max(supp - h - t, 0) + 1) >> 1) + h + t;
}

// x times w^p (p < 8): a signed rotation of the coefficients
template <typename ST> __device__ __forceinline__ Zw mul_unit(const Z4<ST> &x, int p) {
  Zw r;
  switch (p & 3) {
    case 0: r = Zw{x.a, x.b, x.c, x.d}; break;
    case 1: r = Zw{-(int64_t)x.d, x.a, x.b, x.c}; break;
    case 2: r = Zw{-(int64_t)x.c, -(int64_t)x.d, x.a, x.b}; break;
    default: r = Zw{-(int64_t)x.b, -(int64_t)x.c, -(int64_t)x.d, x.a};
  }
  if (p & 4) r = Zw{-r.a, -r.b, -r.c, -r.d};
  return r;
}
// the same in int32, branch free: rotate by 2 if p & 2, by 1 if p & 1, negate if p & 4
__device__ __forceinline__ int4 mul_unit32(int4 x, int p) {
  int4 y = (p & 2) ? make_int4(-x.z, -x.w, x.x, x.y) : x;
  y = (p & 1) ? make_int4(-y.w, y.x, y.y, y.z) : y;
  return (p & 4) ? make_int4(-y.x, -y.y, -y.z, -y.w) : y;
}

// the same for any limb type
template <typename ST> __device__ __forceinline__ Z4<ST> unit_mul(const Z4<ST> &x, int p) {
  Z4<ST> y = (p & 2) ? Z4<ST>{(ST)-x.c, (ST)-x.d, x.a, x.b} : x;
  y = (p & 1) ? Z4<ST>{(ST)-y.d, y.a, y.b, y.c} : y;
  return (p & 4) ? Z4<ST>{(ST)-y.a, (ST)-y.b, (ST)-y.c, (ST)-y.d} : y;
}
// entry lane + 32 j of P g^-1 for a GF_UNITMON gate, mono = its gmono byte for the lane's column (entries lane and
// lane + 32 are in one column)
template <int NQ, typename ST> __device__ __forceinline__ Z4<ST> mono_entry(const Z4<ST> *P, int mono, int lane, int j) {
  constexpr int N = 1 << NQ;
  return unit_mul(P[((lane & ~(N - 1)) | (mono & 15)) + 32 * j], mono >> 4);
}

// normalise the lane's two entries (sqrt2 division while every entry allows it) and store them; returns k
template <int NQ, typename ST, typename V>
__device__ __forceinline__ int finish_child(V (&v)[2], const int (&ei)[2], int k, Z4<ST> *C, int lane, bool &ovf) {
  while (k > 0) {
    const bool ok = (ei[0] < 0 || zdiv2ok(v[0])) && (ei[1] < 0 || zdiv2ok(v[1]));
    if (!__all_sync(FULL, ok)) break;
    v[0] = zdown(v[0]);
    v[1] = zdown(v[1]);
    k--;
  }
  bool of = false;
#pragma unroll
  for (int j = 0; j < 2; j++) {
    if (ei[j] < 0) continue;
    if (sizeof(ST) == 4 && !(fits32(v[j].a) && fits32(v[j].b) && fits32(v[j].c) && fits32(v[j].d))) of = true;
    C[ei[j]] = Z4<ST>{(ST)v[j].a, (ST)v[j].b, (ST)v[j].c, (ST)v[j].d};
  }
  ovf = __any_sync(FULL, of);
  __syncwarp();
  return k;
}
// int32 helpers for the fast path (exact: callers guarantee |coefficient| <= 2^28)
struct I4 { int a, b, c, d; };
__device__ __forceinline__ bool zdiv2ok(const I4 &x) { return !((x.a - x.c) & 1) && !((x.b - x.d) & 1); }
__device__ __forceinline__ I4 zdown(const I4 &x) { return {(x.b - x.d) >> 1, (x.a + x.c) >> 1, (x.b + x.d) >> 1, (x.c - x.a) >> 1}; }
__device__ __forceinline__ bool fits32(int) { return true; }

// one-qubit unit gate: the two outputs of a column pair (entries ei of P), w-powers ph of the inverse at [2 m + lc]
template <typename ST> __device__ __forceinline__ void oneq_pair(const Z4<ST> *P, const int (&ei)[2], const uint8_t *ph, I4 (&v)[2]) {
  const int4 *P4 = (const int4 *)P;
  const int4 x0 = P4[ei[0]], x1 = P4[ei[1]], z = make_int4(0, 0, 0, 0);
  const int p00 = ph[0], p01 = ph[1], p10 = ph[2], p11 = ph[3];
  const int4 a0 = p00 < 8 ? mul_unit32(x0, p00) : z, a1 = p10 < 8 ? mul_unit32(x1, p10) : z;
  const int4 b0 = p01 < 8 ? mul_unit32(x0, p01) : z, b1 = p11 < 8 ? mul_unit32(x1, p11) : z;
  v[0] = I4{a0.x + a1.x, a0.y + a1.y, a0.z + a1.z, a0.w + a1.w};
  v[1] = I4{b0.x + b1.x, b0.y + b1.y, b0.z + b1.z, b0.w + b1.w};
}
// sqrt2 division of the warp's entries (zeros divide) while every one allows it; returns the exponent
__device__ __forceinline__ int normalise_pair(I4 (&v)[2], int k) {
  while (k > 0 && __all_sync(FULL, zdiv2ok(v[0]) && zdiv2ok(v[1]))) {
    v[0] = zdown(v[0]);
    v[1] = zdown(v[1]);
    k--;
  }
  return k;
}

// child residual C = P g^-1, general gate: multiplies the local matrix out over Z[w] in int64
template <int NQ, typename ST>
__device__ __noinline__ int child_general(const Z4<ST> *P, Z4<ST> *C, int g, int kp, const DevSpec *sp, int lane,
                                          bool &ovf) {
  constexpr int N = 1 << NQ, E = N * N;
  Zw v[2] = {Zw{0, 0, 0, 0}, Zw{0, 0, 0, 0}};
  int ei[2] = {-1, -1};
  const int kind = sp->gkind[g];
  const int nq = sp->gnq[g], L = 1 << nq;
  const int q0 = sp->gq[g][0], q1 = nq > 1 ? sp->gq[g][1] : 0, q2 = nq > 2 ? sp->gq[g][2] : 0;
  const int mask = (1 << q0) | (nq > 1 ? 1 << q1 : 0) | (nq > 2 ? 1 << q2 : 0);
  if (kind == GK_ONEQ) {
    const int lo = (1 << q0) - 1;
    if (lane < E / 2) {
      ei[0] = ((lane & ~lo) << 1) | (lane & lo);
      ei[1] = ei[0] | (1 << q0);
      const Z4<ST> x0 = P[ei[0]], x1 = P[ei[1]];
      const int p00 = sp->gph[g][0], p01 = sp->gph[g][1], p10 = sp->gph[g][2], p11 = sp->gph[g][3];
      if (p00 < 8) v[0] = zadd(v[0], mul_unit(x0, p00));
      if (p10 < 8) v[0] = zadd(v[0], mul_unit(x1, p10));
      if (p01 < 8) v[1] = zadd(v[1], mul_unit(x0, p01));
      if (p11 < 8) v[1] = zadd(v[1], mul_unit(x1, p11));
    }
  } else {
    for (int j = 0; j < 2; j++) {
      const int e = lane + 32 * j;
      if (e >= E) continue;
      ei[j] = e;
      const int r = e >> NQ, col = e & (N - 1), base = col & ~mask;
      int lc = (col >> q0) & 1;
      if (nq > 1) lc |= ((col >> q1) & 1) << 1;
      if (nq > 2) lc |= ((col >> q2) & 1) << 2;
      const int4 *gi = sp->ginv + g * 64;
      for (int m = 0; m < L; m++) {
        const int4 gm = __ldg(&gi[m * L + lc]);
        if (!(gm.x | gm.y | gm.z | gm.w)) continue;
        int x = base | ((m & 1) << q0);
        if (nq > 1) x |= ((m >> 1) & 1) << q1;
        if (nq > 2) x |= ((m >> 2) & 1) << q2;
        const Z4<ST> sv = P[r * N + x];
        v[j] = zadd(v[j], zmul(Zw{(int64_t)sv.a, (int64_t)sv.b, (int64_t)sv.c, (int64_t)sv.d},
                               Zw{(int64_t)gm.x, (int64_t)gm.y, (int64_t)gm.z, (int64_t)gm.w}));
      }
    }
  }
  return finish_child<NQ, ST>(v, ei, kp + sp->gik[g], C, lane, ovf);
}

// child residual C = P g^-1, normalised; returns its exponent, sets ovf when a limb leaves the storage type.
// Fast path (int32 limbs, |coefficient| <= 2^28, i.e. parent k <= 56): one-qubit gates whose inverse has only zero
// / w-power entries (x z h s sdg t tdg) pair the entries that differ in the gate's column bit, so each lane owns
// both inputs of its two outputs and every product is a signed rotation; permutation gates (cx, ccx) copy.
// Anything else goes through child_general.
// PART 1: g acts on one qubit (its kind is GK_ONEQ or GK_GENERAL); PART 2: on more (GK_PERM or GK_GENERAL); any
// other kind goes the general way, so each part's code holds one specialised update
template <int NQ, typename ST, int PART = 0>
__device__ __forceinline__ int warp_child(const Z4<ST> *P, Z4<ST> *C, int g, int kp, const DevSpec &sp,
                                          const DevSpec *sps, int lane, bool &ovf) {
  constexpr int N = 1 << NQ, E = N * N;
  const int kind = sp.gkind[g];
  if (sizeof(ST) != 4 || kp > 56 || kind == GK_GENERAL || (PART == 1 && kind != GK_ONEQ) ||
      (PART == 2 && kind != GK_PERM))
    return child_general<NQ, ST>(P, C, g, kp, sps, lane, ovf);
  I4 v[2] = {I4{0, 0, 0, 0}, I4{0, 0, 0, 0}};
  int ei[2] = {-1, -1};
  const int4 *P4 = (const int4 *)P;
  if (kind == GK_ONEQ) {
    const int q = sp.gq[g][0], lo = (1 << q) - 1;
    if (lane < E / 2) {
      ei[0] = ((lane & ~lo) << 1) | (lane & lo);
      ei[1] = ei[0] | (1 << q);
      oneq_pair(P, ei, sp.gph[g], v);
    }
  } else {   // GK_PERM
    const int nq = sp.gnq[g];
    const int q0 = sp.gq[g][0], q1 = nq > 1 ? sp.gq[g][1] : 0, q2 = nq > 2 ? sp.gq[g][2] : 0;
    const int mask = (1 << q0) | (nq > 1 ? 1 << q1 : 0) | (nq > 2 ? 1 << q2 : 0);
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const int e = lane + 32 * j;
      if (e >= E) continue;
      ei[j] = e;
      const int r = e >> NQ, col = e & (N - 1), base = col & ~mask;
      int lc = (col >> q0) & 1;
      if (nq > 1) lc |= ((col >> q1) & 1) << 1;
      if (nq > 2) lc |= ((col >> q2) & 1) << 2;
      const int m = sp.gperm[g][lc];
      int x = base | ((m & 1) << q0);
      if (nq > 1) x |= ((m >> 1) & 1) << q1;
      if (nq > 2) x |= ((m >> 2) & 1) << q2;
      const int4 sv = P4[r * N + x];
      v[j] = I4{sv.x, sv.y, sv.z, sv.w};
    }
  }
  return finish_child<NQ, ST>(v, ei, kp + sp.gik[g], C, lane, ovf);
}

template <int NQ, typename ST> __device__ bool warp_goal(const Z4<ST> *S, int k, const DevSpec &sp, int lane);

// goal test, H structure (2 when S is monomial with a non-affine permutation, cheese.cu:322-338) and the mask of
// qubits S acts on non-trivially (support = its popcount, cheese.cu:305-319) in one pass: each lane reads entries
// lane and lane + 32; the nonzero pattern becomes a 64-bit mask by ballot for the monomial / affine test. Only the
// qubits in test_q are examined for triviality; the others keep the bits of ntriv_in.
struct Cheap { bool goal; int hs, ntriv; };
template <int NQ, typename ST>
__device__ Cheap warp_cheap(const Z4<ST> *S, int k, const DevSpec &sp, int lane, bool maybe_goal, bool need_hs,
                            int test_q, int ntriv_in) {
  constexpr int N = 1 << NQ, E = N * N;
  Z4<ST> x[2];
  bool val[2];
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const int e = lane + 32 * j;
    val[j] = e < E;
    x[j] = val[j] ? S[e] : Z4<ST>{0, 0, 0, 0};
  }
  Cheap out{false, 0, ntriv_in & ~test_q};
  if (maybe_goal) {
    if (sp.goal_id) {
      bool ok = k == 0;
#pragma unroll
      for (int j = 0; j < 2; j++) {
        if (!val[j]) continue;
        const int e = lane + 32 * j, r = e >> NQ, c = e & (N - 1);
        if (r == c ? !(x[j].a == 1 && !x[j].b && !x[j].c && !x[j].d) : !zz(x[j])) ok = false;
      }
      out.goal = __all_sync(FULL, ok);
    } else {
      out.goal = warp_goal<NQ, ST>(S, k, sp, lane);
    }
    if (out.goal) return out;
  }
  if (need_hs) {
    const unsigned b0 = __ballot_sync(FULL, val[0] && !zz(x[0])), b1 = __ballot_sync(FULL, val[1] && !zz(x[1]));
    const uint64_t M = (uint64_t)b0 | ((uint64_t)b1 << 32);
    if (__popcll(M) == N) {                      // monomial iff every column has exactly one nonzero
      int pi[N];
      bool mono = true;
#pragma unroll 1
      for (int c = 0; c < N; c++) {
        uint64_t colm = 0;
#pragma unroll 1
        for (int r = 0; r < N; r++) colm |= ((M >> (r * N + c)) & 1ULL) << r;
        mono = mono && __popcll(colm) == 1;
        pi[c] = __ffsll((long long)colm) - 1;
      }
      if (mono) {
        bool aff = true;
#pragma unroll 1
        for (int j = 0; j < N; j++) {
          int xx = pi[0];
#pragma unroll 1
          for (int i = 0; i < NQ; i++) if ((j >> i) & 1) xx ^= pi[1 << i] ^ pi[0];
          if (pi[j] != xx) aff = false;
        }
        out.hs = aff ? 0 : 2;
      }
    }
  }
#pragma unroll
  for (int q = 0; q < NQ; q++) {
    if (!((test_q >> q) & 1)) continue;
    const int bit = 1 << q;
    bool nt = false;
#pragma unroll
    for (int j = 0; j < 2; j++) {
      if (!val[j]) continue;
      const int e = lane + 32 * j, r = e >> NQ, c = e & (N - 1);
      if ((r ^ c) & bit) { if (!zz(x[j])) nt = true; }
      else if (!((r | c) & bit) && !zq(x[j], S[(r | bit) * N + (c | bit)])) nt = true;
    }
    if (__any_sync(FULL, nt)) out.ntriv |= bit;
  }
  return out;
}

template <int NQ, typename ST> __device__ bool warp_goal(const Z4<ST> *S, int k, const DevSpec &sp, int lane) {
  constexpr int E = (1 << NQ) * (1 << NQ), EPL = E >= 32 ? E / 32 : 1;
  if (k != sp.gk) return false;
  bool ok = true;
#pragma unroll
  for (int j = 0; j < EPL; j++) {
    const int e = lane + 32 * j;
    if (e >= E) continue;
    const longlong2 g0 = __ldg(&sp.goal[2 * e]), g1 = __ldg(&sp.goal[2 * e + 1]);
    const Z4<ST> x = S[e];
    if ((int64_t)x.a != g0.x || (int64_t)x.b != g0.y || (int64_t)x.c != g1.x || (int64_t)x.d != g1.y) ok = false;
  }
  return __all_sync(FULL, ok);
}

// ---------------- state targets (rows j < m: the images of the inputs; cheese.cu:451-583) ----------------
// H: the sde of a row changes by at most 1 per H. T: the stabilizer nullity of a row changes by at most 1 per T and
// not at all under Cliffords. CX: the Schmidt rank of a row across a cut changes by at most a factor 2 per crossing
// two-qubit gate. Ranks are exact (minors in int64 under a coefficient bound), as in the reference.
template <typename ST> __device__ __forceinline__ Zw zw_of(const Z4<ST> &x) { return Zw{x.a, x.b, x.c, x.d}; }
// sqrt2-adic valuation of a nonzero x = a + b w + c w^2 + d w^3 in closed form: 2 = sqrt2^2, and x / 2^m (m the
// least 2-adic valuation of the coefficients) is divisible by sqrt2 exactly when a = c and b = d mod 2.
__device__ __forceinline__ int zval_closed(const Zw &x) {
  const uint64_t o = (uint64_t)(x.a | x.b | x.c | x.d);
  const int m = __ffsll((long long)o) - 1;
  return 2 * m + ((((uint64_t)((x.a ^ x.c) | (x.b ^ x.d)) >> m) & 1) ? 0 : 1);
}
__device__ __forceinline__ int64_t zmax_abs(const Zw &x) {
  const int64_t a = x.a < 0 ? -x.a : x.a, b = x.b < 0 ? -x.b : x.b, c = x.c < 0 ? -x.c : x.c, d = x.d < 0 ? -x.d : x.d;
  return max(max(a, b), max(c, d));
}
__device__ __forceinline__ int warp_imax(int v) {
  for (int m = 16; m; m >>= 1) v = max(v, __shfl_xor_sync(FULL, v, m));
  return v;
}
// fewest crossing two-qubit gates between Schmidt ranks rv (the row's) and rt (the goal's): the rank changes by at
// most a factor 2 per crossing gate, so c = ceil(log2(ceil(hi / lo))); 0 when either rank is unknown (-1) or 0
__device__ __forceinline__ int rank_gates(int rv, int rt) {
  if (rv <= 0 || rt <= 0) return 0;
  const int lo = min(rv, rt), q = (max(rv, rt) + lo - 1) / lo;
  return q > 1 ? 32 - __clz(q - 1) : 0;
}

// ---------------- state targets (rows j < m: the images of the inputs; cheese.cu:451-583) ----------------
// H: the sde of a row changes by at most 1 per H. CX: the Schmidt rank of a row across a cut changes by at most a
// factor 2 per crossing two-qubit gate. T: the stabilizer nullity of a row changes by at most 1 per T and not at all
// under Cliffords. All three are computed exactly, as the reference does (ranks over Q(w), not mod p).
//
// H and CX bounds: h = max over rows of |sde - goal sde|; c2 from the per-cut needs through the CX table. The sde
// part has each lane on entries lane + 32 t (a row = N consecutive lanes, reduced by shuffles). The rank part has
// one lane per (row, cut): the row reshaped to R x C across the cut, with R = 2 at up to 3 qubits (cuts of one
// qubit), has rank 2 when one of its 2 x 2 minors is nonzero, else rank 1 when it is nonzero; a row with a
// coefficient of 2^29 or more has an unknown rank (-1: no bound), like the reference's int64 guard.
template <int NQ, typename ST> __device__ __noinline__ void warp_state_cheap(const Z4<ST> *S, int k, const DevSpec &sp,
                                                                           int lane, int &h, int &c2) {
  static_assert(NQ <= 3, "state bounds: cuts of one qubit (two-row reshapes)");
  constexpr int N = 1 << NQ, E = N * N, PL = E > 32 ? E / 32 : 1;
  const int W = 2 + sp.ncuts;
  int hmax = 0;
#pragma unroll
  for (int t = 0; t < PL; t++) {
    const int e = lane + 32 * t, j = e / N;
    const Zw x = e < E ? zw_of(S[e]) : Zw{0, 0, 0, 0};
    int v = zzero(x) ? 1 << 30 : zval_closed(x);
#pragma unroll
    for (int o = 1; o < N; o <<= 1) v = min(v, __shfl_xor_sync(FULL, v, o));
    if (j < sp.m && e < E && (e & (N - 1)) == 0) {
      const int sde = v == (1 << 30) || k < v ? 0 : k - v;
      hmax = max(hmax, abs(sde - sp.ginfo[j * W]));
    }
  }
  h = warp_imax(hmax);
  int need[CUTMAX];
  for (int c = 0; c < CUTMAX; c++) need[c] = 0;
  for (int it = lane; it < sp.m * sp.ncuts; it += 32) {
    const int j = it / sp.ncuts, c = it % sp.ncuts, A = sp.cutmask[c];
    Zw M[2][N / 2];
    int64_t big = 0;
    bool nonzero = false;
    for (int x = 0; x < N; x++) {
      int ia = 0, ib = 0, nb = 0;
      for (int q = 0; q < NQ; q++) {
        if ((A >> q) & 1) ia = (x >> q) & 1;
        else ib |= ((x >> q) & 1) << nb++;
      }
      M[ia][ib] = zw_of(S[j * N + x]);
      big = max(big, zmax_abs(M[ia][ib]));
      nonzero |= !zzero(M[ia][ib]);
    }
    int rank = nonzero ? 1 : 0;
    if (big >= (1LL << 29)) rank = -1;
    else
      for (int p = 0; p < N / 2 && rank == 1; p++)
        for (int q = p + 1; q < N / 2; q++)
          if (!zeq(zmul(M[0][p], M[1][q]), zmul(M[0][q], M[1][p]))) { rank = 2; break; }
    need[c] = max(need[c], rank_gates(rank, sp.ginfo[j * W + 2 + c]));
  }
  int idx = 0, mult = 1, mx = 0;
  for (int c = 0; c < sp.ncuts; c++) {
    const int nd = min(warp_imax(need[c]), sp.rad[c] - 1);
    idx += nd * mult;
    mult *= sp.rad[c];
    mx = max(mx, nd);
  }
  c2 = sp.have_table && idx < sp.ncx ? __ldg(&sp.cxtable[idx]) : mx;
}
// T bound: max over rows of |stabilizer nullity - the goal's|, nullity = n - log2 of the number of Paulis P with
// <v|P|v> = +-<v|v>. One lane per (row, X part f) (a row = N consecutive lanes): with the Pauli's Z part z,
// <v|P|v> = i^{|f & z|} W(z), W = the N-point Walsh-Hadamard transform over x of conj(v[x ^ f]) v[x], so one small
// transform gives the row's N Paulis of X part f; <v|v> is W(0) of the row's f = 0 lane. Rows with a coefficient of
// 2^27 or more are skipped (the reference's int64 guard; the transform stays below 2^62).
template <int NQ, typename ST> __device__ __noinline__ int warp_state_t(const Z4<ST> *S, const DevSpec &sp, int lane) {
  static_assert(NQ <= 3, "state bounds: one row per N lanes");
  constexpr int N = 1 << NQ, E = N * N, PL = E > 32 ? E / 32 : 1;
  const int W = 2 + sp.ncuts;
  int best = 0;
#pragma unroll
  for (int t = 0; t < PL; t++) {
    const int task = lane + 32 * t, j = task / N, f = task & (N - 1);
    const bool live = task < E && j < sp.m;
    Zw w[N];
    int64_t big = 0;
#pragma unroll
    for (int x = 0; x < N; x++) {
      const Zw v = live ? zw_of(S[j * N + x]) : Zw{0, 0, 0, 0}, u = live ? zw_of(S[j * N + (x ^ f)]) : Zw{0, 0, 0, 0};
      big = max(big, zmax_abs(v));
      w[x] = zmul(zconj(u), v);
    }
#pragma unroll
    for (int hb = 1; hb < N; hb <<= 1)
#pragma unroll
      for (int x = 0; x < N; x++)
        if (!(x & hb)) { const Zw a = w[x], b = w[x | hb]; w[x] = zadd(a, b); w[x | hb] = zsub(a, b); }
    // <v|v>, from the row's f = 0 lane
    const int src = (lane & ~(N - 1)) & 31;
    const Zw nrm{__shfl_sync(FULL, w[0].a, src), __shfl_sync(FULL, w[0].b, src), __shfl_sync(FULL, w[0].c, src),
                 __shfl_sync(FULL, w[0].d, src)};
    int cnt = 0;
#pragma unroll
    for (int z = 0; z < N; z++) {
      // i^{|f & z|} W(z) = +-nrm  <=>  W(z) = +-i^{-|f & z|} nrm; i = w^2 turns (a, b, c, d) into (-c, -d, a, b)
      Zw tg = nrm;
      if (__popc(f & z) & 1) tg = Zw{tg.c, tg.d, -tg.a, -tg.b};                 // times -i (up to the sign)
      cnt += zeq(w[z], tg) || zeq(w[z], Zw{-tg.a, -tg.b, -tg.c, -tg.d});
    }
#pragma unroll
    for (int o = 1; o < N; o <<= 1) {
      cnt += __shfl_xor_sync(FULL, cnt, o);
      big = max(big, (int64_t)__shfl_xor_sync(FULL, (long long)big, o));
    }
    if (live && f == 0 && big < (1LL << 27)) {
      const int r = 31 - __clz(cnt);                                                // cnt >= 1: the identity
      best = max(best, abs((NQ - r) - sp.ginfo[j * W + 1]));
    }
  }
  return warp_imax(best);
}

// class key: the smallest key over the symmetry orbit of S (qubit relabellings, with conjugation for some), so
// every member of a class gets the same key; classes are always compared exactly, so the key only has to be
// class-invariant, and a collision costs an exact comparison, never a wrong answer.
// Per orbit element two 32-bit position-weighted sums of per-entry 32-bit hashes, sum_e h(S[e]) W[pi(e)] mod 2^32
// (A and B: independent hashes and weights), form a 64-bit value, finalised with the exponent k. Each lane adds its
// entries' terms for every element (hash of the entry or of its conjugate, by the element's conjugation); a
// reduce-scatter over the 32 (element, A/B) sums then leaves lane s with A_s and lane 16 + s with B_s, and the
// minimum over the elements is taken across lanes. W[pos] packs (weight A, weight B); perm[s][x] is the image of
// basis index x under element s.
__device__ __forceinline__ uint32_t fmix32(uint32_t h) {
  h ^= h >> 16; h *= 0x85ebca6bu; h ^= h >> 13; h *= 0xc2b2ae35u; h ^= h >> 16;
  return h;
}
template <typename ST> __device__ __forceinline__ void entry_hash(const Z4<ST> &x, uint32_t &ha, uint32_t &hb) {
  // the limbs as 64-bit values (so int32 and int64 storage of one residual hash alike): low and high words
  const uint64_t a = (uint64_t)(int64_t)x.a, b = (uint64_t)(int64_t)x.b, c = (uint64_t)(int64_t)x.c,
                 d = (uint64_t)(int64_t)x.d;
  const uint32_t lo0 = (uint32_t)a * 0x9e3779b1u + (uint32_t)b * 0x85ebca77u + (uint32_t)c * 0xc2b2ae3du +
                       (uint32_t)d * 0x27d4eb2fu;
  const uint32_t lo1 = (uint32_t)a * 0x165667b1u + (uint32_t)b * 0xd3a2646cu + (uint32_t)c * 0xfd7046c5u +
                       (uint32_t)d * 0xb55a4f09u;
  const uint32_t hi = (uint32_t)(a >> 32) * 0x61c88647u + (uint32_t)(b >> 32) * 0x7a646e4du +
                      (uint32_t)(c >> 32) * 0x3c6ef372u + (uint32_t)(d >> 32) * 0x5bd1e995u;
  ha = fmix32(lo0 ^ hi);
  hb = fmix32(lo1 + (hi ^ 0x1b873593u));
}
// x: the lane's two entries, at positions ei (negative: none; every position in one lane); weight(s, e): W[pi_s(e)].
template <int NQ, typename ST, typename Weight>
__device__ __forceinline__ void warp_key_entries(const Z4<ST> (&x)[2], const int (&ei)[2], int k, int nsym, unsigned conjmask,
                                                 Weight weight, int lane, uint64_t &k1, uint64_t &k2) {
  static_assert(SYMMAX == 12, "the reduce-scatter halves 12 elements twice and keeps 3 per lane");
  uint32_t fa[2], fb[2], ca[2], cb[2];
#pragma unroll
  for (int j = 0; j < 2; j++) {
    entry_hash(x[j], fa[j], fb[j]);
    entry_hash(zcj(x[j]), ca[j], cb[j]);
    if (ei[j] < 0) fa[j] = fb[j] = ca[j] = cb[j] = 0;
  }
  uint32_t v[24];                            // A of element s at s, B at 12 + s
#pragma unroll
  for (int s = 0; s < 12; s++) {
    v[s] = v[12 + s] = 0;
    if (s >= nsym) continue;
    const bool cj = (conjmask >> s) & 1;
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const uint64_t w = weight(s, max(ei[j], 0));
      v[s] += (cj ? ca[j] : fa[j]) * (uint32_t)w;
      v[12 + s] += (cj ? cb[j] : fb[j]) * (uint32_t)(w >> 32);
    }
  }
  // reduce-scatter: at offset o a lane keeps the half of its values on its side of lane bit o and adds the partner's
  // copy of that half: A or B by bit 4, six elements by bit 3, three by bit 2, summed over bits 1 and 0
#pragma unroll
  for (int o = 16, n = 12; o >= 4; o >>= 1, n >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < n; i++) {
      const uint32_t keep = up ? v[n + i] : v[i], give = up ? v[i] : v[n + i];
      v[i] = keep + __shfl_xor_sync(FULL, give, o);
    }
  }
#pragma unroll
  for (int i = 0; i < 3; i++) {
    v[i] += __shfl_xor_sync(FULL, v[i], 2);
    v[i] += __shfl_xor_sync(FULL, v[i], 1);
  }
  const int r = lane & 3, el = 6 * ((lane >> 3) & 1) + 3 * ((lane >> 2) & 1) + r;   // the lane's element (r < 3)
  const uint32_t mine = r == 0 ? v[0] : (r == 1 ? v[1] : v[2]);
  const uint32_t other = __shfl_xor_sync(FULL, mine, 16);                           // lanes < 16: A here, B there
  uint64_t x1 = ~0ULL;
  if (lane < 16 && r < 3 && el < nsym) x1 = fmix64((((uint64_t)mine << 32) | other) + (uint64_t)k * 0xa0761d6478bd642fULL);
  const uint32_t hi = __reduce_min_sync(FULL, (uint32_t)(x1 >> 32));
  const uint32_t lo = __reduce_min_sync(FULL, (uint32_t)(x1 >> 32) == hi ? (uint32_t)x1 : ~0u);
  k1 = ((uint64_t)hi << 32) | lo;
  k2 = fmix64(k1 ^ 0xe7037ed1a0b428dbULL);
}
// of the residual S in shared memory, the weights by position W through the group's basis maps
template <int NQ, typename ST>
__device__ __forceinline__ void warp_class_key(const Z4<ST> *S, int k, int nsym, unsigned conjmask, const uint8_t (*perm)[8],
                                               const uint64_t *W, int lane, uint64_t &k1, uint64_t &k2) {
  constexpr int N = 1 << NQ, E = N * N;
  Z4<ST> x[2];
  int ei[2];
#pragma unroll
  for (int j = 0; j < 2; j++) {
    ei[j] = lane + 32 * j < E ? lane + 32 * j : -1;
    x[j] = ei[j] >= 0 ? S[ei[j]] : Z4<ST>{0, 0, 0, 0};
  }
  warp_key_entries<NQ, ST>(x, ei, k, nsym, conjmask,
                           [&](int s, int e) { return W[perm[s][e >> NQ] * N + perm[s][e & (N - 1)]]; }, lane, k1, k2);
}

template <int NQ, typename ST> struct ExpandSmem {
  static constexpr int E = (1 << NQ) * (1 << NQ), NB = sizeof(ST) == 4 ? 2 : 1;
  Z4<ST> P[EXP_WARPS][NB][E];      // a warp's parent, and its next one arriving
  Z4<ST> C[EXP_WARPS][E];
  uint64_t Wt[SYMMAX][E];          // the class key's weights per group element, W[pi_s(e)]
  uint32_t F[EXP_WARPS][E];        // the parent's entries in F_p
};

// the class key's position weights: (weight A, weight B), both odd
__device__ __forceinline__ uint64_t key_weight(int pos) {
  return fmix64(0x243f6a8885a308d3ULL + (uint64_t)pos * 0x13198a2e03707345ULL) | 0x0000000100000001ULL;
}
__device__ __forceinline__ void init_weights(uint64_t *W, int E) {
  for (int i = threadIdx.x; i < E; i += blockDim.x) W[i] = key_weight(i);
}
// the same for every element of the symmetry group, through its basis maps
template <int NQ> __device__ __forceinline__ void init_group_weights(uint64_t (*Wt)[(1 << NQ) * (1 << NQ)], const DevSpec &sp) {
  constexpr int N = 1 << NQ, E = N * N;
  for (int i = threadIdx.x; i < sp.nsym * E; i += blockDim.x) {
    const int s = i / E, e = i % E;
    Wt[s][e] = key_weight(sp.symperm[s][e >> NQ] * N + sp.symperm[s][e & (N - 1)]);
  }
}

// ---------------- the level kernel ----------------
// per-warp tallies of one job's children, flushed to that job's DevStats
struct WarpTally {
  unsigned long long w2 = 0, w3 = 0, dead = 0, alive = 0, found = 0, teval = 0, child = 0, full = 0;
  unsigned long long first = ~0ULL;
  bool ovf = false;
  __device__ __forceinline__ void flush(DevStats *st, int lane) {
    if (lane == 0) {
      if (w2) atomicAdd(&st->w2, w2);
      if (w3) atomicAdd(&st->w3, w3);
      if (dead) atomicAdd(&st->dead, dead);
      if (alive) atomicAdd(&st->alive, alive);
      if (found) { atomicAdd(&st->found, found); atomicMin(&st->first_found, first); }
      if (teval) atomicAdd(&st->t_evals, teval);
      if (child) atomicAdd(&st->children, child);
      if (full) atomicAdd(&st->full, full);
      if (ovf) st->ovf = 1;
    }
    *this = WarpTally{};
  }
};
// a survivor is a 32-byte record (class key, child index, bounds); its residual is recomputed from the parent
// where it is needed (exact class comparison, the next frontier)
template <typename ST> struct ExpandOut {
  DevStats *st;                    // survivor slot counter and overflow flag
  unsigned long long cap;
  uint64_t *sh1, *sh2, *sidx;
  NodeMeta *smeta;
  TQEntry *tq;                     // deferred T evaluations (nullptr: evaluate in place)
  unsigned long long tqcap;
};

// every child of parent p (residual already in P): window rules, exact prechecks, child residual, bounds, class key,
// survivor append. sp is the parent's spec (kernel parameter or a shared copy), sps its shared-memory address for
// the out-of-line helpers; child index = p * GS + g; F: the warp's room for the parent's F_p image; weight: the class
// key's weights.
// PART: 0 every candidate; 1 the one-qubit gates; 2 the multi-qubit gates. The plain level runs the two parts as
// two launches: each warp then walks the code of one kind of child (instruction fetch is the level kernel's main
// stall; measured 3 % faster than one launch), at the price of reading each parent twice. (Three parts, the odd
// diagonals on their own, measured slower than one.)
//
// Most children never have their residual computed. When the cut around a gate's qubit has F_p Schmidt rank >= 2 the
// parent is no product there, so no gate on that qubit alone makes it act trivially: the support of a one-qubit child is
// the parent's. A unit monomial (x z s sdg t tdg) keeps the exponent, one-qubit gates the CX bound, affine monomials
// the H structure and Cliffords the T bound, so such a child's bounds are the parent's own: the Clifford ones are decided
// one per lane, the odd diagonals queued one per lane. A two-qubit permutation (cx) changes only the ranks of the cuts it
// crosses; they are eliminated straight from the parent's F_p image (computed once per parent) with its columns permuted.
// Only survivors' entries are then formed, in registers, for the class key. Deep
// proofs (budget 12, two targets, 2.74 M parents): both parts 19.9 -> 12.6 ms, 10.5 ms with the ranks of warp_cx_pair; bound by
// issue (80 %) and, for the one-qubit part, by instruction fetch.
template <int NQ, typename ST, bool STATES = false, int PART = 0, typename Weight>
__device__ __forceinline__ void expand_parent(const DevSpec &sp, const DevSpec *sps, Weight weight, unsigned conjmask,
                                              const Z4<ST> *P, Z4<ST> *C, uint32_t *F, unsigned long long p,
                                              const NodeMeta pm, int rem, bool keep, int GS, const ExpandOut<ST> &o,
                                              WarpTally &c, int lane, int split = 1, int sub = 0) {
  constexpr int N = 1 << NQ, E = N * N, EPL = E >= 32 ? E / 32 : 1;
  const int G = sp.G;
  const int g1 = pm.g1 == 0xff ? -1 : pm.g1, g2 = pm.g2 == 0xff ? -1 : pm.g2;
  const int kP = pm.k, TP = pm.T, c2P = pm.c2, hsP = (pm.hsn & 1) ? 2 : 0, ntP = (pm.hsn >> 1) & 7;
  const int suppP = __popc(ntP);
  const bool pre_ok = !STATES && sp.standard && !sp.states && kP < INHERIT_KMAX;
  // the cut around qubit q has rank >= 2 (needs as packed in NodeMeta)
  auto entangled = [&](int q, int needs) { const int b = sps->qcut[q]; return b != QC_NONE && ((needs >> b) & 3) != 0; };
  unsigned long long pend[3] = {0, 0, 0};    // per qubit: 1 + queue entry of its deferred odd-diagonal child
  auto put_entry = [&](unsigned long long e, int ga, int gb, int n, int k, int c2, int needs, int hs, int ntriv) {
    TQEntry q;
    q.p = p; q.k = (int16_t)k; q.n = (uint8_t)n; q.g[0] = (uint8_t)ga; q.g[1] = (uint8_t)gb; q.c2 = (uint8_t)c2;
    q.needs = (uint8_t)needs; q.hs = (uint8_t)hs; q.ntriv[0] = (uint8_t)ntriv; q.ntriv[1] = n > 1 ? (uint8_t)ntriv : 0;
    q.pad[0] = q.pad[1] = q.pad[2] = q.pad[3] = 0;
    o.tq[e] = q;
  };
  // queue a deferred T evaluation: a second odd diagonal on the same qubit joins its sibling's entry
  auto defer = [&](int g, int k, int c2, int needs, int hs, int ntriv, int q0, bool tdiag) {
    if (tdiag && pend[q0]) {
      const unsigned long long e = pend[q0] - 1;
      if (lane == 0) { o.tq[e].g[1] = (uint8_t)g; o.tq[e].ntriv[1] = (uint8_t)ntriv; o.tq[e].n = 2; }
      pend[q0] = 0;                          // an entry holds two children
      return;
    }
    unsigned long long e = 0;
    if (lane == 0) e = atomicAdd(&o.st->n_tq, 1ULL);
    e = __shfl_sync(FULL, e, 0);
    if (e >= o.tqcap) return;                // counted: the host redoes the level with room for every entry
    if (lane == 0) put_entry(e, g, 0xff, 1, k, c2, needs, hs, ntriv);
    if (tdiag) pend[q0] = e + 1;
  };
  // the fates decided without the child's residual, one candidate per lane: window cuts (W2, W3) and the exact
  // prechecks. Lower bounds on the child's bounds from the parent's: k drops by at most the gate's sqrt2 exponent;
  // H structure, T and CX bounds are unchanged by monomial-affine / Clifford / one-qubit gates; an odd diagonal
  // changes T by at most 1; a gate of Schmidt rank 2 changes the CX bound by at most 1; support changes only on
  // the gate's qubits (not at all under a one-qubit gate on an entangled one). combine is monotone in every argument,
  // so exceeding the budget with these proves the child dead (the goal has all bounds 0 and is never removed here).
  // The other children are decided as their kind allows, or evaluated in order.
  enum { NONE, W2, W3, DEADP, QUEUE, FULLC, ALIVEP, RANKS, HADA };
  const bool need_b = sp.standard != 0 && !sp.states;
  for (int g0 = 0; g0 < G; g0 += 32) {
    const int g = g0 + lane;
    int fate = NONE, q0 = 0;
    // with several warps to a parent, this one's share: the odd diagonals by qubit (siblings share a queue entry), the
    // other candidates by index
    const bool share = split == 1 || (g < G && ((sps->gflags[g] & GF_TDIAG) ? sps->gq[g][0] : g) % split == sub);
    if (g < G && share && (PART == 0 || ((sp.gflags[g] & GF_ONEQ) != 0) == (PART == 1))) {
      fate = FULLC;
      if (g1 >= 0 && __ldg(&sp.bad2[g1 * G + g])) fate = W2;
      else if (g2 >= 0) {
        const uint32_t tri = ((uint32_t)g2 * G + (uint32_t)g1) * G + (uint32_t)g;
        if ((__ldg(&sp.bad3[tri >> 5]) >> (tri & 31)) & 1) fate = W3;
      }
      if (fate == FULLC && pre_ok) {
        const uint8_t fl = sps->gflags[g];
        q0 = sps->gq[g][0];
        const int ik = sps->gik[g] > 0 ? sps->gik[g] : 0;
        const bool oneq = fl & GF_ONEQ, ent = oneq && entangled(q0, pm.needs);
        int hlo = kP - ik;
        if ((fl & GF_MONAFF) && hsP > hlo) hlo = hsP;
        const int tlo = (fl & GF_CLIFFORD) ? TP : ((fl & GF_TDIAG) ? (NQ == 3 ? cols_t_least(pm.cols, TP, q0) : TP - 1) : 0);
        const int clo = oneq ? c2P : ((fl & GF_RANK2) ? c2P - 1 : 0);
        const int slo = ent ? suppP : suppP - sps->gnq[g];
        if (combine(max(hlo, 0), max(tlo, 0), max(clo, 0), max(slo, 0)) > rem) fate = DEADP;
        else if (!sp.lite && (fl & (GF_UNITMON | GF_MONAFF)) == (GF_UNITMON | GF_MONAFF)) {
          if (PART != 2 && ent) {
            if (fl & GF_CLIFFORD) fate = ALIVEP;             // every bound above was exact
            else if (fl & GF_TDIAG) fate = QUEUE;
          } else if (PART != 1 && !oneq && (fl & GF_CLIFFORD) && sps->gkind[g] == GK_PERM && sps->gnq[g] == 2 &&
                     (ntP & ~sps->gmask[g])) {               // (else the child may be the goal)
            fate = RANKS;
          }
        } else if (PART != 2 && !sp.lite && sp.unit && ent && (fl & GF_CLIFFORD) && sps->gkind[g] == GK_ONEQ &&
                   sizeof(ST) == 4 && kP <= 56) {
          fate = HADA;
        }
      }
    }
    c.w2 += __popc(__ballot_sync(FULL, fate == W2));
    c.w3 += __popc(__ballot_sync(FULL, fate == W3));
    c.child += __popc(__ballot_sync(FULL, fate >= DEADP));
    c.dead += __popc(__ballot_sync(FULL, fate == DEADP));
    unsigned todo = __ballot_sync(FULL, fate >= FULLC);
    if constexpr (!STATES && PART != 2) {
      const unsigned m = __ballot_sync(FULL, fate == ALIVEP);
      if (!keep) { c.alive += __popc(m); todo &= ~m; }        // counted only
      if (__ballot_sync(FULL, fate == QUEUE)) {
        // the odd diagonals of one qubit two by two (their T bounds agree: they differ by a power of S)
        const unsigned peers = __match_any_sync(FULL, fate == QUEUE ? q0 : 8), below = (1u << lane) - 1;
        const bool lead = fate == QUEUE && !(__popc(peers & below) & 1);
        const unsigned leads = __ballot_sync(FULL, lead);
        unsigned long long e = 0;
        if (lane == 0) e = atomicAdd(&o.st->n_tq, (unsigned long long)__popc(leads));
        e = __shfl_sync(FULL, e, 0) + __popc(leads & below);
        if (lead && e < o.tqcap) {           // (entries past the room are counted: the host redoes the level)
          const unsigned after = peers & ~below & ~(1u << lane);
          put_entry(e, g, after ? g0 + __ffs(after) - 1 : 0xff, after ? 2 : 1, kP, c2P, pm.needs, hsP, ntP);
        }
      }
    }
    if constexpr (!STATES && PART != 1) {
      if (__ballot_sync(FULL, fate == RANKS)) {
        __syncwarp();
#pragma unroll
        for (int j = 0; j < EPL; j++)
          if (lane + 32 * j < E) F[lane + 32 * j] = to_fp(P[lane + 32 * j], *sps);
        __syncwarp();
      }
    }
    for (; todo; todo &= todo - 1) {
      const int g = g0 + __ffs(todo) - 1;
      int kind = STATES ? (int)FULLC : __shfl_sync(FULL, fate, g - g0);
      const uint8_t fl = sp.gflags[g];
      const int gm = sp.gmask[g], gq0 = sp.gq[g][0];
      // the child's bounds (the parent's until shown otherwise) and the lane's entries of its residual
      int k = kP, T = TP, c2 = c2P, hs = hsP, needs = pm.needs, ntriv = ntP, ei[2] = {-1, -1};
      Z4<ST> x[2] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
      bool alive = true;
      if (!STATES && PART != 1 && kind == RANKS) {
        const uint8_t *mono = sps->gmono[g];
        if (NQ == 3 && sps->cuts3) c2 = warp_cx_pair(F, mono, *sps, lane, gq0, sps->gq[g][1], pm.needs, needs);
        else c2 = warp_cx_elems<NQ>([&](int r, int i) { return F[(r << NQ) + (mono[i] & 15)]; }, *sps, lane, gm, pm.needs, needs);
        ntriv = ntP | gm;
        if (!entangled(gq0, needs) || !entangled(sps->gq[g][1], needs)) kind = FULLC;   // one may have become trivial
        else alive = combine(max(kP, hsP), TP, c2, __popc(ntriv)) <= rem;
      }
      if (!STATES && PART != 2 && kind == HADA) {
        // a Hadamard-like Clifford on an entangled qubit: only the exponent is open (and, for a small one, the H
        // structure: a unitary residual of exponent 1 or more in normal form is not monomial)
        if constexpr (sizeof(ST) == 4) {
          const int lo = (1 << gq0) - 1;
          I4 v[2] = {I4{0, 0, 0, 0}, I4{0, 0, 0, 0}};
          if (lane < E / 2) {
            ei[0] = ((lane & ~lo) << 1) | (lane & lo);
            ei[1] = ei[0] | (1 << gq0);
            oneq_pair(P, ei, sps->gph[g], v);
          }
          k = normalise_pair(v, kP + sps->gik[g]);
          c.full++;
          if (k < 1) {
            ei[0] = ei[1] = -1;
            kind = FULLC;
            c.full--;
          } else {
            hs = 0;
            alive = combine(k, TP, c2P, suppP) <= rem;
#pragma unroll
            for (int j = 0; j < 2; j++) x[j] = Z4<ST>{(ST)v[j].a, (ST)v[j].b, (ST)v[j].c, (ST)v[j].d};
          }
        }
      } else if (kind != FULLC) {
        if (alive && keep) {
          const int mono = sps->gmono[g][lane & (N - 1)];
#pragma unroll
          for (int j = 0; j < EPL; j++)
            if (lane + 32 * j < E) {
              ei[j] = lane + 32 * j;
              x[j] = mono_entry<NQ>(P, mono, lane, j);
            }
        }
      }
      if (kind == FULLC) {
        bool ovf;
        c.full++;
        k = warp_child<NQ, ST, PART>(P, C, g, kP, sp, sps, lane, ovf);
        if (ovf) { c.ovf = true; continue; }
        const bool need_hs = need_b && !(fl & GF_MONAFF);
        // the child is the goal only if the parent equals the gate, i.e. acts on no other qubit (unitary targets); the
        // qubit of a one-qubit gate stays non-trivial when it is entangled
        const int test_q = !need_b || (pre_ok && (fl & GF_ONEQ) && entangled(gq0, pm.needs)) ? 0 : gm;
        const Cheap ch = warp_cheap<NQ, ST>(C, k, sp, lane, (ntP & ~gm) == 0 || !need_b, need_hs, test_q, ntP);
        if (ch.goal) {
          if (sp.nogoal) c.dead++;
          else {
            c.found++;
            const unsigned long long oi = p * (unsigned long long)GS + g;
            if (oi < c.first) c.first = oi;
          }
          continue;
        }
        const bool inheritT = (fl & GF_CLIFFORD) && k <= INHERIT_KMAX && kP <= INHERIT_KMAX;
        const bool cacheT = (fl & GF_TDIAG) && k <= INHERIT_KMAX;
        T = 0; c2 = 0; hs = 0; needs = 0;
        ntriv = need_b ? ch.ntriv : 0;
        if constexpr (STATES) {                    // state targets (cheese.cu:683-716): no inherited bounds
          if (sp.standard || sp.lite) {
            int h = k;
            if (!sp.lite) warp_state_cheap<NQ, ST>(C, k, *sps, lane, h, c2);
            if (combine(h, 0, c2, 0) > rem) alive = false;
            else {
              T = warp_state_t<NQ, ST>(C, *sps, lane); c.teval++;
              alive = combine(h, T, c2, 0) <= rem;
            }
          }
        } else if (sp.lite) {
          if (k > rem) alive = false;
          else {
            if (inheritT) T = TP;
            else { defer(g, k, 0, 0, 0, 0, gq0, cacheT && (fl & GF_ONEQ) && k == kP); continue; }
            alive = k + (T + sp.tdiv - 1) / sp.tdiv <= rem;
          }
        } else if (need_b) {
          hs = need_hs ? ch.hs : hsP;
          const int h = k > hs ? k : hs;
          const int supp = __popc(ch.ntriv);
          if (PART == 1 || (PART == 0 && (fl & GF_ONEQ))) { c2 = c2P; needs = pm.needs; }
          else c2 = warp_cx_bound<NQ, ST>(C, *sps, lane, gm, pm.needs, needs);
          if (combine(h, 0, c2, supp) > rem) alive = false;
          else {
            if (inheritT) T = TP;
            else {
              // siblings share an entry only when every bound but support is the parent's (one-qubit monomial gates)
              const bool share = cacheT && (fl & GF_ONEQ) && (fl & GF_MONAFF) && k == kP;
              defer(g, k, c2, needs, hs, ch.ntriv, gq0, share);
              continue;
            }
            alive = combine(h, T, c2, supp) <= rem;
          }
        }
        if (alive && keep) {
#pragma unroll
          for (int j = 0; j < EPL; j++)
            if (lane + 32 * j < E) {
              ei[j] = lane + 32 * j;
              x[j] = C[lane + 32 * j];
            }
        }
      }
      if (!alive) { c.dead++; continue; }
      c.alive++;
      if (!keep) continue;
      uint64_t k1, k2;
      warp_key_entries<NQ, ST>(x, ei, k, sp.nsym, conjmask, weight, lane, k1, k2);
      unsigned long long slot = 0;
      if (lane == 0) slot = atomicAdd(&o.st->n_surv, 1ULL);
      slot = __shfl_sync(FULL, slot, 0);
      if (slot < o.cap) {
        if (lane == 0) {
          o.sh1[slot] = k1; o.sh2[slot] = k2; o.sidx[slot] = p * (unsigned long long)GS + g;
          NodeMeta nm;
          nm.k = (int16_t)k; nm.T = (uint8_t)(T > 255 ? 255 : T); nm.c2 = (uint8_t)c2; nm.g1 = (uint8_t)g; nm.g2 = pm.g1;
          nm.hsn = (uint8_t)((hs == 2 ? 1 : 0) | (ntriv << 1));
          nm.needs = (uint8_t)needs;
          nm.cols = NQ == 3 && (fl & GF_CLIFFORD) ? cols_after(pm.cols, sps->gcol[g]) : 0;   // (only Cliffords get here)
          o.smeta[slot] = nm;
        }
      } else if (lane == 0) {
        o.st->surv_overflow = 1;
      }
      __syncwarp();
    }
  }
}

// goal pass, step 1: parents whose stored bounds allow a goal child (combine of H, T, CX and support <= 1)
__global__ void k_goal_candidates(const NodeMeta *meta, long long m, uint32_t *list, GoalShort *gs) {
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < m; p += (long long)gridDim.x * blockDim.x) {
    const NodeMeta pm = meta[p];
    const int hs = (pm.hsn & 1) ? 2 : 0, h = pm.k > hs ? pm.k : hs;
    if (combine(h, pm.T, pm.c2, __popc((pm.hsn >> 1) & 7)) > 1) continue;
    const unsigned long long i = atomicAdd(&gs->count, 1ULL);
    if (i < GOAL_LIST) list[i] = (uint32_t)p;
  }
}
// goal pass, step 2 (one warp per candidate parent): its children past the window rules, tested for the goal
template <int NQ, typename ST>
__global__ void __launch_bounds__(EXP_WARPS * 32) k_goal_level(const DevSpec sp, const Z4<ST> *R, const NodeMeta *meta,
                                                              const uint32_t *list, int GS, GoalShort *gs) {
  constexpr int E = (1 << NQ) * (1 << NQ), EPL = E >= 32 ? E / 32 : 1;
  __shared__ Z4<ST> sP[EXP_WARPS][E], sC[EXP_WARPS][E];
  __shared__ DevSpec s_sp;
  for (int i = threadIdx.x; i < (int)(sizeof(DevSpec) / 4); i += blockDim.x) ((int *)&s_sp)[i] = ((const int *)&sp)[i];
  __syncthreads();
  const unsigned long long n = gs->count;
  if (n > GOAL_LIST) return;                   // the list is not complete: no shortcut for this level
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int G = s_sp.G;
  unsigned long long found = 0, first = ~0ULL;
  bool ovf = false;
  for (unsigned long long i = blockIdx.x * (unsigned long long)EXP_WARPS + w; i < n;
       i += (unsigned long long)gridDim.x * EXP_WARPS) {
    const uint32_t p = list[i];
    const NodeMeta pm = meta[p];
    const int g1 = pm.g1 == 0xff ? -1 : pm.g1, g2 = pm.g2 == 0xff ? -1 : pm.g2;
    __syncwarp();
#pragma unroll
    for (int q = 0; q < EPL; q++) {
      const int e = lane + 32 * q;
      if (e < E) sP[w][e] = R[(size_t)p * E + e];
    }
    __syncwarp();
    for (int g = 0; g < G; g++) {
      if (g1 >= 0 && __ldg(&s_sp.bad2[g1 * G + g])) continue;
      if (g2 >= 0) {
        const uint32_t tri = ((uint32_t)g2 * G + (uint32_t)g1) * G + (uint32_t)g;
        if ((__ldg(&s_sp.bad3[tri >> 5]) >> (tri & 31)) & 1) continue;
      }
      bool o;
      const int k = warp_child<NQ, ST>(sP[w], sC[w], g, pm.k, s_sp, &s_sp, lane, o);
      if (o) { ovf = true; continue; }
      const Cheap ch = warp_cheap<NQ, ST>(sC[w], k, s_sp, lane, true, false, 0, 0);
      if (ch.goal) {
        found++;
        const unsigned long long oi = (unsigned long long)p * GS + g;
        if (oi < first) first = oi;
      }
    }
  }
  if (lane == 0) {
    if (found) { atomicAdd(&gs->found, found); atomicMin(&gs->first, first); }
    if (ovf) atomicExch(&gs->ovf, 1u);
  }
}

// A warp's parents: taken from a counter two ahead, the residual one ahead (copied into shared memory by cp.async while
// the current parent is expanded), so neither the counter nor the loads are waited for. body(p, P, meta, sub). A level
// with fewer parents than warps on the chip splits each parent's candidates over `split` warps (sub = 0 .. split - 1).
// AHEAD false: a warp takes a parent only when it is done with the one before. So for state targets: their children cost so
// much (0.1 ms of a warp each) that a parent held by a busy warp delays the level's end, and the loads hidden are nothing beside
// it (a 3-qubit search of 5.9 M prefixes: 71.1 ms of level kernels taking ahead, 66.5 ms so).
template <int NQ, typename ST, bool AHEAD = true, typename Body>
__device__ __forceinline__ void walk_parents(ExpandSmem<NQ, ST> &sm, unsigned long long *counter, unsigned long long p0,
                                             unsigned long long end, const Z4<ST> *R, const NodeMeta *meta, int w, int lane,
                                             int split, Body body) {
  constexpr int E = (1 << NQ) * (1 << NQ), NB = ExpandSmem<NQ, ST>::NB, CHUNKS = E * (int)sizeof(Z4<ST>) / 16;
  auto grab = [&]() { return lane == 0 ? p0 + atomicAdd(counter, 1ULL) : 0ULL; };
  auto parent = [&](unsigned long long it) { return split == 1 ? it : (unsigned long long)((unsigned)it / (unsigned)split); };
  auto fetch = [&](unsigned long long it, int b, NodeMeta &m) {
    if (it < end) {
      const unsigned long long p = parent(it);
      const char *src = (const char *)(R + p * (unsigned long long)E);
      char *dst = (char *)sm.P[w][b];
      for (int i = lane; i < CHUNKS; i += 32) cp_async16(dst + 16 * i, src + 16 * i);
      m = meta[p];
    }
    cp_async_commit();
  };
  NodeMeta m{}, mn{};
  if constexpr (!AHEAD) {
    for (;;) {
      const unsigned long long p = __shfl_sync(FULL, grab(), 0);
      if (p >= end) return;
      fetch(p, 0, m);
      cp_async_wait<0>();
      __syncwarp();
      body(parent(p), sm.P[w][0], m, split == 1 ? 0 : (int)((unsigned)p % (unsigned)split));
      __syncwarp();
    }
  }
  unsigned long long p = __shfl_sync(FULL, grab(), 0), raw = grab();
  int b = 0;
  fetch(p, 0, m);
  while (p < end) {
    const unsigned long long pn = __shfl_sync(FULL, raw, 0);
    if (NB == 2) fetch(pn, b ^ 1, mn);
    raw = grab();
    if (NB == 2) cp_async_wait<1>();
    else cp_async_wait<0>();
    __syncwarp();
    body(parent(p), sm.P[w][b], m, split == 1 ? 0 : (int)((unsigned)p % (unsigned)split));
    __syncwarp();
    if (NB == 1) fetch(pn, 0, mn);
    p = pn;
    m = mn;
    b ^= NB - 1;
  }
  cp_async_wait<0>();
}

template <int NQ, typename ST, bool STATES = false, int PART = 0>
__global__ void __launch_bounds__(EXP_WARPS * 32, EXP_MINB) k_expand(const DevSpec sp, const ExpandArgs<ST> a) {
  constexpr int E = (1 << NQ) * (1 << NQ);
  if (a.gshort && a.gshort->found && !a.gshort->ovf && a.gshort->count <= GOAL_LIST) return;   // the found level
  __shared__ ExpandSmem<NQ, ST> sm;
  __shared__ DevSpec s_sp;                     // the spec for out-of-line helpers (a shared address, no local copy)
  for (int i = threadIdx.x; i < (int)(sizeof(DevSpec) / 4); i += blockDim.x) ((int *)&s_sp)[i] = ((const int *)&sp)[i];
  __syncthreads();
  init_group_weights<NQ>(sm.Wt, s_sp);
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned conjmask = 0;
  for (int i = 0; i < sp.nsym; i++) conjmask |= (unsigned)(sp.symconj[i] != 0) << i;
  const ExpandOut<ST> o{a.st, a.cap, a.sh1, a.sh2, a.sidx, a.smeta, a.tq, a.tqcap};
  const auto weight = [&](int s, int e) { return sm.Wt[s][e & (E - 1)]; };
  WarpTally c;
  walk_parents<NQ, ST, !STATES>(sm, PART == 2 ? &a.st->work2 : &a.st->work, 0, (unsigned long long)a.m * a.split, a.R, a.meta, w,
                       lane, a.split, [&](unsigned long long p, const Z4<ST> *P, const NodeMeta &pm, int sub) {
    expand_parent<NQ, ST, STATES, PART>(sp, &s_sp, weight, conjmask, P, sm.C[w], sm.F[w], p, pm, a.rem, a.keep != 0, sp.G,
                                        o, c, lane, a.split, sub);
  });
  c.flush(a.st, lane);
}

// ---------------- the batched level kernel ----------------
// Many searches of one qubit count in one launch: the frontier is the concatenation of every job's nodes (each
// job's nodes contiguous, in its own order), fjob gives each node's job, specs[job] its device spec, jt[job] its
// current level. Child indices are p * 64 + g over the batch frontier, so each job's children keep its own order.
constexpr int BATCH_GS = 64;
constexpr int MAXDEPTH_WALK = 48;   // deepest circuit of a batched job
template <typename ST> struct BatchArgs {
  long long m, p0;                 // the chunk of the frontier this launch expands: nodes [p0, m)
  const Z4<ST> *R;
  const NodeMeta *meta;
  const uint32_t *fjob;             // job of every frontier node
  const DevSpec *specs;
  const int *jt;
  DevStats *jst;                   // per job
  DevStats *st;                    // batch-wide: work counter, survivor slots
  unsigned long long cap;
  uint64_t *sh1, *sh2, *sidx;
  NodeMeta *smeta;
  TQEntry *tq;
  unsigned long long tqcap;
  const GoalShort *gshort = nullptr;  // the chunk's goal pass (nullptr: none) and its per-job results
  const ulonglong2 *jgoal = nullptr;  // per job: goal children found by the pass, first of them
};

// a level's statistics block cleared (first found: none), the goal pass's header, and a batch chunk's per-job goal
// results (none found) — each when given
__global__ void k_level_init(GoalShort *gs, DevStats *st, ulonglong2 *jg = nullptr, int jn = 0) {
  const int i = threadIdx.x;
  constexpr int W = (int)(sizeof(DevStats) / 8);
  static_assert(sizeof(DevStats) % 8 == 0, "statistics block of 8-byte words");
  if (st)
    for (int j = i; j < W; j += blockDim.x) ((unsigned long long *)st)[j] = 0;
  for (int j = i; j < jn; j += blockDim.x) jg[j] = make_ulonglong2(0ULL, ~0ULL);
  __syncthreads();
  if (i == 0) {
    if (st) st->first_found = ~0ULL;
    if (gs) { gs->count = 0; gs->found = 0; gs->first = ~0ULL; gs->ovf = 0; gs->pad = 0; }
  }
}

// the batch's goal pass: candidate parents (stored lower bound <= 1) of jobs whose spec has the bounds, in nodes
// [p0, p1); then their children tested for the goal, per job
__global__ void k_goal_candidates_batch(const NodeMeta *meta, const uint32_t *fjob, const DevSpec *specs, long long p0,
                                        long long p1, uint32_t *list, GoalShort *gs) {
  for (long long p = p0 + blockIdx.x * (long long)blockDim.x + threadIdx.x; p < p1;
       p += (long long)gridDim.x * blockDim.x) {
    const DevSpec &sp = specs[fjob[p]];
    if (!sp.standard || sp.states || sp.nogoal) continue;
    const NodeMeta pm = meta[p];
    const int hs = (pm.hsn & 1) ? 2 : 0, h = pm.k > hs ? pm.k : hs;
    if (combine(h, pm.T, pm.c2, __popc((pm.hsn >> 1) & 7)) > 1) continue;
    const unsigned long long i = atomicAdd(&gs->count, 1ULL);
    if (i < GOAL_LIST) list[i] = (uint32_t)p;
  }
}
template <int NQ, typename ST>
__global__ void __launch_bounds__(EXP_WARPS * 32) k_goal_level_batch(const DevSpec *specs, const uint32_t *fjob,
                                                                    const Z4<ST> *R, const NodeMeta *meta,
                                                                    const uint32_t *list, GoalShort *gs,
                                                                    ulonglong2 *jgoal) {
  constexpr int E = (1 << NQ) * (1 << NQ), EPL = E >= 32 ? E / 32 : 1;
  __shared__ Z4<ST> sP[EXP_WARPS][E], sC[EXP_WARPS][E];
  __shared__ DevSpec sps[EXP_WARPS];
  const unsigned long long n = gs->count;
  if (n > GOAL_LIST) return;                   // incomplete list: no shortcut in this chunk
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  DevSpec &sp = sps[w];
  int cur = -1;                                // the job whose spec the warp holds
  for (unsigned long long i = blockIdx.x * (unsigned long long)EXP_WARPS + w; i < n;
       i += (unsigned long long)gridDim.x * EXP_WARPS) {
    const uint32_t p = list[i];
    const int job = (int)fjob[p];
    __syncwarp();
    if (job != cur) {
      for (int x = lane; x < (int)(sizeof(DevSpec) / 4); x += 32) ((int *)&sp)[x] = ((const int *)(specs + job))[x];
      cur = job;
    }
    const NodeMeta pm = meta[p];
    const int g1 = pm.g1 == 0xff ? -1 : pm.g1, g2 = pm.g2 == 0xff ? -1 : pm.g2;
#pragma unroll
    for (int q = 0; q < EPL; q++) {
      const int e = lane + 32 * q;
      if (e < E) sP[w][e] = R[(size_t)p * E + e];
    }
    __syncwarp();
    const int G = sp.G;
    unsigned long long found = 0, first = ~0ULL;
    bool ovf = false;
    for (int g = 0; g < G; g++) {
      if (g1 >= 0 && __ldg(&sp.bad2[g1 * G + g])) continue;
      if (g2 >= 0) {
        const uint32_t tri = ((uint32_t)g2 * G + (uint32_t)g1) * G + (uint32_t)g;
        if ((__ldg(&sp.bad3[tri >> 5]) >> (tri & 31)) & 1) continue;
      }
      bool o;
      const int k = warp_child<NQ, ST>(sP[w], sC[w], g, pm.k, sp, &sp, lane, o);
      if (o) { ovf = true; continue; }
      const Cheap ch = warp_cheap<NQ, ST>(sC[w], k, sp, lane, true, false, 0, 0);
      if (ch.goal) {
        found++;
        const unsigned long long oi = (unsigned long long)p * BATCH_GS + g;
        if (oi < first) first = oi;
      }
    }
    if (lane == 0) {
      if (found) { atomicAdd(&jgoal[job].x, found); atomicMin(&jgoal[job].y, first); }
      if (ovf) atomicExch(&gs->ovf, 1u);
    }
  }
}

template <int NQ, typename ST>
__global__ void __launch_bounds__(EXP_WARPS * 32, EXPB_MINB) k_expand_batch(const BatchArgs<ST> a) {
  constexpr int N = 1 << NQ, E = N * N, EPL = E >= 32 ? E / 32 : 1;
  __shared__ Z4<ST> sP[EXP_WARPS][E], sC[EXP_WARPS][E];
  __shared__ uint64_t W[E];
  __shared__ uint32_t sF[EXP_WARPS][E];
  __shared__ DevSpec sps[EXP_WARPS];           // each warp's current job spec
  init_weights(W, E);
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  Z4<ST> *P = sP[w], *C = sC[w];
  DevSpec &sp = sps[w];
  const ExpandOut<ST> o{a.st, a.cap, a.sh1, a.sh2, a.sidx, a.smeta, a.tq, a.tqcap};
  WarpTally c;
  int job = -1, rem = 0;
  bool keep = false, skip = false;
  unsigned conjmask = 0;
  const bool pass_ok = a.gshort && !a.gshort->ovf && a.gshort->count <= GOAL_LIST;
  for (;;) {
    unsigned long long p = 0;
    if (lane == 0) p = a.p0 + atomicAdd(&a.st->work, 1ULL);
    p = __shfl_sync(FULL, p, 0);
    if ((long long)p >= a.m) break;
    const int pj = (int)a.fjob[p];
    if (pj != job) {                             // another job: flush the tallies, load its spec
      if (job >= 0) c.flush(a.jst + job, lane);
      job = pj;
      skip = pass_ok && a.jgoal[job].x > 0;      // the goal pass found this job's goal: its found level
      if (skip) continue;
      __syncwarp();
      for (int i = lane; i < (int)(sizeof(DevSpec) / 4); i += 32) ((int *)&sp)[i] = ((const int *)(a.specs + job))[i];
      __syncwarp();
      const int t = a.jt[job];
      rem = sp.depth - t;
      keep = t < sp.depth;
      conjmask = 0;
      for (int i = 0; i < sp.nsym; i++) conjmask |= (unsigned)(sp.symconj[i] != 0) << i;
    }
    if (skip) continue;
#pragma unroll
    for (int j = 0; j < EPL; j++) {
      const int e = lane + 32 * j;
      if (e < E) P[e] = a.R[p * E + e];
    }
    const NodeMeta pm = a.meta[p];
    __syncwarp();
    const auto weight = [&](int s, int e) {
      return W[sp.symperm[s][(e >> NQ) & (N - 1)] * N + sp.symperm[s][e & (N - 1)]];
    };
    expand_parent<NQ, ST>(sp, &sp, weight, conjmask, P, C, sF[w], p, pm, rem, keep, BATCH_GS, o, c, lane);
    __syncwarp();
  }
  if (job >= 0) c.flush(a.jst + job, lane);
}

// A chunk that holds one job: its spec is a kernel parameter, as in the plain level kernel (k_expand), so the level
// code keeps that kernel's register allocation (the many-job kernel above reads the spec from shared memory and
// spills at the same register limit); outputs, child indices and the job's tallies are the many-job kernel's.
template <int NQ, typename ST, int PART>
__global__ void __launch_bounds__(EXP_WARPS * 32, EXP_MINB) k_expand_solo(const DevSpec sp, const BatchArgs<ST> a,
                                                                         int job) {
  constexpr int E = (1 << NQ) * (1 << NQ);
  if (a.gshort && !a.gshort->ovf && a.gshort->count <= GOAL_LIST && a.jgoal[job].x > 0) return;   // its found level
  __shared__ ExpandSmem<NQ, ST> sm;
  __shared__ DevSpec s_sp;
  for (int i = threadIdx.x; i < (int)(sizeof(DevSpec) / 4); i += blockDim.x) ((int *)&s_sp)[i] = ((const int *)&sp)[i];
  __syncthreads();
  init_group_weights<NQ>(sm.Wt, s_sp);
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned conjmask = 0;
  for (int i = 0; i < sp.nsym; i++) conjmask |= (unsigned)(sp.symconj[i] != 0) << i;
  const int t = a.jt[job];
  const ExpandOut<ST> o{a.st, a.cap, a.sh1, a.sh2, a.sidx, a.smeta, a.tq, a.tqcap};
  const auto weight = [&](int s, int e) { return sm.Wt[s][e & (E - 1)]; };
  WarpTally c;
  walk_parents<NQ, ST>(sm, PART == 2 ? &a.st->work2 : &a.st->work, (unsigned long long)a.p0, (unsigned long long)a.m, a.R,
                       a.meta, w, lane, 1, [&](unsigned long long p, const Z4<ST> *P, const NodeMeta &pm, int) {
    expand_parent<NQ, ST, false, PART>(sp, &s_sp, weight, conjmask, P, sm.C[w], sm.F[w], p, pm, sp.depth - t, t < sp.depth,
                                       BATCH_GS, o, c, lane);
  });
  c.flush(a.jst + job, lane);
}

// a survivor's residual: its parent (index sidx / GS in frontier R) times its gate g = sidx % GS, into C; P is the
// warp's staging buffer. The same warp_child as the level kernel, so the result is the residual it evaluated.
template <int NQ, typename ST>
__device__ __forceinline__ void warp_materialize(const Z4<ST> *R, const NodeMeta *meta, unsigned long long sidx, int GS,
                                                 const DevSpec &sp, const DevSpec *sps, Z4<ST> *P, Z4<ST> *C, int lane) {
  constexpr int E = (1 << NQ) * (1 << NQ), EPL = E >= 32 ? E / 32 : 1;
  const unsigned long long p = sidx / (unsigned long long)GS;
  const int g = (int)(sidx % (unsigned long long)GS);
  __syncwarp();
#pragma unroll
  for (int j = 0; j < EPL; j++) {
    const int e = lane + 32 * j;
    if (e < E) P[e] = R[p * E + e];
  }
  __syncwarp();
  bool ovf;
  (void)warp_child<NQ, ST>(P, C, g, meta[p].k, sp, sps, lane, ovf);
  __syncwarp();
}

// child index o = parent * GS + gate: below 2^32 by one 32-bit division
__device__ __forceinline__ unsigned long long child_parent(unsigned long long o, int GS, int &g) {
  const unsigned long long p = (o >> 32) ? o / (unsigned long long)GS : (unsigned long long)((unsigned)o / (unsigned)GS);
  g = (int)(o - p * (unsigned long long)GS);
  return p;
}
// The lane's entries of a survivor's residual, straight from its parent Pg in global memory: unit monomials read the
// permuted entry, one-qubit unit gates their column pair; any other gate goes through warp_child and shared memory (P, C).
// x[j] is the entry at ei[j] (negative: none); every position is in one lane.
template <int NQ, typename ST>
__device__ __forceinline__ void child_entries(const Z4<ST> *Pg, int kp, int g, const DevSpec &sp, Z4<ST> *P, Z4<ST> *C, int lane,
                                              Z4<ST> (&x)[2], int (&ei)[2]) {
  constexpr int N = 1 << NQ, E = N * N;
  ei[0] = ei[1] = -1;
  x[0] = x[1] = Z4<ST>{0, 0, 0, 0};
  if (sp.gflags[g] & GF_UNITMON) {
    const int mono = sp.gmono[g][lane & (N - 1)];
#pragma unroll
    for (int j = 0; j < 2; j++)
      if (lane + 32 * j < E) {
        ei[j] = lane + 32 * j;
        x[j] = mono_entry<NQ>(Pg, mono, lane, j);
      }
    return;
  }
  if constexpr (sizeof(ST) == 4) {
    if (sp.gkind[g] == GK_ONEQ && kp <= 56) {
      const int q = sp.gq[g][0], lo = (1 << q) - 1;
      I4 v[2] = {I4{0, 0, 0, 0}, I4{0, 0, 0, 0}};
      if (lane < E / 2) {
        ei[0] = ((lane & ~lo) << 1) | (lane & lo);
        ei[1] = ei[0] | (1 << q);
        oneq_pair(Pg, ei, sp.gph[g], v);
      }
      (void)normalise_pair(v, kp + sp.gik[g]);
#pragma unroll
      for (int j = 0; j < 2; j++) x[j] = Z4<ST>{(ST)v[j].a, (ST)v[j].b, (ST)v[j].c, (ST)v[j].d};
      return;
    }
  }
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 2; j++)
    if (lane + 32 * j < E) P[lane + 32 * j] = Pg[lane + 32 * j];
  __syncwarp();
  bool ovf;
  (void)warp_child<NQ, ST>(P, C, g, kp, sp, &sp, lane, ovf);
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 2; j++)
    if (lane + 32 * j < E) {
      ei[j] = lane + 32 * j;
      x[j] = C[lane + 32 * j];
    }
}

// ---------------- deferred T bounds ----------------
// One warp per queued entry: recompute the child from its parent, evaluate the T bound once for the entry's
// children, finish their alive test, and write the survivors' records, as the level kernel would have. With jobs
// (fjob != nullptr) the parent's job gives the spec, level and counters.
constexpr int TB_WARPS = 8;
constexpr int TB_MINB = 2;   // blocks per SM asked for: 2 (128 registers) 6.40 ms, 3 (80) 6.87 ms, 4 (64, spills) 6.51 ms
                             // over the two budget 12 proofs
template <typename ST> struct TBoundArgs {
  const Z4<ST> *R;
  const NodeMeta *meta;
  const TQEntry *tq;
  unsigned long long tqcap;
  uint32_t *left;                   // the entries that the packed form leaves to the general one (nullptr: all of them)
  int GS, rem, keep;                // rem, keep: without jobs
  const uint32_t *fjob;
  const DevSpec *specs;
  const int *jt;
  DevStats *jst;
  DevStats *st;                     // queue counters, survivor slots (and the counters without jobs)
  unsigned long long cap;
  uint64_t *sh1, *sh2, *sidx;
  NodeMeta *smeta;
};
// One block's warps walk the queue with a fixed stride. Bound by issue: a dead entry (most are) is the child's update,
// its packing and one packed round. 3.96 M entries of two budget 12 proofs: 32.7 ms with 32-bit components, 11.7 ms
// packed, 5.9 ms with the diagonal update in registers, the general form apart and one alive test; with the children
// that their parent's columns already decide (cols_t_least) left out, 0.57 M entries in 2.4 ms.
// GENERAL: the general form, in a launch of its own over the entries that the packed one listed (or the whole queue): its
// 128 transform values per lane take the registers of one block per SM.
template <int NQ, typename ST, bool BATCHED, bool GENERAL>
__global__ void __launch_bounds__(TB_WARPS * 32, GENERAL ? 1 : TB_MINB)
    k_tbound(const __grid_constant__ DevSpec sp0, const TBoundArgs<ST> a) {
  constexpr int N = 1 << NQ, E = N * N, EPL = E >= 32 ? E / 32 : 1, CHUNKS = E * (int)sizeof(Z4<ST>) / 16;
  constexpr bool PACKED = !GENERAL;
  static_assert(GENERAL || sizeof(ST) == 4, "the packed form is of int32 limbs");
  constexpr int NB = sizeof(ST) == 4 ? 2 : 1;            // int64 limbs: one buffer (shared memory), no overlap
  __shared__ __align__(16) Z4<ST> sP[TB_WARPS][NB][E];  // the entry's parent, and the next entry's arriving
  __shared__ Z4<ST> sC[TB_WARPS][E];
  __shared__ int4 sY[PACKED ? TB_WARPS : 1][PACKED ? E : 1];
  __shared__ int sX[PACKED ? TB_WARPS : 1][PACKED ? E : 1];
  __shared__ uint64_t W[E];
  __shared__ DevSpec s_sp;
  const unsigned long long queued = GENERAL && a.left ? a.st->n_left : a.st->n_tq, n = queued < a.tqcap ? queued : a.tqcap;
  const unsigned long long stride = (unsigned long long)gridDim.x * TB_WARPS;
  if ((unsigned long long)blockIdx.x * TB_WARPS >= n) return;
  init_weights(W, E);
  // the search's spec is copied to shared memory once; a batch's entries read their job's spec where it lies (the
  // entries of a many-job chunk change job often, and the specs stay in cache)
  unsigned conjmask = 0;
  if constexpr (!BATCHED) {
    for (int i = threadIdx.x; i < (int)(sizeof(DevSpec) / 4); i += blockDim.x) ((int *)&s_sp)[i] = ((const int *)&sp0)[i];
    for (int i = 0; i < sp0.nsym; i++) conjmask |= (unsigned)(sp0.symconj[i] != 0) << i;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  Z4<ST> *C = sC[w];
  const DevSpec *spp = &s_sp;
  unsigned nalive = 0, ndead = 0, neval = 0;           // tallies of the current job (or the whole search)
  auto flush = [&](DevStats *st) {
    if (lane == 0) {
      if (ndead) atomicAdd(&st->dead, (unsigned long long)ndead);
      if (nalive) atomicAdd(&st->alive, (unsigned long long)nalive);
      if (neval) atomicAdd(&st->t_evals, (unsigned long long)neval);
    }
    nalive = ndead = neval = 0;
  };
  int job = -2, rem = a.rem;
  bool keep = a.keep != 0;
  // entries are read one ahead: the next entry's parent residual is copied into shared memory asynchronously
  // (cp.async) while the current entry's T bound runs
  auto take = [&](TQEntry &q, unsigned long long e, int b) {
    if (e >= n) return false;
    q = a.tq[GENERAL && a.left ? a.left[e] : e];
    const char *src = (const char *)(a.R + q.p * (unsigned long long)E);
    char *dst = (char *)sP[w][b];
    for (int i = lane; i < CHUNKS; i += 32) cp_async16(dst + 16 * i, src + 16 * i);
    return true;
  };
  TQEntry q;
  int b = 0;
  unsigned long long e = (unsigned long long)blockIdx.x * TB_WARPS + w;
  bool have = take(q, e, 0);
  cp_async_commit();
  while (have) {
    TQEntry q2;
    bool more = false;
    e += stride;
    if constexpr (NB == 2) {
      more = take(q2, e, b ^ 1);
      cp_async_commit();
      cp_async_wait<1>();                            // this entry's parent has arrived (the next may be in flight)
    } else {
      cp_async_wait<0>();
    }
    __syncwarp();
    const Z4<ST> *P = sP[w][b];
    if constexpr (BATCHED) {
      const int pj = (int)a.fjob[q.p];
      if (pj != job) {                               // the spec of this entry's job
        if (job >= 0) flush(a.jst + job);
        job = pj;
        spp = a.specs + job;
        const int t = a.jt[job];
        rem = spp->depth - t; keep = t < spp->depth;
        conjmask = 0;
        for (int i = 0; i < spp->nsym; i++) conjmask |= (unsigned)(spp->symconj[i] != 0) << i;
      }
    }
    const DevSpec &sp = *spp;
    const NodeMeta pm = a.meta[q.p];
    // the largest T bound a child lives with: lane T tries T (combine is monotone in it), so one evaluation per child
    int thr[2];
    const int h = q.k > q.hs ? q.k : q.hs;
#pragma unroll
    for (int s2 = 0; s2 < 2; s2++) {
      const bool ok = s2 < q.n && (sp.lite ? q.k + (lane + sp.tdiv - 1) / sp.tdiv <= rem
                                           : combine(h, lane, q.c2, __popc(q.ntriv[s2])) <= rem);
      thr[s2] = 31 - __clz((int)__ballot_sync(FULL, ok));
    }
    // the packed form takes the children of one-qubit unit monomials (t, tdg): the parent's entries times units, so the
    // exponent stays the parent's (tbound_forms knows when every entry is such)
    const int col = lane & (N - 1);
    int mine = q.n;                                  // the entry's children, none when it is left to the general form
    if (PACKED && !(sp.unit && NQ + q.k <= PACK_MAX && q.k == pm.k && (sp.gflags[q.g[0]] & GF_UNITMON) &&
                    (q.n < 2 || (sp.gflags[q.g[1]] & GF_UNITMON)))) {
      mine = 0;
      if (lane == 0) {
        const unsigned long long l = atomicAdd(&a.st->n_left, 1ULL);
        if (a.left) a.left[l] = (uint32_t)(e - stride);
      }
    }
    bool ovf;
    int T = 0;
    uint64_t cols = 0;
    if (mine) neval++;
    if constexpr (GENERAL) {
      (void)warp_child<NQ, ST>(P, C, q.g[0], pm.k, sp, &sp, lane, ovf);   // the level kernel's child residual
      __syncwarp();
      T = ptm_bound<NQ, ST>(C, q.k, lane);
    } else if (mine) {
      const int mono0 = sp.gmono[q.g[0]][col];
#pragma unroll
      for (int j = 0; j < EPL; j++)
        if (lane + 32 * j < E) {
          const int4 y = pack_entry(mono_entry<NQ>(P, mono0, lane, j));
          sY[w][lane + 32 * j] = y;
          sX[w][lane + 32 * j] = y.x;
        }
      __syncwarp();
      T = packed_tbound<NQ>(sY[w], sX[w], q.k, lane, max(thr[0], thr[1]), keep && NQ == 3, cols);   // T <= 2 (NQ + k) < 31:
                                                                                          // thr is exact
    }
    for (int s2 = 0; s2 < mine; s2++) {
      const bool alive = T < 31 ? T <= thr[s2]
                                : (sp.lite ? q.k + (T + sp.tdiv - 1) / sp.tdiv <= rem
                                           : combine(h, T, q.c2, __popc(q.ntriv[s2])) <= rem);
      if (!alive) { ndead++; continue; }
      nalive++;
      if (!keep) continue;
      if constexpr (GENERAL) {
        if (s2) {                                    // the sibling's residual
          __syncwarp();
          (void)warp_child<NQ, ST>(P, C, q.g[s2], pm.k, sp, &sp, lane, ovf);
        }
      } else {
#pragma unroll
        for (int j = 0; j < EPL; j++)
          if (lane + 32 * j < E) C[lane + 32 * j] = mono_entry<NQ>(P, sp.gmono[q.g[s2]][col], lane, j);
      }
      __syncwarp();
      uint64_t k1, k2;
      warp_class_key<NQ, ST>(C, q.k, sp.nsym, conjmask, sp.symperm, W, lane, k1, k2);
      unsigned long long slot = 0;
      if (lane == 0) slot = atomicAdd(&a.st->n_surv, 1ULL);
      slot = __shfl_sync(FULL, slot, 0);
      if (slot < a.cap) {
        if (lane == 0) {
          a.sh1[slot] = k1; a.sh2[slot] = k2; a.sidx[slot] = q.p * (unsigned long long)a.GS + q.g[s2];
          NodeMeta nm;
          nm.k = q.k; nm.T = (uint8_t)(T > 255 ? 255 : T); nm.c2 = q.c2; nm.g1 = q.g[s2]; nm.g2 = pm.g1;
          nm.hsn = (uint8_t)((q.hs == 2 ? 1 : 0) | (q.ntriv[s2] << 1));
          nm.needs = q.needs;
          nm.cols = cols;
          if (s2 && cols) {                        // the sibling differs by a power of S: an odd one exchanges X and Y
            const uint8_t *a0 = sp.gph[q.g[0]], *a1 = sp.gph[q.g[1]];
            if ((a0[3] - a0[0] - a1[3] + a1[0]) & 3) nm.cols = cols_after(cols, COL_S | sp.gq[q.g[0]][0] << 3);
          }
          a.smeta[slot] = nm;
        }
      } else if (lane == 0) {
        a.st->surv_overflow = 1;
      }
      __syncwarp();
    }
    __syncwarp();                                    // every lane is done with this buffer before it is refilled
    if constexpr (NB == 1) {
      more = take(q2, e, 0);
      cp_async_commit();
    }
    have = more;
    q = q2;
    b ^= NB - 1;
  }
  cp_async_wait<0>();
  if constexpr (BATCHED) { if (job >= 0) flush(a.jst + job); }
  else flush(a.st);
}

// the root node's bounds (the target itself), inherited or bracketed by its children
template <int NQ, typename ST> __global__ void k_root(const DevSpec sp, const Z4<ST> *R, NodeMeta *meta, int tk) {
  constexpr int E = (1 << NQ) * (1 << NQ);
  __shared__ Z4<ST> S[E];
  __shared__ int4 Y[E];
  __shared__ int X[E];
  const int lane = threadIdx.x;
  for (int e = lane; e < E; e += 32) S[e] = R[e];
  __syncwarp();
  int T = 0, c2 = 0, needs = 0;
  uint64_t cols = 0;
  Cheap ch{false, 0, 0};
  if (sp.standard || sp.lite) {
    if (sp.unit && NQ + tk <= PACK_MAX) {
      for (int e = lane; e < E; e += 32) { Y[e] = pack_entry(S[e]); X[e] = Y[e].x; }
      __syncwarp();
      T = packed_tbound<NQ>(Y, X, tk, lane, INT_MAX, NQ == 3, cols);
    } else {
      T = ptm_bound<NQ, ST>(S, tk, lane);
    }
  }
  if (sp.standard) {
    c2 = warp_cx_bound<NQ, ST>(S, sp, lane, 0, 0, needs);
    ch = warp_cheap<NQ, ST>(S, tk, sp, lane, false, true, (1 << NQ) - 1, 0);
  }
  if (lane == 0) {
    NodeMeta m;
    m.k = (int16_t)tk; m.T = (uint8_t)(T > 255 ? 255 : T); m.c2 = (uint8_t)c2; m.g1 = m.g2 = 0xff;
    m.hsn = (uint8_t)((ch.hs == 2 ? 1 : 0) | (ch.ntriv << 1));
    m.needs = (uint8_t)needs;
    m.cols = cols;
    *meta = m;
  }
}

// bounds of caller-given residuals (one warp each): T bound, CX bound, H structure, support
template <int NQ, typename ST>
__global__ void __launch_bounds__(EXP_WARPS * 32) k_eval_bounds(const DevSpec sp, const Z4<ST> *R, const int *ks,
                                                               int count, int4 *out) {
  constexpr int E = (1 << NQ) * (1 << NQ);
  __shared__ Z4<ST> S[EXP_WARPS][E];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int i = blockIdx.x * EXP_WARPS + w; i < count; i += gridDim.x * EXP_WARPS) {
    for (int e = lane; e < E; e += 32) S[w][e] = R[(size_t)i * E + e];
    __syncwarp();
    const int T = ptm_bound<NQ, ST>(S[w], ks[i], lane);
    int needs = 0;
    const int c2 = sp.ncuts ? warp_cx_bound<NQ, ST>(S[w], sp, lane, 0, 0, needs) : 0;
    const Cheap ch = warp_cheap<NQ, ST>(S[w], ks[i], sp, lane, true, true, (1 << NQ) - 1, 0);
    if (lane == 0) out[i] = make_int4(T, c2, ch.goal ? -1 : ch.hs, ch.goal ? -1 : __popc(ch.ntriv));
    __syncwarp();
  }
}

// ---------------- dedupe ----------------
__global__ void k_sort_init(const uint64_t *h1, size_t n, uint64_t *keys, uint32_t *vals) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    keys[i] = h1[i];
    vals[i] = (uint32_t)i;
  }
}

// runs of equal top-32 key bits: singletons are kept at once, longer runs go to the exact resolver
__global__ void k_runs(const uint64_t *keys, const uint32_t *slots, size_t n, const uint64_t *sidx, uint64_t *kidx,
                       uint32_t *kslot, uint2 *work, DevStats *st) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t hk = (uint32_t)(keys[i] >> 32);
    if (i > 0 && (uint32_t)(keys[i - 1] >> 32) == hk) continue;
    size_t j = i + 1;
    while (j < n && (uint32_t)(keys[j] >> 32) == hk) j++;
    if (j == i + 1) {
      const unsigned long long pos = atomicAdd(&st->n_kept, 1ULL);
      kidx[pos] = sidx[slots[i]];
      kslot[pos] = slots[i];
    } else {
      const unsigned long long w = atomicAdd(&st->n_work, 1ULL);
      work[w] = make_uint2((unsigned)i, (unsigned)(j - i));
    }
  }
}

// are A (the lane's entries av at positions ei) and B (in shared memory) one class: some group element maps A to B
template <int NQ, typename ST>
__device__ __forceinline__ bool warp_same_entries(const Z4<ST> (&av)[2], const int (&ei)[2], const Z4<ST> *B, const DevSpec &sp,
                                                  const uint8_t (*perm)[8]) {
  constexpr int N = 1 << NQ;
  for (int s = 0; s < sp.nsym; s++) {
    bool eq = true;
#pragma unroll
    for (int j = 0; j < 2; j++) {
      if (ei[j] < 0) continue;
      const Z4<ST> v = sp.symconj[s] ? zcj(av[j]) : av[j];
      if (!zq(v, B[perm[s][ei[j] >> NQ] * N + perm[s][ei[j] & (N - 1)]])) eq = false;
    }
    if (__all_sync(FULL, eq)) return true;
  }
  return false;
}
template <int NQ, typename ST>
__device__ bool warp_same_class(const Z4<ST> *A, const Z4<ST> *B, const DevSpec &sp, const uint8_t (*perm)[8], int lane) {
  constexpr int E = (1 << NQ) * (1 << NQ);
  Z4<ST> av[2];
  int ei[2];
#pragma unroll
  for (int j = 0; j < 2; j++) {
    ei[j] = lane + 32 * j < E ? lane + 32 * j : -1;
    av[j] = ei[j] >= 0 ? A[ei[j]] : Z4<ST>{0, 0, 0, 0};
  }
  return warp_same_entries<NQ, ST>(av, ei, B, sp, perm);
}

constexpr int RES_WARPS = 4;       // warps per resolve / materialize block
constexpr int RES_MINB = 8;        // resolve blocks per SM: 8 (64 registers) 2.7 ms, 6 3.8 ms, 5 3.6 ms (two budget 12 proofs)
template <int NQ, typename ST> struct ResolveSmem {
  static constexpr int E = (1 << NQ) * (1 << NQ);
  Z4<ST> A[RES_WARPS][E], B[RES_WARPS][E], P[RES_WARPS][E];
  uint8_t ord[RES_WARPS][32];
};

// one warp per run: order members by (h1, h2, index), then keep the first member of every exact class. With jobs
// (fjob != nullptr) members of different jobs are never one class and each job's spec and symmetry group apply.
// A run of up to 32 members (nearly all have two or three) is held one member per lane: ordered by shuffles, its kept
// members a bit mask, written with one counter update. Longer runs order themselves in tmp. Bound by the latency of a
// run's loads (members, then parents): the two budget 12 proofs' runs took 4.5 ms with every run ordered in memory and its
// members rebuilt through shared memory, 2.7 ms so.
template <int NQ, typename ST>
__global__ void __launch_bounds__(RES_WARPS * 32, sizeof(ST) == 4 ? RES_MINB : 4) k_resolve(
    const DevSpec sp, const DevSpec *specs, const uint32_t *fjob, int GS, const Z4<ST> *R, const NodeMeta *meta,
    const uint2 *work, const uint32_t *slots, const uint64_t *sh1, const uint64_t *sh2, const uint64_t *sidx,
    const NodeMeta *smeta, uint32_t *tmp, uint64_t *kidx, uint32_t *kslot, DevStats *st) {
  constexpr int E = (1 << NQ) * (1 << NQ);
  __shared__ ResolveSmem<NQ, ST> sm;
  __shared__ DevSpec s_sp;
  const unsigned long long nwork = st->n_work;
  if ((unsigned long long)blockIdx.x * RES_WARPS >= nwork) return;
  if (!specs)
    for (int i = threadIdx.x; i < (int)(sizeof(DevSpec) / 4); i += blockDim.x) ((int *)&s_sp)[i] = ((const int *)&sp)[i];
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  Z4<ST> *B = sm.B[w], *P = sm.P[w], *C = sm.A[w];
  const unsigned long long nw = (unsigned long long)gridDim.x * RES_WARPS;
  // the exact comparison of two survivors of one job (child indices oa and ob)
  auto same = [&](uint64_t oa, uint64_t ob, uint32_t job) {
    const DevSpec &jsp = specs ? specs[job] : s_sp;
    int ga, gb;
    const unsigned long long pa = child_parent(oa, GS, ga), pb = child_parent(ob, GS, gb);
    Z4<ST> xa[2], xb[2];
    int ea[2], eb[2];
    child_entries<NQ, ST>(R + pa * E, meta[pa].k, ga, jsp, P, C, lane, xa, ea);
    child_entries<NQ, ST>(R + pb * E, meta[pb].k, gb, jsp, P, C, lane, xb, eb);
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 2; j++)
      if (eb[j] >= 0) B[eb[j]] = xb[j];
    __syncwarp();
    const bool r = warp_same_entries<NQ, ST>(xa, ea, B, jsp, jsp.symperm);
    __syncwarp();
    return r;
  };
  auto job_of = [&](uint64_t o) { int g; return fjob ? fjob[child_parent(o, GS, g)] : 0u; };
  for (unsigned long long wi = blockIdx.x * RES_WARPS + w; wi < nwork; wi += nw) {
    const uint2 wk = work[wi];
    const unsigned start = wk.x, len = wk.y;
    if (len <= 32) {
      uint32_t slot = 0, job = 0;
      uint64_t h1 = 0, h2 = 0, idx = 0;
      int k = 0;
      if ((unsigned)lane < len) {
        slot = slots[start + lane];
        h1 = sh1[slot]; h2 = sh2[slot]; idx = sidx[slot];
        k = smeta[slot].k;
        job = job_of(idx);
      }
      int rank = 0;
      for (int b = 0; b < (int)len; b++) {
        const uint64_t bh1 = __shfl_sync(FULL, h1, b), bh2 = __shfl_sync(FULL, h2, b), bix = __shfl_sync(FULL, idx, b);
        rank += (bh1 < h1) || (bh1 == h1 && (bh2 < h2 || (bh2 == h2 && bix < idx)));
      }
      __syncwarp();
      if ((unsigned)lane < len) sm.ord[w][rank] = (uint8_t)lane;
      __syncwarp();
      unsigned kept = 0, group = 0;                    // by lane: kept members; kept members of the current key
      for (unsigned i = 0; i < len; i++) {
        const int li = sm.ord[w][i];
        if (i > 0) {
          const int lp = sm.ord[w][i - 1];
          if (__shfl_sync(FULL, h1, lp) != __shfl_sync(FULL, h1, li) || __shfl_sync(FULL, h2, lp) != __shfl_sync(FULL, h2, li))
            group = 0;
        }
        const int ki = __shfl_sync(FULL, k, li);
        const uint32_t ji = __shfl_sync(FULL, job, li);
        unsigned cand = group & __ballot_sync(FULL, k == ki && job == ji);
        bool dup = false;
        for (; cand && !dup; cand &= cand - 1)
          dup = same(__shfl_sync(FULL, idx, li), __shfl_sync(FULL, idx, __ffs((int)cand) - 1), ji);
        if (!dup) group |= 1u << li;
        kept |= group & (1u << li);
      }
      unsigned long long pos = 0;
      if (lane == 0) pos = atomicAdd(&st->n_kept, (unsigned long long)__popc(kept));
      pos = __shfl_sync(FULL, pos, 0) + __popc(kept & ((1u << lane) - 1));
      if ((kept >> lane) & 1) { kidx[pos] = idx; kslot[pos] = slot; }
      continue;
    }
    for (unsigned a0 = 0; a0 < len; a0 += 32) {          // rank of member a among the run
      const unsigned ai = a0 + lane;
      uint64_t ah1 = 0, ah2 = 0, aix = 0;
      uint32_t as = 0;
      if (ai < len) { as = slots[start + ai]; ah1 = sh1[as]; ah2 = sh2[as]; aix = sidx[as]; }
      unsigned rank = 0;
      for (unsigned b = 0; b < len; b++) {
        const uint32_t bs = slots[start + b];
        const uint64_t bh1 = sh1[bs], bh2 = sh2[bs], bix = sidx[bs];
        rank += (bh1 < ah1) || (bh1 == ah1 && (bh2 < ah2 || (bh2 == ah2 && bix < aix)));
      }
      if (ai < len) tmp[start + rank] = as;
    }
    __syncwarp();
    unsigned gstart = 0;
    for (unsigned i = 0; i < len; i++) {
      const uint32_t si = tmp[start + i] & 0x7fffffffu;
      if (i > 0) {
        const uint32_t sp0 = tmp[start + i - 1] & 0x7fffffffu;
        if (sh1[sp0] != sh1[si] || sh2[sp0] != sh2[si]) gstart = i;
      }
      const uint32_t ji = job_of(sidx[si]);
      bool dup = false;
      for (unsigned i2 = gstart; i2 < i && !dup; i2++) {
        const uint32_t t2 = tmp[start + i2];
        if (!(t2 & 0x80000000u)) continue;
        const uint32_t s2 = t2 & 0x7fffffffu;
        if (smeta[s2].k != smeta[si].k) continue;
        if (fjob && job_of(sidx[s2]) != ji) continue;
        dup = same(sidx[si], sidx[s2], ji);
      }
      if (!dup && lane == 0) {
        tmp[start + i] = si | 0x80000000u;
        const unsigned long long pos = atomicAdd(&st->n_kept, 1ULL);
        kidx[pos] = sidx[si];
        kslot[pos] = si;
      }
      __syncwarp();
    }
  }
}

__global__ void k_keep_all(const uint64_t *sidx, size_t n, uint64_t *kidx, uint32_t *kslot) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    kidx[i] = sidx[i];
    kslot[i] = (uint32_t)i;
  }
}

// kept survivors (in index order) -> the next frontier: residual recomputed from the parent, bounds, tree links
// (and job ids, with jobs). One warp per kept child; consecutive warps mostly share a parent, whose entries come straight
// from L2. Bound by the latency of the chain index -> parent -> entries, and by the 1 KB written per node (3 qubits): 2.6 M
// nodes of two budget 12 proofs took 2.2 ms through shared memory, 1.3 ms so.
template <int NQ, typename ST>
__global__ void __launch_bounds__(RES_WARPS * 32, sizeof(ST) == 4 ? 8 : 4) k_materialize(
    const DevSpec sp, const DevSpec *specs, const uint32_t *fjob, int GS, const Z4<ST> *R, const NodeMeta *meta,
    const uint64_t *kidx, const uint32_t *kslot, size_t nk, const NodeMeta *smeta, Z4<ST> *R2, NodeMeta *meta2, uint32_t *par,
    uint8_t *gat, uint32_t *fjob2) {
  constexpr int E = (1 << NQ) * (1 << NQ);
  __shared__ Z4<ST> sP[RES_WARPS][E], sC[RES_WARPS][E];
  __shared__ DevSpec s_sp;
  if (!specs)
    for (int i = threadIdx.x; i < (int)(sizeof(DevSpec) / 4); i += blockDim.x) ((int *)&s_sp)[i] = ((const int *)&sp)[i];
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const size_t step = (size_t)gridDim.x * RES_WARPS;
  size_t j = blockIdx.x * (size_t)RES_WARPS + w;
  unsigned long long o = j < nk ? kidx[j] : 0;
  for (; j < nk; j += step) {
    const unsigned long long on = j + step < nk ? kidx[j + step] : 0;   // the next child's index, loaded ahead
    int g;
    const unsigned long long p = child_parent(o, GS, g);
    const uint32_t job = fjob ? fjob[p] : 0;
    const DevSpec &jsp = specs ? specs[job] : s_sp;
    Z4<ST> x[2];
    int ei[2];
    child_entries<NQ, ST>(R + p * E, meta[p].k, g, jsp, sP[w], sC[w], lane, x, ei);
#pragma unroll
    for (int q = 0; q < 2; q++)
      if (ei[q] >= 0) R2[j * E + ei[q]] = x[q];
    if (lane == 0) {
      meta2[j] = smeta[kslot[j]];
      par[j] = (uint32_t)p;
      gat[j] = (uint8_t)g;
      if (fjob2) fjob2[j] = job;
    }
    o = on;
  }
}

// ---------------- distance table (--table K) ----------------
__global__ void k_keys_gather(const uint32_t *order, size_t n, const uint64_t *a1, const uint64_t *a2,
                              const uint32_t *ai, const uint32_t *al, uint64_t *s1, uint64_t *s2, uint32_t *si,
                              uint32_t *sl) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t o = order[i];
    s1[i] = a1[o]; s2[i] = a2[o]; si[i] = ai[o]; sl[i] = al[o];
  }
}
// one key record of a table file, as the reference lays it out: {h1, h2, idx, lvl}, 24 bytes
struct KeyRec { uint64_t h1, h2; uint32_t idx, lvl; };
static_assert(sizeof(KeyRec) == 24, "key record layout");
__global__ void k_keys_pack(const uint64_t *s1, const uint64_t *s2, const uint32_t *si, const uint32_t *sl, long long n,
                            KeyRec *r) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    r[i] = KeyRec{s1[i], s2[i], si[i], sl[i]};
}
__global__ void k_keys_unpack(const KeyRec *r, long long n, uint64_t *s1, uint64_t *s2, uint32_t *si, uint32_t *sl) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const KeyRec x = r[i];
    s1[i] = x.h1; s2[i] = x.h2; si[i] = x.idx; sl[i] = x.lvl;
  }
}
// class keys of a materialized frontier from its survivor records: node j came from survivor slot vi[j], whose
// keys the level kernels computed with the same class hash
__global__ void k_keys_from_slots(const uint32_t *vi, long long n, const uint64_t *sh1, const uint64_t *sh2,
                                  uint64_t *F1, uint64_t *F2) {
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < n; j += (long long)gridDim.x * blockDim.x) {
    const uint32_t sl = vi[j];
    F1[j] = sh1[sl];
    F2[j] = sh2[sl];
  }
}
// the (index, level) columns of the keys of one new table level: 0..n-1 and lvl
__global__ void k_level_ids(uint32_t *idx, uint32_t *lv, long long n, uint32_t lvl) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    idx[i] = (uint32_t)i;
    lv[i] = lvl;
  }
}
// the class key of every node of a frontier (one warp each)
template <int NQ, typename ST>
__global__ void __launch_bounds__(RES_WARPS * 32) k_node_keys(const __grid_constant__ DevSpec sp, const Z4<ST> *R,
                                                            const NodeMeta *meta, long long n, uint64_t *F1,
                                                            uint64_t *F2) {
  constexpr int E = (1 << NQ) * (1 << NQ), EPL = E >= 32 ? E / 32 : 1;
  __shared__ Z4<ST> sC[RES_WARPS][E];
  __shared__ uint64_t W[E];
  init_weights(W, E);
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned conjmask = 0;
  for (int i = 0; i < sp.nsym; i++) conjmask |= (unsigned)(sp.symconj[i] != 0) << i;
  for (long long j = blockIdx.x * (long long)RES_WARPS + w; j < n; j += (long long)gridDim.x * RES_WARPS) {
#pragma unroll
    for (int q = 0; q < EPL; q++) {
      const int e = lane + 32 * q;
      if (e < E) sC[w][e] = R[j * E + e];
    }
    __syncwarp();
    uint64_t k1, k2;
    warp_class_key<NQ, ST>(sC[w], meta[j].k, sp.nsym, conjmask, sp.symperm, W, lane, k1, k2);
    if (lane == 0) { F1[j] = k1; F2[j] = k2; }
    __syncwarp();
  }
}

// the residual of table node (lvl, idx): the identity times the inverses of its path's gates, into C (P, path:
// scratch); returns its exponent
template <int NQ, typename ST>
__device__ int warp_replay(const DevSpec &sp, const uint32_t *const *tpar, const uint8_t *const *tgat, int lvl,
                           uint32_t idx, Z4<ST> *P, Z4<ST> *C, uint8_t *path, int lane) {
  constexpr int N = 1 << NQ, E = N * N, EPL = E >= 32 ? E / 32 : 1;
  if (lane == 0)
    for (int l = lvl; l >= 1; l--) { path[l - 1] = tgat[l][idx]; idx = tpar[l][idx]; }
#pragma unroll
  for (int q = 0; q < EPL; q++) {
    const int e = lane + 32 * q;
    if (e < E) C[e] = (e >> NQ) == (e & (N - 1)) ? Z4<ST>{1, 0, 0, 0} : Z4<ST>{0, 0, 0, 0};
  }
  __syncwarp();
  int k = 0;
  for (int i = 0; i < lvl; i++) {
#pragma unroll
    for (int q = 0; q < EPL; q++) {
      const int e = lane + 32 * q;
      if (e < E) P[e] = C[e];
    }
    __syncwarp();
    bool ovf;
    k = warp_child<NQ, ST>(P, C, path[i], k, sp, &sp, lane, ovf);
    __syncwarp();
  }
  return k;
}

__device__ __forceinline__ long long keys_lower(const uint64_t *S1, long long n, uint64_t h1) {
  long long lo = 0, hi = n;
  while (lo < hi) { const long long mid = (lo + hi) >> 1; if (S1[mid] < h1) lo = mid + 1; else hi = mid; }
  return lo;
}

// table build: is each kept child's class already in the table at a lower level? (hash match, then exact)
template <int NQ, typename ST>
__global__ void __launch_bounds__(RES_WARPS * 32) k_seen_filter(
    const __grid_constant__ DevSpec sp, int GS, const Z4<ST> *R, const NodeMeta *meta, const uint64_t *kidx,
    const uint32_t *kslot, size_t nk, const uint64_t *sh1, const uint64_t *sh2, const NodeMeta *smeta,
    const uint64_t *S1, const uint64_t *S2, const uint32_t *Sidx, const uint32_t *Slvl, long long ns,
    const uint32_t *const *tpar, const uint8_t *const *tgat, uint8_t *old) {
  __shared__ ResolveSmem<NQ, ST> sm;
  __shared__ uint8_t spath[RES_WARPS][64];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (size_t i = blockIdx.x * (size_t)RES_WARPS + w; i < nk; i += (size_t)gridDim.x * RES_WARPS) {
    const uint32_t sl = kslot[i];
    const uint64_t h1 = sh1[sl], h2 = sh2[sl];
    const int ka = smeta[sl].k;
    bool dup = false, haveA = false;
    for (long long x = keys_lower(S1, ns, h1); x < ns && S1[x] == h1 && !dup; x++) {
      if (S2[x] != h2) continue;
      if (!haveA) { warp_materialize<NQ, ST>(R, meta, kidx[i], GS, sp, &sp, sm.P[w], sm.A[w], lane); haveA = true; }
      const int kb = warp_replay<NQ, ST>(sp, tpar, tgat, (int)Slvl[x], Sidx[x], sm.P[w], sm.B[w], spath[w], lane);
      if (kb == ka) dup = warp_same_class<NQ, ST>(sm.A[w], sm.B[w], sp, sp.symperm, lane);
    }
    if (lane == 0) old[i] = dup;
    __syncwarp();
  }
}
__global__ void k_drop_old(const uint64_t *kidx, const uint32_t *kslot, size_t nk, const uint8_t *old, uint64_t *kidx2,
                           uint32_t *kslot2, unsigned long long *cnt) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nk; i += (size_t)gridDim.x * blockDim.x)
    if (!old[i]) {
      const unsigned long long p = atomicAdd(cnt, 1ULL);
      kidx2[p] = kidx[i];
      kslot2[p] = kslot[i];
    }
}
// node j of a frontier against the table: the first entry of its class key with level <= maxc, or -1; the nodes
// with a hit are listed (any order) with their entry
__global__ void k_table_lookup(const uint64_t *F1, const uint64_t *F2, long long n, const uint64_t *S1,
                               const uint64_t *S2, const uint32_t *Slvl, long long ns, int maxc, longlong2 *hits,
                               unsigned long long cap, unsigned long long *nhits) {
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < n; j += (long long)gridDim.x * blockDim.x) {
    long long r = -1;
    for (long long x = keys_lower(S1, ns, F1[j]); x < ns && S1[x] == F1[j]; x++)
      if (S2[x] == F2[j] && (int)Slvl[x] <= maxc) { r = x; break; }
    if (r >= 0) {
      const unsigned long long i = atomicAdd(nhits, 1ULL);
      if (i < cap) hits[i] = make_longlong2(j, r);
    }
  }
}
// the tree arrays of a level whose residuals are not kept: node j is child kidx[j] = parent x GS + gate
__global__ void k_tree_only(const uint64_t *kidx, long long n, int GS, uint32_t *par, uint8_t *gat) {
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < n; j += (long long)gridDim.x * blockDim.x) {
    const unsigned long long o = kidx[j];
    par[j] = (uint32_t)(o / (unsigned long long)GS);
    gat[j] = (uint8_t)(o % (unsigned long long)GS);
  }
}
// one warp: the residual of child sidx = parent x GS + gate, from its parent's, and its exponent
template <int NQ, typename ST>
__global__ void k_child_residual(const __grid_constant__ DevSpec sp, const Z4<ST> *R, const NodeMeta *meta,
                                 unsigned long long sidx, int GS, Z4<ST> *out, int *kout) {
  constexpr int E = (1 << NQ) * (1 << NQ), EPL = E >= 32 ? E / 32 : 1;
  __shared__ Z4<ST> P[E], C[E];
  const int lane = threadIdx.x;
  const unsigned long long p = sidx / (unsigned long long)GS;
  const int g = (int)(sidx % (unsigned long long)GS);
#pragma unroll
  for (int q = 0; q < EPL; q++) {
    const int e = lane + 32 * q;
    if (e < E) P[e] = R[p * E + e];
  }
  __syncwarp();
  bool ovf;
  const int k = warp_child<NQ, ST>(P, C, g, meta[p].k, sp, &sp, lane, ovf);
#pragma unroll
  for (int q = 0; q < EPL; q++) {
    const int e = lane + 32 * q;
    if (e < E) out[e] = C[e];
  }
  if (lane == 0) *kout = k;
}
// one warp: every (entry x, symmetry s) from x0 on with s(E_x) == S exactly, in the reference's order
// (cheese.cu:1570-1575); up to cap pairs into out
template <int NQ, typename ST>
__global__ void k_table_confirm(const __grid_constant__ DevSpec sp, const Z4<ST> *S, int ks, const uint64_t *S1,
                                const uint64_t *S2, const uint32_t *Sidx, const uint32_t *Slvl, long long ns,
                                long long x0, int maxc, const uint32_t *const *tpar, const uint8_t *const *tgat,
                                int2 *out, int cap, int *nout) {
  constexpr int N = 1 << NQ, E = N * N, EPL = E >= 32 ? E / 32 : 1;
  __shared__ Z4<ST> A[E], B[E], P[E];
  __shared__ uint8_t path[64];
  const int lane = threadIdx.x;
#pragma unroll
  for (int q = 0; q < EPL; q++) {
    const int e = lane + 32 * q;
    if (e < E) A[e] = S[e];
  }
  __syncwarp();
  int cnt = 0;
  const uint64_t h1 = S1[x0], h2 = S2[x0];
  for (long long x = x0; x < ns && S1[x] == h1; x++) {
    if (S2[x] != h2 || (int)Slvl[x] > maxc) continue;
    const int kb = warp_replay<NQ, ST>(sp, tpar, tgat, (int)Slvl[x], Sidx[x], P, B, path, lane);
    if (kb != ks) continue;
    for (int sy = 0; sy < sp.nsym; sy++) {
      bool eq = true;
#pragma unroll
      for (int q = 0; q < EPL; q++) {
        const int e = lane + 32 * q;
        if (e >= E) continue;
        const Z4<ST> v = sp.symconj[sy] ? zcj(B[e]) : B[e];
        if (!zq(v, A[sp.symperm[sy][e >> NQ] * N + sp.symperm[sy][e & (N - 1)]])) eq = false;
      }
      if (__all_sync(FULL, eq)) {
        if (lane == 0 && cnt < cap) out[cnt] = make_int2((int)x, sy);
        cnt++;
      }
    }
  }
  if (lane == 0) *nout = cnt < cap ? cnt : cap;
}

// keys of table level lvl from its tree (a table file written by another program): replay + class key
template <int NQ, typename ST>
__global__ void __launch_bounds__(RES_WARPS * 32) k_replay_keys(const __grid_constant__ DevSpec sp, int lvl,
                                                              long long n, const uint32_t *const *tpar,
                                                              const uint8_t *const *tgat, uint64_t *F1, uint64_t *F2) {
  constexpr int E = (1 << NQ) * (1 << NQ);
  __shared__ Z4<ST> sP[RES_WARPS][E], sC[RES_WARPS][E];
  __shared__ uint64_t W[E];
  __shared__ uint8_t spath[RES_WARPS][64];
  init_weights(W, E);
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned conjmask = 0;
  for (int i = 0; i < sp.nsym; i++) conjmask |= (unsigned)(sp.symconj[i] != 0) << i;
  for (long long j = blockIdx.x * (long long)RES_WARPS + w; j < n; j += (long long)gridDim.x * RES_WARPS) {
    const int k = warp_replay<NQ, ST>(sp, tpar, tgat, lvl, (uint32_t)j, sP[w], sC[w], spath[w], lane);
    uint64_t k1, k2;
    warp_class_key<NQ, ST>(sC[w], k, sp.nsym, conjmask, sp.symperm, W, lane, k1, k2);
    if (lane == 0) { F1[j] = k1; F2[j] = k2; }
    __syncwarp();
  }
}

// ---------------- meet in the middle (--mitm) ----------------
// the flat list of backward nodes over levels 1..top: node j sits at level l with off[l] <= j < off[l + 1]
struct MitmLevels { long long off[DMAX + 2]; int top; };

// residual of backward node (lvl, idx): S0 (exponent k0) times the inverses of its path's gates, into C; P, path:
// scratch. Returns its exponent.
template <int NQ>
__device__ int warp_replay_from(const DevSpec &sp, const uint32_t *const *tpar, const uint8_t *const *tgat, int lvl,
                                uint32_t idx, const Z4<int32_t> *S0, int k0, Z4<int32_t> *P, Z4<int32_t> *C,
                                uint8_t *path, int lane, bool &ovf) {
  constexpr int N = 1 << NQ, E = N * N, EPL = E >= 32 ? E / 32 : 1;
  if (lane == 0)
    for (int l = lvl; l >= 1; l--) { path[l - 1] = tgat[l][idx]; idx = tpar[l][idx]; }
#pragma unroll
  for (int q = 0; q < EPL; q++) {
    const int e = lane + 32 * q;
    if (e < E) C[e] = S0[e];
  }
  __syncwarp();
  int k = k0;
  ovf = false;
  for (int i = 0; i < lvl; i++) {
#pragma unroll
    for (int q = 0; q < EPL; q++) {
      const int e = lane + 32 * q;
      if (e < E) P[e] = C[e];
    }
    __syncwarp();
    bool o;
    k = warp_child<NQ, int32_t>(P, C, path[i], k, sp, &sp, lane, o);
    ovf = ovf || o;
    __syncwarp();
  }
  (void)N;
  return k;
}

// K = U R (exponents add), normalised; int64 accumulation, ovf when a limb of K leaves int32
template <int NQ>
__device__ int warp_mul_left(const Z4<int32_t> *U, int ku, const Z4<int32_t> *R, int kr, Z4<int32_t> *K, int lane,
                             bool &ovf) {
  constexpr int N = 1 << NQ, E = N * N;
  Zw v[2] = {Zw{0, 0, 0, 0}, Zw{0, 0, 0, 0}};
  int ei[2] = {-1, -1};
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const int e = lane + 32 * j;
    if (e >= E) continue;
    ei[j] = e;
    const int r = e >> NQ, c = e & (N - 1);
    for (int m = 0; m < N; m++) {
      const Z4<int32_t> u = U[r * N + m];
      if (!(u.a | u.b | u.c | u.d)) continue;
      const Z4<int32_t> x = R[m * N + c];
      v[j] = zadd(v[j], zmul(Zw{u.a, u.b, u.c, u.d}, Zw{x.a, x.b, x.c, x.d}));
    }
  }
  return finish_child<NQ, int32_t>(v, ei, ku + kr, K, lane, ovf);
}

// per-block copies of U and U^dag, and per-warp scratch for the backward keys and the confirmation
template <int NQ> struct MitmSmem {
  static constexpr int E = (1 << NQ) * (1 << NQ);
  Z4<int32_t> U[E], Ud[E];
  Z4<int32_t> P[RES_WARPS][E], C[RES_WARPS][E], K[RES_WARPS][E];
  uint64_t W[E];
  uint8_t path[RES_WARPS][64];
};
template <int NQ>
__device__ void mitm_smem_init(MitmSmem<NQ> &sm, const Z4<int32_t> *U, const Z4<int32_t> *Ud) {
  constexpr int E = MitmSmem<NQ>::E;
  for (int e = threadIdx.x; e < E; e += blockDim.x) { sm.U[e] = U[e]; sm.Ud[e] = Ud[e]; }
  init_weights(sm.W, E);
  __syncthreads();
}
// K of backward node j: U times its residual (rebuilt from U^dag), in sm.K[w]; returns K's exponent
template <int NQ>
__device__ int mitm_bwd_residual(const DevSpec &sp, MitmSmem<NQ> &sm, const MitmLevels &lv, const uint32_t *const *tpar,
                                 const uint8_t *const *tgat, long long j, int ku, int w, int lane, bool &ovf) {
  int l = 1;
  while (l < lv.top && j >= lv.off[l + 1]) l++;
  bool o1, o2;
  const int kr = warp_replay_from<NQ>(sp, tpar, tgat, l, (uint32_t)(j - lv.off[l]), sm.Ud, ku, sm.P[w], sm.C[w],
                                      sm.path[w], lane, o1);
  const int k = warp_mul_left<NQ>(sm.U, ku, sm.C[w], kr, sm.K[w], lane, o2);
  ovf = o1 || o2;
  return k;
}

// keys (h1, h2) of every backward node, hashed like the frontier nodes (no symmetry: the join needs exact residuals)
template <int NQ>
__global__ void __launch_bounds__(RES_WARPS * 32) k_mitm_bwd_keys(const __grid_constant__ DevSpec sp,
                                                                const Z4<int32_t> *U, const Z4<int32_t> *Ud, int ku,
                                                                const __grid_constant__ MitmLevels lv,
                                                                const uint32_t *const *tpar, const uint8_t *const *tgat,
                                                                long long nb, uint64_t *B1, uint64_t *B2, int *ovf) {
  __shared__ MitmSmem<NQ> sm;
  mitm_smem_init<NQ>(sm, U, Ud);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (long long j = blockIdx.x * (long long)RES_WARPS + w; j < nb; j += (long long)gridDim.x * RES_WARPS) {
    bool o;
    const int k = mitm_bwd_residual<NQ>(sp, sm, lv, tpar, tgat, j, ku, w, lane, o);
    uint64_t k1, k2;
    warp_class_key<NQ, int32_t>(sm.K[w], k, 1, 0u, sp.symperm, sm.W, lane, k1, k2);
    if (lane == 0) {
      B1[j] = k1; B2[j] = k2;
      if (o) atomicExch(ovf, 1);
    }
    __syncwarp();
  }
}

// forward keys sorted by h1 (stable): gather (h1, h2, forward index) in sorted order
__global__ void k_mitm_sorted(const uint32_t *order, long long n, const uint64_t *F1, const uint64_t *F2, uint64_t *S1,
                              uint64_t *S2, uint32_t *Si) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const uint32_t o = order[i];
    S1[i] = F1[o]; S2[i] = F2[o]; Si[i] = o;
  }
}
// per backward key: the first sorted forward key equal in (h1, h2), or -1; the matching j are listed (any order)
__global__ void k_mitm_match(const uint64_t *B1, const uint64_t *B2, long long nb, const uint64_t *S1,
                             const uint64_t *S2, long long nf, long long *pos, long long *hits,
                             unsigned long long *nhits) {
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < nb; j += (long long)gridDim.x * blockDim.x) {
    long long r = -1;
    for (long long x = keys_lower(S1, nf, B1[j]); x < nf && S1[x] == B1[j]; x++)
      if (S2[x] == B2[j]) { r = x; break; }
    pos[j] = r;
    if (r >= 0) hits[atomicAdd(nhits, 1ULL)] = j;
  }
}
// exact confirmation of hash matches (one warp per candidate j): the first forward node of the equal-key run whose
// residual equals K = U R'_j exactly (entries and exponent), else -1
template <int NQ>
__global__ void __launch_bounds__(RES_WARPS * 32) k_mitm_confirm(
    const __grid_constant__ DevSpec sp, const Z4<int32_t> *U, const Z4<int32_t> *Ud, int ku,
    const __grid_constant__ MitmLevels lv, const uint32_t *const *tpar, const uint8_t *const *tgat, const long long *cand,
    long long nc, const long long *pos, const uint64_t *S1, const uint64_t *S2, const uint32_t *Si, long long nf,
    const Z4<int32_t> *FR, const NodeMeta *FM, long long *match) {
  constexpr int E = MitmSmem<NQ>::E, EPL = E >= 32 ? E / 32 : 1;
  __shared__ MitmSmem<NQ> sm;
  mitm_smem_init<NQ>(sm, U, Ud);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (long long c = blockIdx.x * (long long)RES_WARPS + w; c < nc; c += (long long)gridDim.x * RES_WARPS) {
    const long long j = cand[c];
    bool o;
    const int k = mitm_bwd_residual<NQ>(sp, sm, lv, tpar, tgat, j, ku, w, lane, o);
    long long r = -1;
    const long long x0 = pos[j];
    for (long long x = x0; x0 >= 0 && x < nf && S1[x] == S1[x0] && r < 0; x++) {
      if (S2[x] != S2[x0]) continue;
      const uint32_t f = Si[x];
      bool eq = FM[f].k == k;
#pragma unroll
      for (int q = 0; q < EPL; q++) {
        const int e = lane + 32 * q;
        if (e < E && !zq(FR[(size_t)f * E + e], sm.K[w][e])) eq = false;
      }
      if (__all_sync(FULL, eq) && !o) r = f;
    }
    if (lane == 0) match[c] = r;
    __syncwarp();
  }
}

__global__ void k_widen(const Z4<int32_t> *in, Z4<int64_t> *out, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const Z4<int32_t> x = in[i];
    out[i] = Z4<int64_t>{x.a, x.b, x.c, x.d};
  }
}

// register-resident multiply-add loop: 8 independent IMAD chains per thread (peak int32 throughput probe)
__global__ void k_imad_probe(int iters, uint32_t m, uint32_t *out) {
  uint32_t a[8];
#pragma unroll
  for (int j = 0; j < 8; j++) a[j] = threadIdx.x * 0x9e3779b9u + j * 0x85ebca6bu + blockIdx.x;
  for (int i = 0; i < iters; i++) {
#pragma unroll
    for (int j = 0; j < 8; j++) a[j] = a[j] * m + (uint32_t)j;
  }
  uint32_t x = 0;
#pragma unroll
  for (int j = 0; j < 8; j++) x ^= a[j];
  if (x == 0x12345678u) out[0] = x;     // keeps the loop live; practically never taken
}

// ---------------- host helpers ----------------
double now_s() { return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count(); }

struct CudaError : std::runtime_error { using std::runtime_error::runtime_error; };
void ck(cudaError_t e, const char *what) {
  if (e != cudaSuccess) {
    cudaGetLastError();            // a failed allocation must not be reported again by the next launch check
    throw CudaError(std::string("CUDA error after ") + what + ": " + cudaGetErrorString(e));
  }
}

struct DBuf {
  void *p = nullptr;
  size_t cap = 0;
  void ensure(size_t bytes) {
    if (bytes <= cap) return;
    const size_t old = cap;
    if (p) ck(cudaFree(p), "free");
    p = nullptr;
    cap = 0;
    // grow by half again below 1 GiB (small buffers in 256-byte steps, at least 64 KiB), exactly (2 MiB granules)
    // once a buffer passes 1 GiB: a stream of growing requests reallocates a buffer only a few times
    size_t c = bytes >= ((size_t)1 << 30) ? bytes : std::max(bytes, old + old / 2);
    if (c < ((size_t)2 << 20)) c = std::max<size_t>((c + 255) & ~(size_t)255, (size_t)64 << 10);
    else c = (c + ((size_t)2 << 20) - 1) & ~(((size_t)2 << 20) - 1);
    if (c >= ((size_t)64 << 20) && std::getenv("CZ_TRACE_ALLOC")) {   // large device allocations, for diagnosis
      size_t fr = 0, tot = 0;
      cudaMemGetInfo(&fr, &tot);
      std::fprintf(stderr, "cz alloc %.3f GB (free %.3f GB)\n", c / 1e9, fr / 1e9);
    }
    ck(cudaMalloc(&p, c), "cudaMalloc");
    cap = c;
  }
  template <typename T> T *as() const { return (T *)p; }
  void release() { if (p) cudaFree(p); p = nullptr; cap = 0; }
};

// A device buffer that grows in place. One large virtual address range is reserved for it; physical memory is
// created and mapped into the range as the buffer grows (the driver's virtual memory management), so growing keeps
// the contents without a copy and frees nothing, and the address never changes. Memory goes back to the device only
// at release(). The driver entry points are looked up through the runtime (no link-time dependency on libcuda).
struct Vmm {
  decltype(&::cuMemAddressReserve) reserve = nullptr;
  decltype(&::cuMemAddressFree) addr_free = nullptr;
  decltype(&::cuMemCreate) create = nullptr;
  decltype(&::cuMemRelease) mem_release = nullptr;
  decltype(&::cuMemMap) map = nullptr;
  decltype(&::cuMemUnmap) unmap = nullptr;
  decltype(&::cuMemSetAccess) set_access = nullptr;
  decltype(&::cuMemGetAllocationGranularity) granularity = nullptr;
  bool ok = false;
  static const Vmm &get() {
    static const Vmm v = [] {
      Vmm x;
      auto look = [](const char *name, void **f) {
        cudaDriverEntryPointQueryResult q;
        return cudaGetDriverEntryPoint(name, f, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess;
      };
      x.ok = look("cuMemAddressReserve", (void **)&x.reserve) && look("cuMemAddressFree", (void **)&x.addr_free) &&
             look("cuMemCreate", (void **)&x.create) && look("cuMemRelease", (void **)&x.mem_release) &&
             look("cuMemMap", (void **)&x.map) && look("cuMemUnmap", (void **)&x.unmap) &&
             look("cuMemSetAccess", (void **)&x.set_access) &&
             look("cuMemGetAllocationGranularity", (void **)&x.granularity);
      return x;
    }();
    return v;
  }
};

struct VBuf {
  static constexpr size_t RESERVE = (size_t)256 << 30;    // address range per buffer (more than the device holds)
  static constexpr size_t STEP = (size_t)256 << 20;       // smallest growth step
  void *p = nullptr;                                      // start of the range (nullptr until the first growth)
  size_t cap = 0;                                         // bytes mapped
  std::vector<std::pair<CUmemGenericAllocationHandle, size_t>> maps;   // physical blocks in address order
  static void drv(CUresult r, const char *what) {
    if (r != CUDA_SUCCESS) throw CudaError(std::string("CUDA driver error ") + std::to_string((int)r) + " in " + what);
  }
  void ensure(size_t bytes) {
    if (bytes <= cap) return;
    const Vmm &v = Vmm::get();
    if (!v.ok) throw CudaError("the driver's virtual memory management entry points are missing");
    int dev = 0;
    ck(cudaGetDevice(&dev), "cudaGetDevice");
    CUmemAllocationProp prop{};
    prop.type = CU_MEM_ALLOCATION_TYPE_PINNED;
    prop.location.type = CU_MEM_LOCATION_TYPE_DEVICE;
    prop.location.id = dev;
    size_t gran = 0;
    drv(v.granularity(&gran, &prop, CU_MEM_ALLOC_GRANULARITY_RECOMMENDED), "cuMemGetAllocationGranularity");
    if (!p) {
      CUdeviceptr base = 0;
      drv(v.reserve(&base, RESERVE, 0, 0, 0), "cuMemAddressReserve");
      p = (void *)base;
    }
    const size_t need = bytes - cap;
    size_t step = std::max(need, std::max(STEP, cap / 8));
    step = (step + gran - 1) / gran * gran;
    if (cap + step > RESERVE) step = (need + gran - 1) / gran * gran;
    if (cap + step > RESERVE) throw CudaError("device buffer larger than its address range");
    CUmemGenericAllocationHandle h;
    if (v.create(&h, step, &prop, 0) != CUDA_SUCCESS) {   // no room for the step: the exact need
      step = (need + gran - 1) / gran * gran;
      drv(v.create(&h, step, &prop, 0), "cuMemCreate (device memory exhausted)");
    }
    const CUdeviceptr at = (CUdeviceptr)p + cap;
    CUresult r = v.map(at, step, 0, h, 0);
    if (r == CUDA_SUCCESS) {
      CUmemAccessDesc acc{};
      acc.location = prop.location;
      acc.flags = CU_MEM_ACCESS_FLAGS_PROT_READWRITE;
      r = v.set_access(at, step, &acc, 1);
      if (r != CUDA_SUCCESS) v.unmap(at, step);
    }
    if (r != CUDA_SUCCESS) { v.mem_release(h); drv(r, "cuMemMap"); }
    maps.push_back({h, step});
    cap += step;
  }
  template <typename T> T *as() const { return (T *)p; }
  // the caller has waited for every use of the buffer on the device
  void release() {
    if (!p) return;
    const Vmm &v = Vmm::get();
    size_t off = 0;
    for (auto &m : maps) {
      v.unmap((CUdeviceptr)p + off, m.second);
      v.mem_release(m.first);
      off += m.second;
    }
    v.addr_free((CUdeviceptr)p, RESERVE);
    maps.clear();
    p = nullptr;
    cap = 0;
  }
};

uint64_t powmod_h(uint64_t a, uint64_t e) {
  uint64_t r = 1;
  while (e) { if (e & 1) r = r * a % PRIME; a = a * a % PRIME; e >>= 1; }
  return r;
}

}  // namespace

// survivor records to provision for `children` children at an expected survivor rate: 1.5x the expectation
// plus 4096, at least 1 Mi (never more than every child), at most 8 GiB of records
inline unsigned long long survivor_room(unsigned long long children, double rate, size_t rec,
                                        size_t lim_bytes = (size_t)8 << 30) {
  const unsigned long long lim = lim_bytes / rec;
  double want = 1.5 * rate * (double)children + 4096.0;
  if (want < (double)(1 << 20)) want = (double)(1 << 20);
  unsigned long long cap = want >= (double)children ? children : (unsigned long long)want;
  return cap > lim ? lim : cap;
}

struct Engine::Impl {
  int dev;
  int nsm = 148;
  cudaStream_t s = nullptr;
  cudaEvent_t ev[4];
  DBuf fR, fMeta, fR2, fMeta2;             // frontier, next frontier
  DBuf sH1, sH2, sIdx, sMeta;              // survivors of the current level (40-byte records)
  DBuf tq, tqleft;                         // deferred T evaluations of the current level; TBoundArgs::left
  DBuf k0, k1, v0, v1, hist, part;         // sort
  DBuf work, tmp, kidx, kslot;             // dedupe
  DBuf gshort;                             // the goal pass: its counters and candidate list
  DBuf stats;
  struct SpecDev {                         // device copies of one parsed spec's tables
    uint64_t uid = 0;
    long long used = 0;
    DBuf ginv, bad2, bad3, cxt, goal, ginfo;
    void release() {
      ginv.release(); bad2.release(); bad3.release(); cxt.release(); goal.release(); ginfo.release(); uid = 0;
    }
  };
  SpecDev specs[8];
  long long use_clock = 0;
  std::vector<DBuf> par, gat;              // tree, one level each
  std::vector<long long> level_n;          // nodes per level of the tree
  struct DistTable {                       // --table K: every class within K gates, its tree and sorted keys
    int K = 0, nl = 0;
    std::vector<DBuf> par, gat;            // [l], l = 1..nl
    std::vector<long long> n;              // [0..nl]
    DBuf S1, S2, Sidx, Slvl;               // class keys sorted by S1 (stable: lower levels first)
    long long ns = 0;
    void release() {
      for (auto &b : par) b.release();
      for (auto &b : gat) b.release();
      S1.release(); S2.release(); Sidx.release(); Slvl.release();
    }
  };
  std::map<std::string, DistTable *> dtabs;   // resident tables by cache path
  DistTable *building = nullptr;           // a table build: children are filtered against it, levels added to it
  bool want_keys = false;
  bool lean_level = false;                 // the last level of a levels() call keeps its tree and keys, not its
                                           // residuals (the last searched level of --table K)                  // keep the frontier's class keys (fK1, fK2)
  DBuf fK1, fK2, tptrs, keys2, old;
  DBuf outb;                               // a table candidate's symmetry elements and residual
  DevStats *hstats = nullptr;              // pinned
  long long launches = 0, expand_launches = 0, h2d = 0, d2h = 0;
  long long front_m = 1;                   // nodes in the current frontier
  int level_dir = 0;                       // the "dir" of the level lines: 2 forward, 3 backward (--mitm)
  struct SideTree {                        // --mitm: the backward tree while the forward one is the engine's own
    std::vector<DBuf> par, gat;
    DBuf fR, fMeta;
    long long front_m = 1;
    std::vector<long long> level_n;
    size_t release() {
      size_t n = fR.cap + fMeta.cap;
      for (auto &b : par) { n += b.cap; b.release(); }
      for (auto &b : gat) { n += b.cap; b.release(); }
      fR.release(); fMeta.release();
      return n;
    }
  } side;
  void swap_side() {                       // make the backward tree the current one, or back
    std::swap(par, side.par); std::swap(gat, side.gat);
    std::swap(fR, side.fR); std::swap(fMeta, side.fMeta);
    std::swap(front_m, side.front_m); std::swap(level_n, side.level_n);
  }

  explicit Impl(int d) : dev(d) {
    ck(cudaSetDevice(dev), "cudaSetDevice");
    ck(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "stream");
    for (auto &e : ev) ck(cudaEventCreate(&e), "event");
    ck(cudaMallocHost(&hstats, sizeof(DevStats) + sizeof(GoalShort)), "pinned");
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    stats.ensure(sizeof(DevStats) + sizeof(GoalShort) + sizeof(SortFlags));
    ck(cudaMemsetAsync(sort_flags(), 0, sizeof(SortFlags), s), "memset");
  }
  SortFlags *sort_flags() { return (SortFlags *)(stats.as<char>() + sizeof(DevStats) + sizeof(GoalShort)); }
  size_t trim() {
    size_t n = 0;
    for (DBuf *b : {&fR, &fMeta, &fR2, &fMeta2, &sH1, &sH2, &sIdx, &sMeta, &tq, &tqleft, &k0, &k1, &v0, &v1, &hist, &part,
                    &work, &tmp, &kidx, &kslot, &fK1, &fK2, &keys2, &old, &gshort, &outb}) {
      n += b->cap;
      b->release();
    }
    for (auto &b : par) { n += b.cap; b.release(); }
    for (auto &b : gat) { n += b.cap; b.release(); }
    n += side.release();
    front_m = 0;
    return n;
  }
  ~Impl() {
    cudaSetDevice(dev);
    for (DBuf *b : {&fR, &fMeta, &fR2, &fMeta2, &sH1, &sH2, &sIdx, &sMeta, &tq, &tqleft, &k0, &k1, &v0, &v1, &hist, &part,
                    &work, &tmp, &kidx, &kslot, &stats})
      b->release();
    for (auto &sd : specs) sd.release();
    for (auto &kv : dtabs) { kv.second->release(); delete kv.second; }
    for (DBuf *b : {&fK1, &fK2, &tptrs, &keys2, &old, &gshort, &outb}) b->release();
    for (auto &b : par) b.release();
    for (auto &b : gat) b.release();
    side.release();
    if (hstats) cudaFreeHost(hstats);
    for (auto &e : ev) cudaEventDestroy(e);
    if (s) cudaStreamDestroy(s);
  }

  template <int NQ> int run(const HostSpec &hs, const Options &opt, const std::function<void(const LevelStats &)> &cb,
                            SearchResult &res);
  template <int NQ> DevSpec prepare(const HostSpec &hs, const SymGroup &grp, int depth, bool nogoal);
  template <int NQ, typename ST>
  void eval_bounds(const HostSpec &hs, int count, const int64_t *ent, const int *ks, int *out4);
  template <int NQ, typename ST>
  int levels(const HostSpec &hs, const DevSpec &sp, const Options &opt, int depth, int &t_start,
             const std::function<void(const LevelStats &)> &cb, SearchResult &res, int stop = 1 << 30);
  // --table K
  template <int NQ> int run_table(const HostSpec &hs, const Options &opt, const std::function<void(const LevelStats &)> &cb,
                                  SearchResult &res);
  template <int NQ> DistTable *get_table(const HostSpec &hs, const SymGroup &grp, int K, const Options &opt,
                                         const std::function<void(const LevelStats &)> &cb, SearchResult &res);
  template <int NQ> int table_levels_keys(const DevSpec &sp, long long n);   // keys of the frontier into fK1/fK2
  // --mitm
  template <int NQ> int run_mitm(const HostSpec &hs, const Options &opt, const std::function<void(const LevelStats &)> &cb,
                                 SearchResult &res);
  void seen_add(DistTable &D, long long n, int lvl);                         // append fK1/fK2 level to D's keys
  const void *const *upload_tree(const std::vector<DBuf> &p, const std::vector<DBuf> &g, int upto);
  bool table_load(const std::string &path, DistTable &D, int K, int G);
  void table_save(const std::string &path, const DistTable &D);
};

// the gates of child o (parent * G + gate) of level t, walked back through the tree's levels, first gate first
struct TreeLevels { const uint32_t *par[DMAX + 1]; const uint8_t *gat[DMAX + 1]; };
__global__ void k_walk_back(const __grid_constant__ TreeLevels tree, unsigned long long o, int G, int t, uint8_t *out) {
  out[t - 1] = (uint8_t)(o % (unsigned)G);
  uint32_t i = (uint32_t)(o / (unsigned)G);
  for (int l = t - 1; l >= 1; l--) {
    out[l - 1] = tree.gat[l][i];
    i = tree.par[l][i];
  }
}

// The forms of the T bound that the queue of level t can need. A spec that is not unitary, and int64 limbs, take the general
// one alone. The packed one takes every child of a unit monomial while its exponent k allows: k is at most the root's plus
// the most a gate adds on each of t - 1 levels, and an entry is queued only with k <= depth - t. The general launch is
// left out where that shows it empty (a launch that finds nothing costs about 4 us; small searches make 50 in a millisecond).
struct TboundForms { bool packed, general; };
template <int NQ, typename ST> TboundForms tbound_forms(const HostSpec &hs, const DevSpec &sp, int t, int depth) {
  if (sizeof(ST) != 4 || !sp.unit) return {false, true};
  if (!hs.standard && !hs.lite) return {true, false};          // no bounds, nothing queued
  int up = 0;
  for (int g = 0; g < hs.G; g++) {
    if (!(hs.gflags[g] & GF_CLIFFORD) && !(sp.gflags[g] & GF_UNITMON)) return {true, true};
    up = std::max(up, hs.gik[g]);
  }
  return {true, NQ + std::min(hs.rk + (t - 1) * up, depth - t) > PACK_MAX};
}
template <int NQ, typename ST, bool BATCHED>
int launch_tbound(const DevSpec &sp, TBoundArgs<ST> a, uint32_t *left, TboundForms f, unsigned grid, cudaStream_t s) {
  a.left = left;
  if constexpr (sizeof(ST) == 4) {
    if (f.packed) k_tbound<NQ, ST, BATCHED, false><<<grid, TB_WARPS * 32, 0, s>>>(sp, a);
  }
  if (f.general) {
    if (!f.packed) a.left = nullptr;
    k_tbound<NQ, ST, BATCHED, true><<<grid, TB_WARPS * 32, 0, s>>>(sp, a);
  }
  return (int)f.packed + (int)f.general;
}

template <int NQ, typename ST>
int Engine::Impl::levels(const HostSpec &hs, const DevSpec &sp, const Options &opt, int depth, int &t_start,
                         const std::function<void(const LevelStats &)> &cb, SearchResult &res, int stop) {
  constexpr int E = (1 << NQ) * (1 << NQ);
  const int G = hs.G;
  long long m = front_m;
  double surv_rate = 1.0;                              // survivors per child of the previous level
  bool ded_pending = false;                            // a level's dedupe events recorded, not yet read
  auto read_dedupe = [&]() {                           // (after a wait on the stream)
    if (!ded_pending) return;
    float ms = 0;
    if (cudaEventElapsedTime(&ms, ev[2], ev[3]) == cudaSuccess) res.dedupe_ms += ms;
    ded_pending = false;
  };
  auto walk_back = [&](unsigned long long o, int t) {  // (the statistics have been read: their buffers carry the gates)
    TreeLevels tree{};
    for (int l = 1; l < t; l++) { tree.par[l] = par[l].as<uint32_t>(); tree.gat[l] = gat[l].as<uint8_t>(); }
    k_walk_back<<<1, 1, 0, s>>>(tree, o, G, t, stats.as<uint8_t>());
    launches++;
    ck(cudaGetLastError(), "walk");
    ck(cudaMemcpyAsync(hstats, stats.p, (size_t)t, cudaMemcpyDeviceToHost, s), "d2h");
    d2h += t;
    ck(cudaStreamSynchronize(s), "walk");
    const uint8_t *q = (const uint8_t *)hstats;
    return std::vector<int>(q, q + t);
  };
  if ((int)level_n.size() < t_start) level_n.resize(t_start, 0);
  for (int t = t_start; t <= depth && t <= stop; t++) {
    const double t0 = now_s();
    const bool keep = t < depth;
    // survivors capacity: the previous level's survivor rate with room to spare (at least 1 Mi records, at most
    // every child); when more survive, the level is redone once with the exact count (the kernel counts every
    // survivor, stored or not)
    size_t lim_bytes = (size_t)8 << 30;         // above 8 GiB of records, up to 40 % of the free device memory
    if (keep && 1.5 * surv_rate * (double)m * G * 48.0 > (double)lim_bytes) {
      size_t fr = 0, tot = 0;
      if (cudaMemGetInfo(&fr, &tot) == cudaSuccess) lim_bytes = std::max(lim_bytes, (size_t)(0.4 * (double)fr));
    }
    unsigned long long cap = keep ? survivor_room((unsigned long long)m * G, surv_rate, 48, lim_bytes) : 0;
    DevStats *dst = stats.as<DevStats>();
    // deferred T evaluations: at most one entry per child of a gate whose T bound is not inherited
    int ncl = 0;
    for (int g = 0; g < G; g++) ncl += !(hs.gflags[g] & GF_CLIFFORD);
    unsigned long long tqcap = (unsigned long long)m * (unsigned long long)std::max(1, ncl) + 1024;
    // goal pass: the parents that may have a goal child, their children tested first (a hit makes this the found
    // level and the level kernels return at once)
    GoalShort *gsd = nullptr;
    GoalShort hgs{0, 0, ~0ULL, 0, 0};
    const bool goal_pass = hs.standard && !hs.states && !sp.nogoal && m > 0;
    if (goal_pass) {                         // its header lies behind the level's statistics: one copy brings both back
      gshort.ensure((size_t)GOAL_LIST * 4 + 64);
      gsd = (GoalShort *)(dst + 1);
    }
    // the level's counters and the goal pass's header set on the device (a copy from pageable host memory would
    // wait for the stream)
    k_level_init<<<1, 32, 0, s>>>(gsd, stats.as<DevStats>());
    launches++;
    if (goal_pass) {
      uint32_t *glist = gshort.as<uint32_t>();
      const unsigned gm_ = (unsigned)std::max<long long>(1, std::min<long long>((m + 255) / 256, (long long)nsm * 8));
      k_goal_candidates<<<gm_, 256, 0, s>>>(fMeta.as<NodeMeta>(), m, glist, gsd);
      k_goal_level<NQ, ST><<<(unsigned)nsm * 2, EXP_WARPS * 32, 0, s>>>(sp, fR.as<Z4<ST>>(), fMeta.as<NodeMeta>(), glist,
                                                                       G, gsd);
      launches += 2;
      ck(cudaGetLastError(), "goal pass");
    }
    for (int attempt = 0; attempt < 2; attempt++) {
      if (keep) {
        sH1.ensure(cap * 8); sH2.ensure(cap * 8); sIdx.ensure(cap * 8);
        sMeta.ensure(cap * sizeof(NodeMeta));
      }
      tq.ensure(tqcap * sizeof(TQEntry));
      const TboundForms forms = tbound_forms<NQ, ST>(hs, sp, t, depth);
      if (forms.packed && forms.general) tqleft.ensure(tqcap * 4);
      if (attempt) { k_level_init<<<1, 32, 0, s>>>(nullptr, dst); launches++; }
      ExpandArgs<ST> a;
      a.m = m; a.t = t; a.rem = depth - t; a.keep = keep;
      a.R = fR.as<Z4<ST>>(); a.meta = fMeta.as<NodeMeta>(); a.st = dst; a.cap = cap;
      a.sh1 = sH1.as<uint64_t>(); a.sh2 = sH2.as<uint64_t>(); a.sidx = sIdx.as<uint64_t>();
      a.smeta = sMeta.as<NodeMeta>();
      a.tq = tq.as<TQEntry>(); a.tqcap = tqcap; a.gshort = gsd;
      // fewer parents than the chip has warps: up to 8 warps share a parent's candidates (a 2-qubit search's level kernels
      // are then a chain of 3 children instead of 16; eight searches: 1.16 -> 0.75 ms of level kernels)
      a.split = (int)std::max<long long>(1, std::min<long long>(8, (long long)nsm * EXP_MINB * EXP_WARPS / std::max<long long>(m, 1)));
      const long long want = (m * a.split + EXP_WARPS - 1) / EXP_WARPS;
      const long long grid = std::max<long long>(1, std::min<long long>(want, (long long)nsm * EXP_MINB));   // one wave
      if (opt.profile) ck(cudaEventRecord(ev[0], s), "event");
      if (hs.states) k_expand<NQ, ST, true><<<(unsigned)grid, EXP_WARPS * 32, 0, s>>>(sp, a);
      else {                                     // one-qubit gates, then the others: two smaller loop bodies
        k_expand<NQ, ST, false, 1><<<(unsigned)grid, EXP_WARPS * 32, 0, s>>>(sp, a);
        k_expand<NQ, ST, false, 2><<<(unsigned)grid, EXP_WARPS * 32, 0, s>>>(sp, a);
        launches++;
      }
      TBoundArgs<ST> tb;
      tb.R = fR.as<Z4<ST>>(); tb.meta = fMeta.as<NodeMeta>(); tb.tq = tq.as<TQEntry>(); tb.tqcap = tqcap;
      tb.GS = G; tb.rem = depth - t; tb.keep = keep; tb.fjob = nullptr; tb.specs = nullptr; tb.jt = nullptr;
      tb.jst = nullptr; tb.st = dst; tb.cap = cap; tb.sh1 = sH1.as<uint64_t>(); tb.sh2 = sH2.as<uint64_t>();
      tb.sidx = sIdx.as<uint64_t>(); tb.smeta = sMeta.as<NodeMeta>();
      launches += 1 + launch_tbound<NQ, ST, false>(sp, tb, forms.general ? tqleft.as<uint32_t>() : nullptr, forms,
                                                   (unsigned)nsm * 4, s);
      expand_launches++;
      ck(cudaGetLastError(), "expand kernel");
      if (opt.profile) ck(cudaEventRecord(ev[1], s), "event");
      const size_t back = sizeof(DevStats) + (gsd ? sizeof(GoalShort) : 0);
      ck(cudaMemcpyAsync(hstats, dst, back, cudaMemcpyDeviceToHost, s), "d2h");
      d2h += (long long)back;
      ck(cudaStreamSynchronize(s), "expand");
      if (gsd) hgs = *(const GoalShort *)(hstats + 1);
      read_dedupe();
      if (gsd && hgs.found && !hgs.ovf && hgs.count <= GOAL_LIST) break;   // the found level (kernels skipped)
      if (opt.profile) { float ms = 0; cudaEventElapsedTime(&ms, ev[0], ev[1]); res.expand_ms += ms; }
      if (hstats->ovf) return -2;                       // promote to int64 limbs and redo this level
      if (!hstats->surv_overflow && hstats->n_tq <= tqcap) break;
      cap = std::max<unsigned long long>(cap, hstats->n_surv);   // exact counts: grow and redo once
      tqcap = std::max<unsigned long long>(tqcap, hstats->n_tq);
    }
    if (gsd && hgs.found && !hgs.ovf && hgs.count <= GOAL_LIST) {   // found by the goal pass
      const unsigned long long o = hgs.first;
      res.circuit = walk_back(o, t);
      res.n_found = (long long)hgs.found;
      res.levels = t;
      return RC_CIRCUIT;
    }
    if (hstats->n_tq > tqcap) { res.error = "T queue overflow"; return RC_CUDA; }
    if (hstats->n_left && !tbound_forms<NQ, ST>(hs, sp, t, depth).general) {
      res.error = "T bounds left over";
      return RC_CUDA;
    }
    if (hstats->surv_overflow) { res.error = "survivor buffer overflow"; return RC_CUDA; }
    const DevStats h = *hstats;
    if (m * G > 0) surv_rate = (double)h.alive / ((double)m * G);
    res.t_evals += (long long)h.t_evals;
    res.children += (long long)h.children;
    res.children_full += (long long)h.full;
    LevelStats L;
    L.t = t; L.parents = m; L.prefixes = m * G - (long long)h.w2; L.cut_w3 = (long long)h.w3;
    L.cut_lb = (long long)h.dead; L.survivors = (long long)h.alive;
    res.prefixes += L.prefixes;
    if (h.found) {                                     // the lexicographically first circuit of this level
      const unsigned long long o = h.first_found;
      res.circuit = walk_back(o, t);
      res.n_found = (long long)h.found;
      res.levels = t;
      return RC_CIRCUIT;
    }
    long long distinct = 0;
    const size_t ns = keep ? (size_t)h.n_surv : 0;
    if (ns) {
      if (opt.profile > 1) ck(cudaEventRecord(ev[2], s), "event");
      k0.ensure(ns * 8); k1.ensure(ns * 8); v0.ensure(ns * 4); v1.ensure(ns * 4);
      kidx.ensure(ns * 8); kslot.ensure(ns * 4);
      hist.ensure(sort_hist_words(ns) * 4);
      part.ensure(scan_partials_words(sort_hist_words(ns)) * 4);
      SortScratch sc{hist.as<uint32_t>(), part.as<uint32_t>(), hist.cap / 4, part.cap / 4};
      const unsigned gb = (unsigned)std::min<size_t>((ns + 255) / 256, (size_t)nsm * 16);
      if (opt.dedupe && ns > 1) {
        work.ensure(ns * sizeof(uint2)); tmp.ensure(ns * 4);
        k_sort_init<<<gb, 256, 0, s>>>(sH1.as<uint64_t>(), ns, k0.as<uint64_t>(), v0.as<uint32_t>());
        launches++;
        int nl = 0;
        const bool f = radix_sort(k0.as<uint64_t>(), v0.as<uint32_t>(), k1.as<uint64_t>(), v1.as<uint32_t>(), ns, 32,
                                  64, sc, s, &nl);
        launches += nl;
        const uint64_t *sk = f ? k1.as<uint64_t>() : k0.as<uint64_t>();
        const uint32_t *sv = f ? v1.as<uint32_t>() : v0.as<uint32_t>();
        k_runs<<<gb, 256, 0, s>>>(sk, sv, ns, sIdx.as<uint64_t>(), kidx.as<uint64_t>(), kslot.as<uint32_t>(),
                                  work.as<uint2>(), dst);
        k_resolve<NQ, ST><<<(unsigned)nsm * 8, RES_WARPS * 32, 0, s>>>(
            sp, nullptr, nullptr, G, fR.as<Z4<ST>>(), fMeta.as<NodeMeta>(), work.as<uint2>(), sv, sH1.as<uint64_t>(),
            sH2.as<uint64_t>(), sIdx.as<uint64_t>(), sMeta.as<NodeMeta>(), tmp.as<uint32_t>(), kidx.as<uint64_t>(),
            kslot.as<uint32_t>(), dst);
        launches += 2;
        ck(cudaGetLastError(), "dedupe");
        ck(cudaMemcpyAsync(hstats, dst, sizeof(DevStats), cudaMemcpyDeviceToHost, s), "d2h");
        d2h += sizeof(DevStats);
        ck(cudaStreamSynchronize(s), "dedupe");
        distinct = (long long)hstats->n_kept;
      } else {
        k_keep_all<<<gb, 256, 0, s>>>(sIdx.as<uint64_t>(), ns, kidx.as<uint64_t>(), kslot.as<uint32_t>());
        launches++;
        distinct = (long long)ns;
      }
      if (building && distinct) {   // a table level: drop classes the table holds at a lower level
        const void *const *tp = upload_tree(par, gat, t - 1);
        old.ensure((size_t)distinct + 8); keys2.ensure((size_t)distinct * 12 + 16);
        const unsigned gq = (unsigned)std::max<long long>(1, std::min<long long>((distinct + RES_WARPS - 1) / RES_WARPS,
                                                                                 (long long)nsm * 16));
        k_seen_filter<NQ, ST><<<gq, RES_WARPS * 32, 0, s>>>(
            sp, G, fR.as<Z4<ST>>(), fMeta.as<NodeMeta>(), kidx.as<uint64_t>(), kslot.as<uint32_t>(), (size_t)distinct,
            sH1.as<uint64_t>(), sH2.as<uint64_t>(), sMeta.as<NodeMeta>(), building->S1.as<uint64_t>(),
            building->S2.as<uint64_t>(), building->Sidx.as<uint32_t>(), building->Slvl.as<uint32_t>(), building->ns,
            (const uint32_t *const *)tp, (const uint8_t *const *)(tp + t), old.as<uint8_t>());
        ck(cudaMemsetAsync(&dst->n_work, 0, 8, s), "memset");
        uint64_t *ki2 = (uint64_t *)keys2.p;
        uint32_t *ks2 = (uint32_t *)(ki2 + distinct);
        k_drop_old<<<gb, 256, 0, s>>>(kidx.as<uint64_t>(), kslot.as<uint32_t>(), (size_t)distinct, old.as<uint8_t>(),
                                      ki2, ks2, &dst->n_work);
        launches += 2;
        unsigned long long kept_new = 0;
        ck(cudaMemcpyAsync(&kept_new, &dst->n_work, 8, cudaMemcpyDeviceToHost, s), "d2h");
        ck(cudaStreamSynchronize(s), "table filter");
        ck(cudaMemcpyAsync(kidx.p, ki2, kept_new * 8, cudaMemcpyDeviceToDevice, s), "d2d");
        ck(cudaMemcpyAsync(kslot.p, ks2, kept_new * 4, cudaMemcpyDeviceToDevice, s), "d2d");
        distinct = (long long)kept_new;
      }
      // restore lexicographic order: sort kept (index, slot) pairs by index
      int bits = 1;
      while (bits < 64 && ((unsigned long long)m * G) >> bits) bits++;
      const int hi = ((bits + 7) / 8) * 8;
      int nl2 = 0;
      const bool f2 = radix_sort(kidx.as<uint64_t>(), kslot.as<uint32_t>(), k1.as<uint64_t>(), v1.as<uint32_t>(),
                                 (size_t)distinct, 0, hi, sc, s, &nl2);
      launches += nl2;
      const uint64_t *ki = f2 ? k1.as<uint64_t>() : kidx.as<uint64_t>();
      const uint32_t *vi = f2 ? v1.as<uint32_t>() : kslot.as<uint32_t>();
      if ((int)par.size() <= t) { par.resize(t + 1); gat.resize(t + 1); }
      par[t].ensure((size_t)distinct * 4);
      gat[t].ensure((size_t)distinct);
      if (lean_level && t == stop) {               // tree and keys only; the frontier stays the parents'
        k_tree_only<<<gb, 256, 0, s>>>(ki, distinct, G, par[t].as<uint32_t>(), gat[t].as<uint8_t>());
        launches++;
        ck(cudaGetLastError(), "tree");
      } else {
        fR2.ensure((size_t)distinct * E * sizeof(Z4<ST>));
        fMeta2.ensure((size_t)distinct * sizeof(NodeMeta));
        const unsigned gg = (unsigned)std::max<size_t>(1, std::min<size_t>(((size_t)distinct + RES_WARPS - 1) / RES_WARPS,
                                                                           (size_t)nsm * 16));
        k_materialize<NQ, ST><<<gg, RES_WARPS * 32, 0, s>>>(sp, nullptr, nullptr, G, fR.as<Z4<ST>>(),
                                                            fMeta.as<NodeMeta>(), ki, vi, (size_t)distinct,
                                                            sMeta.as<NodeMeta>(), fR2.as<Z4<ST>>(),
                                                            fMeta2.as<NodeMeta>(), par[t].as<uint32_t>(),
                                                            gat[t].as<uint8_t>(), nullptr);
        launches++;
        ck(cudaGetLastError(), "gather");
        std::swap(fR, fR2);
        std::swap(fMeta, fMeta2);
      }
      if ((building || want_keys) && distinct) {   // the frontier's class keys, from its survivor records
        fK1.ensure(distinct * 8 + 8); fK2.ensure(distinct * 8 + 8);
        k_keys_from_slots<<<gb, 256, 0, s>>>(vi, distinct, sH1.as<uint64_t>(), sH2.as<uint64_t>(), fK1.as<uint64_t>(),
                                             fK2.as<uint64_t>());
        launches++;
      }
      if (building && distinct) seen_add(*building, distinct, t);
      // no wait here: the next level's work queues behind the gather on the stream (the host only needs the
      // counts it already has); the dedupe's device time is read at the next wait
      if (opt.profile > 1) { ck(cudaEventRecord(ev[3], s), "event"); ded_pending = true; }
      ck(cudaGetLastError(), "gather");
    }
    L.distinct = distinct;
    L.proved_unsat = distinct == 0;
    L.seconds = now_s() - t0;
    L.dir = building ? 1 : level_dir;
    res.levels = t;
    cb(L);
    if (!distinct) { ck(cudaStreamSynchronize(s), "gather"); read_dedupe(); return RC_PROOF; }
    m = distinct;
    front_m = m;
    if ((int)level_n.size() <= t) level_n.resize(t + 1, 0);
    level_n[t] = distinct;
    t_start = t + 1;
    if (t == stop) { ck(cudaStreamSynchronize(s), "gather"); read_dedupe(); return RC_STOP; }
  }
  ck(cudaStreamSynchronize(s), "gather");
  read_dedupe();
  return RC_PROOF;   // stopped at the last level (not reachable: the last level keeps nothing)
}

// ---------------- distance table (--table K), host ----------------
// device array of the tree's per-level pointers: par[0..upto] then gat[0..upto]
const void *const *Engine::Impl::upload_tree(const std::vector<DBuf> &p, const std::vector<DBuf> &g, int upto) {
  std::vector<const void *> v(2 * (upto + 1), nullptr);
  for (int l = 1; l <= upto && l < (int)p.size(); l++) { v[l] = p[l].p; v[upto + 1 + l] = g[l].p; }
  tptrs.ensure(v.size() * sizeof(void *) + 16);
  ck(cudaMemcpyAsync(tptrs.p, v.data(), v.size() * sizeof(void *), cudaMemcpyHostToDevice, s), "h2d");
  return (const void *const *)tptrs.p;
}

template <int NQ>
int Engine::Impl::table_levels_keys(const DevSpec &sp, long long n) {
  fK1.ensure(n * 8 + 8); fK2.ensure(n * 8 + 8);
  const unsigned g = (unsigned)std::max<long long>(1, std::min<long long>((n + RES_WARPS - 1) / RES_WARPS, (long long)nsm * 16));
  k_node_keys<NQ, int32_t><<<g, RES_WARPS * 32, 0, s>>>(sp, fR.as<Z4<int32_t>>(), fMeta.as<NodeMeta>(), n,
                                                        fK1.as<uint64_t>(), fK2.as<uint64_t>());
  launches++;
  ck(cudaGetLastError(), "node keys");
  return 0;
}

// append level `lvl` (its keys in fK1/fK2, n nodes) to the table's keys, kept sorted by h1 (stable)
void Engine::Impl::seen_add(DistTable &D, long long n, int lvl) {
  const size_t tot = (size_t)(D.ns + n);
  DBuf a1, a2, ai, al;
  a1.ensure(tot * 8); a2.ensure(tot * 8); ai.ensure(tot * 4); al.ensure(tot * 4);
  if (D.ns) {
    ck(cudaMemcpyAsync(a1.p, D.S1.p, D.ns * 8, cudaMemcpyDeviceToDevice, s), "d2d");
    ck(cudaMemcpyAsync(a2.p, D.S2.p, D.ns * 8, cudaMemcpyDeviceToDevice, s), "d2d");
    ck(cudaMemcpyAsync(ai.p, D.Sidx.p, D.ns * 4, cudaMemcpyDeviceToDevice, s), "d2d");
    ck(cudaMemcpyAsync(al.p, D.Slvl.p, D.ns * 4, cudaMemcpyDeviceToDevice, s), "d2d");
  }
  ck(cudaMemcpyAsync(a1.as<uint64_t>() + D.ns, fK1.p, n * 8, cudaMemcpyDeviceToDevice, s), "d2d");
  ck(cudaMemcpyAsync(a2.as<uint64_t>() + D.ns, fK2.p, n * 8, cudaMemcpyDeviceToDevice, s), "d2d");
  {
    const unsigned gi = (unsigned)std::max<long long>(1, std::min<long long>((n + 255) / 256, (long long)nsm * 16));
    k_level_ids<<<gi, 256, 0, s>>>(ai.as<uint32_t>() + D.ns, al.as<uint32_t>() + D.ns, n, (uint32_t)lvl);
    launches++;
  }
  k0.ensure(tot * 8); k1.ensure(tot * 8); v0.ensure(tot * 4); v1.ensure(tot * 4);
  hist.ensure(sort_hist_words(tot) * 4); part.ensure(scan_partials_words(sort_hist_words(tot)) * 4);
  SortScratch sc{hist.as<uint32_t>(), part.as<uint32_t>(), hist.cap / 4, part.cap / 4};
  const unsigned gb = (unsigned)std::max<size_t>(1, std::min<size_t>((tot + 255) / 256, (size_t)nsm * 16));
  k_sort_init<<<gb, 256, 0, s>>>(a1.as<uint64_t>(), tot, k0.as<uint64_t>(), v0.as<uint32_t>());
  const bool f = radix_sort(k0.as<uint64_t>(), v0.as<uint32_t>(), k1.as<uint64_t>(), v1.as<uint32_t>(), tot, 0, 64, sc,
                            s, nullptr);
  launches += 1 + 1 + 8;
  const uint32_t *order = f ? v1.as<uint32_t>() : v0.as<uint32_t>();
  D.S1.ensure(tot * 8); D.S2.ensure(tot * 8); D.Sidx.ensure(tot * 4); D.Slvl.ensure(tot * 4);
  k_keys_gather<<<gb, 256, 0, s>>>(order, tot, a1.as<uint64_t>(), a2.as<uint64_t>(), ai.as<uint32_t>(),
                                   al.as<uint32_t>(), D.S1.as<uint64_t>(), D.S2.as<uint64_t>(), D.Sidx.as<uint32_t>(),
                                   D.Slvl.as<uint32_t>());
  launches++;
  ck(cudaStreamSynchronize(s), "table keys");
  a1.release(); a2.release(); ai.release(); al.release();
  D.ns = (long long)tot;
}

namespace {
uint64_t fnv_bytes(uint64_t h, const void *p, size_t n) {
  const unsigned char *c = (const unsigned char *)p;
  for (size_t i = 0; i < n; i++) { h ^= c[i]; h *= 0x100000001b3ULL; }
  return h;
}
// the cache file name of the reference (cheese.cu:1442-1451): FNV-1a over the candidate names, n, K, the symmetry
// group and the window tables, so either program finds a table the other wrote
std::string dist_table_path(const HostSpec &hs, const SymGroup &grp, int K, const std::string &dir) {
  uint64_t h = 0xcbf29ce484222325ULL;
  for (const auto &nm : hs.names) h = fnv_bytes(h, nm.c_str(), nm.size() + 1);
  h = fnv_bytes(h, &hs.n, sizeof hs.n);
  h = fnv_bytes(h, &K, sizeof K);
  h = fnv_bytes(h, grp.bperm.data(), grp.bperm.size());
  h = fnv_bytes(h, grp.conj.data(), grp.conj.size());
  h = fnv_bytes(h, hs.bad2.data(), hs.bad2.size());
  h = fnv_bytes(h, hs.bad3.data(), hs.bad3.size() * 4);
  char buf[96];
  std::snprintf(buf, sizeof buf, "table-n%d-k%d-%016llx.bin", hs.n, K, (unsigned long long)h);
  return dir.empty() ? std::string() : dir + "/" + buf;
}
constexpr uint32_t DT_MAGIC = 0x54445a43u;   // "CZDT": the file's keys use this build's class hash
constexpr uint32_t DT_KEY_VERSION = 2;   // 2: 32-bit weighted sums per orbit element

// exact check on the host: the circuit's gates, applied to the target (residual times each gate's inverse), give
// the goal (the identity, exponent 0)
bool host_circuit_ok(const HostSpec &hs, const std::vector<int> &c) {
  const int n = hs.n, N = 1 << n;
  std::vector<Zw> S(hs.root.begin(), hs.root.end()), T(N * N);
  int k = hs.rk;
  for (int g : c) {
    const int nq = hs.gnq[g], L = 1 << nq;
    int mask = 0;
    for (int j = 0; j < nq; j++) mask |= 1 << hs.gq[g][j];
    for (int r = 0; r < N; r++)
      for (int col = 0; col < N; col++) {
        const int base = col & ~mask;
        int lc = 0;
        for (int j = 0; j < nq; j++) lc |= ((col >> hs.gq[g][j]) & 1) << j;
        Zw v{0, 0, 0, 0};
        for (int m2 = 0; m2 < L; m2++) {
          int x = base;
          for (int j = 0; j < nq; j++) x |= ((m2 >> j) & 1) << hs.gq[g][j];
          v = zadd(v, zmul(S[r * N + x], hs.ginv[g][m2 * L + lc]));
        }
        T[r * N + col] = v;
      }
    S.swap(T);
    k += hs.gik[g];
    while (k > 0) {
      bool ok = true;
      for (const Zw &z : S) ok = ok && zdiv2ok(z);
      if (!ok) break;
      for (Zw &z : S) z = zdown(z);
      k--;
    }
  }
  if (k != 0) return false;
  for (int r = 0; r < N; r++)
    for (int col = 0; col < N; col++) {
      const Zw z = S[r * N + col];
      if (r == col ? !(z.a == 1 && !z.b && !z.c && !z.d) : !zzero(z)) return false;
    }
  return true;
}
}  // namespace

bool Engine::Impl::table_load(const std::string &path, DistTable &D, int K, int G) {
  FILE *f = path.empty() ? nullptr : std::fopen(path.c_str(), "rb");
  if (!f) return false;
  std::fseek(f, 0, SEEK_END);
  const long size = std::ftell(f);
  std::fseek(f, 0, SEEK_SET);
  int nl = 0;
  bool ok = std::fread(&nl, sizeof nl, 1, f) == 1 && nl >= 0 && nl <= K;
  std::vector<std::vector<uint32_t>> P;
  std::vector<std::vector<uint8_t>> Gt;
  for (int l = 1; ok && l <= nl; l++) {
    long n = 0;
    ok = std::fread(&n, sizeof n, 1, f) == 1 && n > 0 && n <= size;
    if (!ok) break;
    P.emplace_back(n); Gt.emplace_back(n);
    ok = std::fread(P.back().data(), 4, n, f) == (size_t)n && std::fread(Gt.back().data(), 1, n, f) == (size_t)n;
  }
  long ns = 0;
  std::vector<KeyRec> keys;
  bool trusted = false;
  if (ok && std::fread(&ns, sizeof ns, 1, f) == 1 && ns > 0 && ns <= size) {
    // the keys are read only when the file ends with this library's trailer (the same class hash)
    uint32_t trailer[2] = {0, 0};
    const long pos = std::ftell(f);
    trusted = pos >= 0 && std::fseek(f, pos + ns * (long)sizeof(KeyRec), SEEK_SET) == 0 &&
              std::fread(trailer, 4, 2, f) == 2 && trailer[0] == DT_MAGIC && trailer[1] == DT_KEY_VERSION;
    if (trusted) {
      keys.resize(ns);
      trusted = std::fseek(f, pos, SEEK_SET) == 0 && std::fread(keys.data(), sizeof(KeyRec), ns, f) == (size_t)ns;
    }
  } else {
    ok = false;
  }
  std::fclose(f);
  // every parent index and candidate in range (a damaged file is rebuilt, never replayed out of bounds), and every
  // trusted key record names a node of the tree
  for (int l = 1; ok && l <= nl; l++) {
    const size_t below = l == 1 ? 1 : P[l - 2].size();
    for (size_t j = 0; ok && j < P[l - 1].size(); j++) ok = P[l - 1][j] < below && (int)Gt[l - 1][j] < G;
  }
  if (!ok) return false;
  for (size_t i = 0; trusted && i < keys.size(); i++)
    trusted = keys[i].lvl == 0 ? keys[i].idx == 0 : (keys[i].lvl <= (uint32_t)nl && keys[i].idx < P[keys[i].lvl - 1].size());
  D.K = K; D.nl = nl;
  D.par.assign(nl + 1, DBuf{}); D.gat.assign(nl + 1, DBuf{}); D.n.assign(nl + 1, 0);
  D.n[0] = 1;
  for (int l = 1; l <= nl; l++) {
    const long long n = (long long)P[l - 1].size();
    D.n[l] = n;
    D.par[l].ensure(n * 4 + 4); D.gat[l].ensure(n + 4);
    ck(cudaMemcpyAsync(D.par[l].p, P[l - 1].data(), n * 4, cudaMemcpyHostToDevice, s), "h2d");
    ck(cudaMemcpyAsync(D.gat[l].p, Gt[l - 1].data(), n, cudaMemcpyHostToDevice, s), "h2d");
  }
  if (trusted) {
    D.S1.ensure(ns * 8); D.S2.ensure(ns * 8); D.Sidx.ensure(ns * 4); D.Slvl.ensure(ns * 4);
    tmp.ensure(ns * sizeof(KeyRec));
    ck(cudaMemcpyAsync(tmp.p, keys.data(), ns * sizeof(KeyRec), cudaMemcpyHostToDevice, s), "h2d");
    const unsigned gb = (unsigned)std::max<long>(1, std::min<long>((ns + 255) / 256, (long)nsm * 16));
    k_keys_unpack<<<gb, 256, 0, s>>>(tmp.as<KeyRec>(), ns, D.S1.as<uint64_t>(), D.S2.as<uint64_t>(),
                                     D.Sidx.as<uint32_t>(), D.Slvl.as<uint32_t>());
    launches++;
    D.ns = ns;
  }
  ck(cudaStreamSynchronize(s), "table load");
  return true;   // untrusted keys: the caller recomputes them (D.ns == 0)
}

void Engine::Impl::table_save(const std::string &path, const DistTable &D) {
  if (path.empty()) return;
  FILE *f = std::fopen(path.c_str(), "wb");
  if (!f) { std::fprintf(stderr, "cannot write %s (table not cached)\n", path.c_str()); return; }
  const int nl = D.nl;
  std::fwrite(&nl, sizeof nl, 1, f);
  for (int l = 1; l <= nl; l++) {
    const long n = (long)D.n[l];
    std::vector<uint32_t> P(n);
    std::vector<uint8_t> G(n);
    cudaMemcpy(P.data(), D.par[l].p, n * 4, cudaMemcpyDeviceToHost);
    cudaMemcpy(G.data(), D.gat[l].p, n, cudaMemcpyDeviceToHost);
    std::fwrite(&n, sizeof n, 1, f); std::fwrite(P.data(), 4, n, f); std::fwrite(G.data(), 1, n, f);
  }
  const long ns = (long)D.ns;
  std::vector<KeyRec> keys(ns);     // the reference's key record layout; the keys are this library's class hash
  {
    DBuf rec;
    rec.ensure(ns * sizeof(KeyRec) + 16);
    const unsigned gb = (unsigned)std::max<long>(1, std::min<long>((ns + 255) / 256, (long)nsm * 16));
    k_keys_pack<<<gb, 256, 0, s>>>(D.S1.as<uint64_t>(), D.S2.as<uint64_t>(), D.Sidx.as<uint32_t>(),
                                   D.Slvl.as<uint32_t>(), ns, rec.as<KeyRec>());
    ck(cudaMemcpyAsync(keys.data(), rec.p, ns * sizeof(KeyRec), cudaMemcpyDeviceToHost, s), "d2h");
    ck(cudaStreamSynchronize(s), "table keys");
    rec.release();
  }
  std::fwrite(&ns, sizeof ns, 1, f);
  std::fwrite(keys.data(), sizeof(KeyRec), ns, f);
  const uint32_t trailer[2] = {DT_MAGIC, DT_KEY_VERSION};   // past the reference's layout: its reader stops before
  std::fwrite(trailer, 4, 2, f);
  std::fclose(f);
}

// the table of (spec tables, symmetry group, K): resident, else the cache file, else built from the identity by the
// level search without bounds, each level filtered against the classes of the lower ones (cheese.cu:1495-1517)
template <int NQ>
Engine::Impl::DistTable *Engine::Impl::get_table(const HostSpec &hs, const SymGroup &grp, int K, const Options &opt,
                                                 const std::function<void(const LevelStats &)> &cb,
                                                 SearchResult &res) {
  constexpr int N = 1 << NQ, E = N * N;
  const std::string path = dist_table_path(hs, grp, K, opt.cache_dir);
  const std::string key = path.empty() ? dist_table_path(hs, grp, K, ".") : path;
  res.table_path = path;
  auto it = dtabs.find(key);
  if (it != dtabs.end()) return it->second;
  const double t0 = now_s();
  HostSpec hI = hs;                                   // the identity as target, no bounds, never "found"
  hI.target.assign(E, Zw{0, 0, 0, 0});
  for (int i = 0; i < N; i++) hI.target[i * N + i] = Zw{1, 0, 0, 0};
  hI.root = hI.target;
  hI.tk = hI.rk = 0; hI.standard = 0; hI.lite = 0; hI.uid = hs.uid ^ 0x7461626c65ULL;
  const DevSpec sp = prepare<NQ>(hI, grp, K + 1, true);
  DistTable *D = new DistTable;
  if (table_load(path, *D, K, hs.G)) {
    res.table_loaded = true;
    if (!D->ns) {                                     // another program's keys: recompute them with this build's hash
      fK1.ensure(16); fK2.ensure(16);
      fR.ensure(E * sizeof(Z4<int32_t>)); fMeta.ensure(sizeof(NodeMeta));
      std::vector<Z4<int32_t>> id(E, Z4<int32_t>{0, 0, 0, 0});
      for (int i = 0; i < N; i++) id[i * N + i] = Z4<int32_t>{1, 0, 0, 0};
      ck(cudaMemcpyAsync(fR.p, id.data(), E * sizeof(Z4<int32_t>), cudaMemcpyHostToDevice, s), "h2d");
      k_root<NQ, int32_t><<<1, 32, 0, s>>>(sp, fR.as<Z4<int32_t>>(), fMeta.as<NodeMeta>(), 0);
      table_levels_keys<NQ>(sp, 1);
      seen_add(*D, 1, 0);
      for (int l = 1; l <= D->nl; l++) {
        const void *const *tp = upload_tree(D->par, D->gat, l);
        const long long n = D->n[l];
        fK1.ensure(n * 8 + 8); fK2.ensure(n * 8 + 8);
        const unsigned g = (unsigned)std::max<long long>(1, std::min<long long>((n + RES_WARPS - 1) / RES_WARPS, (long long)nsm * 16));
        k_replay_keys<NQ, int32_t><<<g, RES_WARPS * 32, 0, s>>>(sp, l, n, (const uint32_t *const *)tp,
                                                                (const uint8_t *const *)(tp + l + 1),
                                                                fK1.as<uint64_t>(), fK2.as<uint64_t>());
        launches++;
        ck(cudaGetLastError(), "table keys");
        seen_add(*D, n, l);
      }
    }
  } else {
    D->release();
    *D = DistTable{};
    D->K = K;
    fR.ensure(E * sizeof(Z4<int32_t>)); fMeta.ensure(sizeof(NodeMeta));
    std::vector<Z4<int32_t>> id(E, Z4<int32_t>{0, 0, 0, 0});
    for (int i = 0; i < N; i++) id[i * N + i] = Z4<int32_t>{1, 0, 0, 0};
    ck(cudaMemcpyAsync(fR.p, id.data(), E * sizeof(Z4<int32_t>), cudaMemcpyHostToDevice, s), "h2d");
    k_root<NQ, int32_t><<<1, 32, 0, s>>>(sp, fR.as<Z4<int32_t>>(), fMeta.as<NodeMeta>(), 0);
    launches++;
    table_levels_keys<NQ>(sp, 1);
    seen_add(*D, 1, 0);
    front_m = 1;
    level_n.assign(1, 1);
    building = D;
    Options o = opt;
    o.dedupe = true;
    o.nogoal = true;
    int t = 1;
    const int rc = levels<NQ, int32_t>(hI, sp, o, K + 1, t, cb, res, K);
    building = nullptr;
    if (rc == -2) { delete D; throw std::overflow_error("coefficient overflow (int32) in the distance table"); }
    D->nl = t - 1;                                    // levels that added classes
    D->par.assign(D->nl + 1, DBuf{}); D->gat.assign(D->nl + 1, DBuf{}); D->n.assign(D->nl + 1, 1);
    for (int l = 1; l <= D->nl; l++) {                // the tree levels move into the table
      std::swap(D->par[l], par[l]);
      std::swap(D->gat[l], gat[l]);
      D->n[l] = level_n[l];
    }
    res.table_built = true;
    table_save(path, *D);
  }
  res.table_seconds = now_s() - t0;
  dtabs[key] = D;
  return D;
}

// the search with a distance table (cheese.cu:1804-1838): levels 1 .. D - K, and after each level (and for the
// target itself) every node whose class is in the table within the remaining budget is a circuit candidate,
// confirmed exactly; past level D - K every residual outside the table needs more than K gates
template <int NQ>
int Engine::Impl::run_table(const HostSpec &hs, const Options &opt, const std::function<void(const LevelStats &)> &cb,
                            SearchResult &res) {
  constexpr int N = 1 << NQ, E = N * N;
  const int depth = opt.depth >= 0 ? opt.depth : hs.depth;
  const int K = opt.table_k;
  const SymGroup grp = sym_group(hs, opt.sym);
  res.nsym = grp.nsym;
  res.table_k = K;
  {
    bool done = hs.tk == 0;
    for (int r = 0; r < N && done; r++)
      for (int c = 0; c < N && done; c++) {
        const Zw x = hs.target[r * N + c];
        done = r == c ? (x.a == 1 && !x.b && !x.c && !x.d) : zzero(x);
      }
    if (done) { res.depth0 = true; return RC_CIRCUIT; }
  }
  for (const Zw &z : hs.target)
    if (!fits32(z.a) || !fits32(z.b) || !fits32(z.c) || !fits32(z.d)) {
      res.error = "target coefficients exceed int32";
      return RC_OVERFLOW;
    }
  DistTable *D;
  try {
    D = get_table<NQ>(hs, grp, K, opt, cb, res);
  } catch (const std::overflow_error &e) {
    res.error = e.what();
    return RC_OVERFLOW;
  }
  res.table_classes = D->ns;
  res.table_levels = D->nl;
  const DevSpec sp = prepare<NQ>(hs, grp, depth, false);
  {
    std::vector<Z4<int32_t>> t32(E);
    for (int i = 0; i < E; i++) t32[i] = {(int32_t)hs.root[i].a, (int32_t)hs.root[i].b, (int32_t)hs.root[i].c, (int32_t)hs.root[i].d};
    fR.ensure(E * sizeof(Z4<int32_t>)); fMeta.ensure(sizeof(NodeMeta));
    ck(cudaMemcpyAsync(fR.p, t32.data(), E * sizeof(Z4<int32_t>), cudaMemcpyHostToDevice, s), "h2d");
    k_root<NQ, int32_t><<<1, 32, 0, s>>>(sp, fR.as<Z4<int32_t>>(), fMeta.as<NodeMeta>(), hs.rk);
    launches++;
    table_levels_keys<NQ>(sp, 1);
    ck(cudaStreamSynchronize(s), "root");
  }
  front_m = 1;
  level_n.assign(1, 1);
  const std::vector<int> inv = inverse_gates(hs);
  want_keys = true;
  int t_next = 1;
  for (int t = 0; t <= depth - K || t == 0; t++) {
    bool lean = false;
    if (t > 0) {
      lean_level = t == depth - K;      // the last level searched: its residuals are rebuilt only for candidates
      const int rc = levels<NQ, int32_t>(hs, sp, opt, depth, t_next, cb, res, t);
      lean = lean_level;
      lean_level = false;
      if (rc == -2) { want_keys = false; res.error = "coefficient overflow (int32) in table mode"; return RC_OVERFLOW; }
      if (rc != RC_STOP) { want_keys = false; return rc; }
    }
    // candidates: nodes of level t whose class is in the table within depth - t gates, cheapest first
    const long long n = front_m;
    const int maxc = depth - t;
    const unsigned long long hcap = 1 << 16;
    tmp.ensure(hcap * sizeof(longlong2) + 16);
    unsigned long long *nh_d = (unsigned long long *)(tmp.as<longlong2>() + hcap);
    ck(cudaMemsetAsync(nh_d, 0, 8, s), "memset");
    k_table_lookup<<<(unsigned)std::max<long long>(1, std::min<long long>((n + 255) / 256, (long long)nsm * 16)), 256, 0, s>>>(
        fK1.as<uint64_t>(), fK2.as<uint64_t>(), n, D->S1.as<uint64_t>(), D->S2.as<uint64_t>(), D->Slvl.as<uint32_t>(),
        D->ns, maxc, tmp.as<longlong2>(), hcap, nh_d);
    launches++;
    unsigned long long nh = 0;
    ck(cudaMemcpyAsync(&nh, nh_d, 8, cudaMemcpyDeviceToHost, s), "d2h");
    ck(cudaStreamSynchronize(s), "table lookup");
    if (nh > hcap) { want_keys = false; res.error = "table lookup: more than 65536 candidates"; return RC_CUDA; }
    std::vector<longlong2> hl(nh);
    if (nh) ck(cudaMemcpy(hl.data(), tmp.p, nh * sizeof(longlong2), cudaMemcpyDeviceToHost), "d2h");
    std::vector<std::pair<std::pair<int, long long>, long long>> cand;   // ((table level, node), table entry)
    for (const longlong2 &h : hl) {
      uint32_t lv = 0;
      ck(cudaMemcpy(&lv, D->Slvl.as<uint32_t>() + h.y, 4, cudaMemcpyDeviceToHost), "d2h");
      cand.push_back({{(int)lv, h.x}, h.y});
    }
    std::sort(cand.begin(), cand.end());
    const void *const *tp = upload_tree(D->par, D->gat, D->nl);
    outb.ensure(64 * sizeof(int2) + 16 + E * sizeof(Z4<int32_t>) + 16);
    Z4<int32_t> *cres = (Z4<int32_t> *)((char *)outb.p + 64 * sizeof(int2) + 16);
    for (const auto &cd : cand) {
      const long long j = cd.first.second, hitj = cd.second;
      int kj = 0;
      const Z4<int32_t> *Sj = fR.as<Z4<int32_t>>() + j * E;
      if (lean) {                       // rebuild the node from its parent
        uint32_t pp = 0;
        uint8_t gg = 0;
        ck(cudaMemcpy(&pp, par[t].as<uint32_t>() + j, 4, cudaMemcpyDeviceToHost), "d2h");
        ck(cudaMemcpy(&gg, gat[t].as<uint8_t>() + j, 1, cudaMemcpyDeviceToHost), "d2h");
        k_child_residual<NQ, int32_t><<<1, 32, 0, s>>>(sp, fR.as<Z4<int32_t>>(), fMeta.as<NodeMeta>(),
                                                       (unsigned long long)pp * hs.G + gg, hs.G, cres,
                                                       (int *)(outb.as<int2>() + 64) + 1);
        launches++;
        ck(cudaMemcpyAsync(&kj, (int *)(outb.as<int2>() + 64) + 1, 4, cudaMemcpyDeviceToHost, s), "d2h");
        ck(cudaStreamSynchronize(s), "candidate");
        Sj = cres;
      } else {
        NodeMeta mj;
        ck(cudaMemcpy(&mj, fMeta.as<NodeMeta>() + j, sizeof mj, cudaMemcpyDeviceToHost), "d2h");
        kj = mj.k;
      }
      k_table_confirm<NQ, int32_t><<<1, 32, 0, s>>>(sp, Sj, kj, D->S1.as<uint64_t>(),
                                                    D->S2.as<uint64_t>(), D->Sidx.as<uint32_t>(), D->Slvl.as<uint32_t>(),
                                                    D->ns, hitj, maxc, (const uint32_t *const *)tp,
                                                    (const uint8_t *const *)(tp + D->nl + 1), outb.as<int2>(), 64,
                                                    (int *)(outb.as<int2>() + 64));
      launches++;
      int nout = 0;
      std::vector<int2> pairs(64);
      ck(cudaMemcpyAsync(&nout, outb.as<int2>() + 64, 4, cudaMemcpyDeviceToHost, s), "d2h");
      ck(cudaMemcpyAsync(pairs.data(), outb.p, 64 * sizeof(int2), cudaMemcpyDeviceToHost, s), "d2h");
      ck(cudaStreamSynchronize(s), "table confirm");
      if (!nout) continue;
      std::vector<int> pre(t);                        // the node's prefix
      {
        uint32_t i = (uint32_t)j;
        for (int l = t; l >= 1; l--) {
          uint8_t gg; uint32_t pp;
          ck(cudaMemcpy(&gg, gat[l].as<uint8_t>() + i, 1, cudaMemcpyDeviceToHost), "d2h");
          ck(cudaMemcpy(&pp, par[l].as<uint32_t>() + i, 4, cudaMemcpyDeviceToHost), "d2h");
          pre[l - 1] = gg; i = pp;
        }
      }
      for (int q = 0; q < nout; q++) {
        const int x = pairs[q].x, sy = pairs[q].y;
        uint32_t lv = 0, ix = 0;
        ck(cudaMemcpy(&lv, D->Slvl.as<uint32_t>() + x, 4, cudaMemcpyDeviceToHost), "d2h");
        ck(cudaMemcpy(&ix, D->Sidx.as<uint32_t>() + x, 4, cudaMemcpyDeviceToHost), "d2h");
        std::vector<int> w(lv);                       // the table sequence, from the identity
        uint32_t i = ix;
        for (int l = (int)lv; l >= 1; l--) {
          uint8_t gg; uint32_t pp;
          ck(cudaMemcpy(&gg, D->gat[l].as<uint8_t>() + i, 1, cudaMemcpyDeviceToHost), "d2h");
          ck(cudaMemcpy(&pp, D->par[l].as<uint32_t>() + i, 4, cudaMemcpyDeviceToHost), "d2h");
          w[l - 1] = gg; i = pp;
        }
        std::vector<int> full = pre;                  // the suffix: w reversed, inverted, relabelled by the symmetry
        bool okmap = true;
        for (int a = (int)w.size() - 1; a >= 0; a--) {
          const int gi = inv[w[a]];
          if (gi < 0) { okmap = false; break; }
          full.push_back(grp.gmap[sy][gi]);
        }
        if (okmap && host_circuit_ok(hs, full)) {
          want_keys = false;
          res.circuit = full;
          res.n_found = 1;
          res.table_split[0] = t;
          res.table_split[1] = (int)full.size() - t;
          return RC_CIRCUIT;
        }
      }
    }
  }
  want_keys = false;
  res.table_proof = true;
  return RC_PROOF;
}

// the meet-in-the-middle search (cheese.cu:1595-1760): the search on U (forward) and on U^dag (backward) grow one
// level at a time, the side with the smaller frontier first, until their depths add up to D; a circuit found by a
// side's own levels ends the search (a backward one is reversed and inverted). Then every backward node q
// (levels 1..b) is joined with the forward frontier at level a: K = U R'_q equals a forward residual exactly iff the
// forward prefix followed by q^-1 is a circuit. No match is a proof. Symmetry classes are off (exact residuals).
template <int NQ>
int Engine::Impl::run_mitm(const HostSpec &hs, const Options &opt, const std::function<void(const LevelStats &)> &cb,
                           SearchResult &res) {
  constexpr int N = 1 << NQ, E = N * N;
  const int depth = opt.depth >= 0 ? opt.depth : hs.depth;
  const SymGroup grp = sym_group(hs, false);
  res.nsym = grp.nsym;
  {
    bool done = hs.tk == 0;
    for (int r = 0; r < N && done; r++)
      for (int c = 0; c < N && done; c++) {
        const Zw x = hs.target[r * N + c];
        done = r == c ? (x.a == 1 && !x.b && !x.c && !x.d) : zzero(x);
      }
    if (done) { res.depth0 = true; return RC_CIRCUIT; }
  }
  const std::vector<int> inv = inverse_gates(hs);
  for (int g = 0; g < hs.G; g++)
    if (inv[g] < 0) { res.error = "--mitm: no inverse candidate for " + hs.names[g]; return RC_USAGE; }
  for (const Zw &z : hs.target)
    if (!fits32(z.a) || !fits32(z.b) || !fits32(z.c) || !fits32(z.d)) {
      res.error = "--mitm: target coefficients exceed int32";
      return RC_OVERFLOW;
    }
  const DevSpec sp = prepare<NQ>(hs, grp, depth, false);
  std::vector<Z4<int32_t>> hU(E), hUd(E);
  for (int r = 0; r < N; r++)
    for (int c = 0; c < N; c++) {
      const Zw x = hs.root[r * N + c];
      hU[r * N + c] = {(int32_t)x.a, (int32_t)x.b, (int32_t)x.c, (int32_t)x.d};
      const Zw t = hs.root[c * N + r];                  // U^dag (conjugate transpose), same sqrt2 exponent
      const Zw y{t.a, -t.d, -t.c, -t.b};
      hUd[r * N + c] = {(int32_t)y.a, (int32_t)y.b, (int32_t)y.c, (int32_t)y.d};
    }
  DBuf dU;
  dU.ensure(2 * E * sizeof(Z4<int32_t>));
  ck(cudaMemcpyAsync(dU.p, hU.data(), E * sizeof(Z4<int32_t>), cudaMemcpyHostToDevice, s), "h2d");
  ck(cudaMemcpyAsync(dU.as<Z4<int32_t>>() + E, hUd.data(), E * sizeof(Z4<int32_t>), cudaMemcpyHostToDevice, s), "h2d");
  h2d += 2 * E * sizeof(Z4<int32_t>);
  const Z4<int32_t> *U = dU.as<Z4<int32_t>>(), *Ud = U + E;
  auto root = [&](const Z4<int32_t> *M) {              // the current tree restarts at M
    fR.ensure(E * sizeof(Z4<int32_t>)); fMeta.ensure(sizeof(NodeMeta));
    ck(cudaMemcpyAsync(fR.p, M, E * sizeof(Z4<int32_t>), cudaMemcpyDeviceToDevice, s), "d2d");
    k_root<NQ, int32_t><<<1, 32, 0, s>>>(sp, fR.as<Z4<int32_t>>(), fMeta.as<NodeMeta>(), hs.rk);
    launches++;
    ck(cudaGetLastError(), "root kernel");
    front_m = 1;
    level_n.assign(1, 1);
  };
  root(U);
  swap_side();
  root(Ud);
  swap_side();
  ck(cudaStreamSynchronize(s), "roots");
  int a = 0, b = 0;
  long long nF = 1, nB = 1;
  bool bdead = false;
  auto done = [&]() { level_dir = 0; dU.release(); };
  while (a + b < depth) {
    const bool fwd = bdead || nF <= nB;
    if (!fwd) swap_side();
    level_dir = fwd ? 2 : 3;
    int t = (fwd ? a : b) + 1;
    const int stop = t;
    res.circuit.clear();
    res.n_found = 0;
    const int rc = levels<NQ, int32_t>(hs, sp, opt, depth, t, cb, res, stop);
    if (fwd) { a = t - 1; nF = front_m; } else { b = t - 1; nB = front_m; }
    if (!fwd) swap_side();
    if (rc == RC_CIRCUIT) {
      if (!fwd) {                                       // a circuit q for U^dag: U = q^-1
        std::vector<int> c;
        for (int i = (int)res.circuit.size() - 1; i >= 0; i--) c.push_back(inv[res.circuit[i]]);
        res.circuit = c;
      }
      done();
      return RC_CIRCUIT;
    }
    if (rc == -2) { done(); res.error = "--mitm: coefficients exceed int32"; return RC_OVERFLOW; }
    if (rc == RC_PROOF) {
      if (fwd) { done(); return RC_PROOF; }
      bdead = true;                                     // no suffix is longer than b: the join below is complete
      break;
    }
    if (rc != RC_STOP) { done(); return rc; }
  }
  level_dir = 0;
  res.mitm_split[0] = a;
  res.mitm_split[1] = b;
  const long long nf = level_n.size() > (size_t)a ? level_n[a] : 0;
  MitmLevels lv;
  std::memset(&lv, 0, sizeof lv);
  lv.top = b;
  long long nb = 0;
  for (int l = 1; l <= b; l++) { lv.off[l] = nb; nb += side.level_n[l]; }
  lv.off[b + 1] = nb;
  if (!nb || !nf) { res.mitm_proof = true; done(); return RC_PROOF; }
  const double tj = now_s();
  // forward keys, sorted by h1 (stable), with their frontier index
  table_levels_keys<NQ>(sp, nf);
  DBuf S1, S2, Si, B1, B2, pos, hits, flags;
  k0.ensure(nf * 8); k1.ensure(nf * 8); v0.ensure(nf * 4); v1.ensure(nf * 4);
  hist.ensure(sort_hist_words(nf) * 4); part.ensure(scan_partials_words(sort_hist_words(nf)) * 4);
  SortScratch sc{hist.as<uint32_t>(), part.as<uint32_t>(), hist.cap / 4, part.cap / 4};
  const unsigned gf = (unsigned)std::max<long long>(1, std::min<long long>((nf + 255) / 256, (long long)nsm * 16));
  k_sort_init<<<gf, 256, 0, s>>>(fK1.as<uint64_t>(), nf, k0.as<uint64_t>(), v0.as<uint32_t>());
  const bool fl = radix_sort(k0.as<uint64_t>(), v0.as<uint32_t>(), k1.as<uint64_t>(), v1.as<uint32_t>(), nf, 0, 64, sc,
                             s, nullptr);
  launches += 1 + 1 + 8;
  S1.ensure(nf * 8); S2.ensure(nf * 8); Si.ensure(nf * 4);
  k_mitm_sorted<<<gf, 256, 0, s>>>(fl ? v1.as<uint32_t>() : v0.as<uint32_t>(), nf, fK1.as<uint64_t>(),
                                   fK2.as<uint64_t>(), S1.as<uint64_t>(), S2.as<uint64_t>(), Si.as<uint32_t>());
  launches++;
  // backward keys: every backward node rebuilt from U^dag, multiplied by U, hashed
  const void *const *tp = upload_tree(side.par, side.gat, b);
  B1.ensure(nb * 8); B2.ensure(nb * 8); flags.ensure(16);
  ck(cudaMemsetAsync(flags.p, 0, 16, s), "memset");
  const unsigned gw = (unsigned)std::max<long long>(1, std::min<long long>((nb + RES_WARPS - 1) / RES_WARPS, (long long)nsm * 16));
  k_mitm_bwd_keys<NQ><<<gw, RES_WARPS * 32, 0, s>>>(sp, U, Ud, hs.rk, lv, (const uint32_t *const *)tp,
                                                    (const uint8_t *const *)(tp + b + 1), nb, B1.as<uint64_t>(),
                                                    B2.as<uint64_t>(), flags.as<int>());
  launches++;
  ck(cudaGetLastError(), "mitm keys");
  pos.ensure(nb * 8); hits.ensure(nb * 8);
  unsigned long long *nh_d = (unsigned long long *)(flags.as<int>() + 2);
  const unsigned gb = (unsigned)std::max<long long>(1, std::min<long long>((nb + 255) / 256, (long long)nsm * 16));
  k_mitm_match<<<gb, 256, 0, s>>>(B1.as<uint64_t>(), B2.as<uint64_t>(), nb, S1.as<uint64_t>(), S2.as<uint64_t>(), nf,
                                  pos.as<long long>(), hits.as<long long>(), nh_d);
  launches++;
  int hflags[4] = {0, 0, 0, 0};
  ck(cudaMemcpyAsync(hflags, flags.p, 16, cudaMemcpyDeviceToHost, s), "d2h");
  ck(cudaStreamSynchronize(s), "mitm join");
  d2h += 16;
  if (hflags[0]) {
    S1.release(); S2.release(); Si.release(); B1.release(); B2.release(); pos.release(); hits.release(); flags.release();
    done();
    res.error = "--mitm: coefficients exceed int32";
    return RC_OVERFLOW;
  }
  unsigned long long nh = 0;
  std::memcpy(&nh, hflags + 2, 8);
  res.mitm_join = true;
  res.mitm_forward = nf;
  res.mitm_backward = nb;
  res.mitm_hash_matches = (long long)nh;
  res.mitm_seconds = now_s() - tj;
  int rc = RC_PROOF;
  if (nh) {                                             // exact confirmation, candidates in backward order
    std::vector<long long> cand(nh), match(nh);
    ck(cudaMemcpyAsync(cand.data(), hits.p, nh * 8, cudaMemcpyDeviceToHost, s), "d2h");
    ck(cudaStreamSynchronize(s), "d2h");
    std::sort(cand.begin(), cand.end());
    ck(cudaMemcpyAsync(hits.p, cand.data(), nh * 8, cudaMemcpyHostToDevice, s), "h2d");
    DBuf mb;
    mb.ensure(nh * 8);
    const unsigned gc = (unsigned)std::max<unsigned long long>(1, std::min<unsigned long long>((nh + RES_WARPS - 1) / RES_WARPS, (unsigned long long)nsm * 16));
    k_mitm_confirm<NQ><<<gc, RES_WARPS * 32, 0, s>>>(sp, U, Ud, hs.rk, lv, (const uint32_t *const *)tp,
                                                     (const uint8_t *const *)(tp + b + 1), hits.as<long long>(),
                                                     (long long)nh, pos.as<long long>(), S1.as<uint64_t>(),
                                                     S2.as<uint64_t>(), Si.as<uint32_t>(), nf, fR.as<Z4<int32_t>>(),
                                                     fMeta.as<NodeMeta>(), mb.as<long long>());
    launches++;
    ck(cudaGetLastError(), "mitm confirm");
    ck(cudaMemcpyAsync(match.data(), mb.p, nh * 8, cudaMemcpyDeviceToHost, s), "d2h");
    ck(cudaStreamSynchronize(s), "mitm confirm");
    mb.release();
    auto path = [&](const std::vector<DBuf> &P, const std::vector<DBuf> &G, int l, uint32_t i) {
      std::vector<int> q(l);
      for (; l >= 1; l--) {
        uint8_t gg; uint32_t pp;
        ck(cudaMemcpy(&gg, G[l].as<uint8_t>() + i, 1, cudaMemcpyDeviceToHost), "d2h");
        ck(cudaMemcpy(&pp, P[l].as<uint32_t>() + i, 4, cudaMemcpyDeviceToHost), "d2h");
        q[l - 1] = gg; i = pp;
      }
      return q;
    };
    for (unsigned long long c = 0; c < nh && rc == RC_PROOF; c++) {
      if (match[c] < 0) continue;
      const long long j = cand[c];
      int l = 1;
      while (l < b && j >= lv.off[l + 1]) l++;
      const std::vector<int> q = path(side.par, side.gat, l, (uint32_t)(j - lv.off[l]));
      std::vector<int> full = path(par, gat, a, (uint32_t)match[c]);
      for (int i = (int)q.size() - 1; i >= 0; i--) full.push_back(inv[q[i]]);
      if (!host_circuit_ok(hs, full)) continue;
      res.circuit = full;
      res.n_found = 1;
      res.mitm_found = true;
      res.mitm_split[1] = (int)q.size();
      rc = RC_CIRCUIT;
    }
  }
  if (rc == RC_PROOF) res.mitm_proof = true;
  S1.release(); S2.release(); Si.release(); B1.release(); B2.release(); pos.release(); hits.release(); flags.release();
  done();
  return rc;
}

// M M^dag = 2^k I exactly (an N x N matrix of Z[w] entries over sqrt2^k); large coefficients count as not unitary
bool unitary(const Zw *M, int N, int k) {
  if (k < 0 || k > 40) return false;
  constexpr int64_t LIM = (int64_t)1 << 20;
  for (int e = 0; e < N * N; e++)
    for (int64_t v : {M[e].a, M[e].b, M[e].c, M[e].d})
      if (v > LIM || v < -LIM) return false;
  for (int r = 0; r < N; r++)
    for (int r2 = 0; r2 < N; r2++) {
      Zw s{0, 0, 0, 0};
      for (int c = 0; c < N; c++) s = zadd(s, zmul(M[r * N + c], zconj(M[r2 * N + c])));
      if (!zeq(s, Zw{r == r2 ? (int64_t)1 << k : 0, 0, 0, 0})) return false;
    }
  return true;
}

// host part of the device spec: every field, plus the gate-matrix (gi) and goal (gl) tables to place on the device
template <int NQ>
DevSpec devspec_host(const HostSpec &hs, const SymGroup &grp, int depth, bool nogoal, std::vector<int4> &gi,
                     std::vector<longlong2> &gl) {
  constexpr int N = 1 << NQ, E = N * N;
  DevSpec sp;
  std::memset(&sp, 0, sizeof sp);
  sp.n = hs.n; sp.G = hs.G; sp.depth = depth; sp.standard = hs.standard; sp.lite = hs.lite;
  sp.tdiv = hs.tdiv < 1 ? 1 : hs.tdiv; sp.ncuts = (int)hs.cutmask.size(); sp.have_table = !hs.cxtable.empty();
  sp.ncx = (int)hs.cxtable.size();
  sp.nsym = grp.nsym; sp.nogoal = nogoal; sp.gk = 0;
  for (int i = 0; i < sp.ncuts; i++) { sp.cutmask[i] = hs.cutmask[i]; sp.cutsize[i] = hs.cutsize[i]; sp.rad[i] = hs.rad[i]; }
  sp.w1 = powmod_h(3, (PRIME - 1) / 8); sp.w2 = sp.w1 * sp.w1 % PRIME; sp.w3 = sp.w2 * sp.w1 % PRIME;
  sp.wm[0] = (uint32_t)((sp.w1 << 32) % PRIME); sp.wm[1] = (uint32_t)((sp.w2 << 32) % PRIME);
  sp.wm[2] = (uint32_t)((sp.w3 << 32) % PRIME);
  for (int s2 = 0; s2 < grp.nsym; s2++) {
    for (int x = 0; x < N; x++) sp.symperm[s2][x] = grp.bperm[s2 * N + x];
    sp.symconj[s2] = grp.conj[s2];
  }
  sp.goal_id = 1;
  for (int g = 0; g < hs.G; g++) {
    sp.gflags[g] = hs.gflags[g]; sp.gnq[g] = (int8_t)hs.gnq[g]; sp.gik[g] = (int8_t)hs.gik[g];
    sp.gmask[g] = 0;
    for (int j = 0; j < hs.gnq[g]; j++) sp.gmask[g] |= (uint8_t)(1 << hs.gq[g][j]);
    for (int j = 0; j < 3; j++) sp.gq[g][j] = (int8_t)hs.gq[g][j];
    // how the child update multiplies by this gate: w-power entries (one qubit), a permutation, or general
    const int L = 1 << hs.gnq[g];
    auto unit_power = [](const Zw &z) -> int {   // p with z = w^p, 8 for zero, -1 otherwise
      if (zzero(z)) return 8;
      const int64_t c[4] = {z.a, z.b, z.c, z.d};
      int nz = -1;
      for (int i = 0; i < 4; i++) if (c[i]) { if (nz >= 0) return -1; nz = i; }
      if (c[nz] == 1) return nz;
      if (c[nz] == -1) return nz + 4;
      return -1;
    };
    sp.gkind[g] = GK_GENERAL;
    if (L == 2) {
      bool ok = true;
      for (int i = 0; i < 4; i++) { const int pw = unit_power(hs.ginv[g][i]); ok = ok && pw >= 0; sp.gph[g][i] = (uint8_t)(pw < 0 ? 8 : pw); }
      if (ok) sp.gkind[g] = GK_ONEQ;
    }
    if (sp.gkind[g] == GK_GENERAL) {
      bool perm = true;
      int rowuse = 0;
      for (int lc = 0; lc < L && perm; lc++) {
        int one = -1;
        for (int m = 0; m < L && perm; m++) {
          const Zw z = hs.ginv[g][m * L + lc];
          if (zzero(z)) continue;
          if (one >= 0 || !(z.a == 1 && !z.b && !z.c && !z.d)) perm = false;
          one = m;
        }
        if (one < 0 || (rowuse >> one) & 1) perm = false;
        else { rowuse |= 1 << one; sp.gperm[g][lc] = (uint8_t)one; }
      }
      if (perm) sp.gkind[g] = GK_PERM;
    }
  }
  for (int g = 0; g < hs.G; g++) {      // unit monomials: per column its source column and power
    const int nq = hs.gnq[g], L = 1 << nq;
    bool ok = hs.gik[g] == 0;
    for (int c = 0; c < N && ok; c++) {
      int lc = 0, cnt = 0;
      for (int j = 0; j < nq; j++) lc |= ((c >> hs.gq[g][j]) & 1) << j;
      for (int m = 0; m < L && ok; m++) {
        const Zw z = hs.ginv[g][m * L + lc];
        if (zzero(z)) continue;
        int p = -1;
        for (int w = 0; w < 8; w++) if (zeq(z, zwpow(w))) p = w;
        int src = c;
        for (int j = 0; j < nq; j++) src = (src & ~(1 << hs.gq[g][j])) | (((m >> j) & 1) << hs.gq[g][j]);
        ok = p >= 0 && ++cnt == 1;
        sp.gmono[g][c] = (uint8_t)(src | p << 4);
      }
      ok = ok && cnt == 1;
    }
    if (ok) sp.gflags[g] |= GF_UNITMON;
  }
  for (int g = 0; g < hs.G; g++) {      // the Cliffords whose action on the Paulis is one of the simple ones
    sp.gcol[g] = COL_UNKNOWN;
    if (!(hs.gflags[g] & GF_CLIFFORD) || hs.states) continue;
    const int q = hs.gq[g][0];
    if (sp.gkind[g] == GK_ONEQ) {
      const int p00 = sp.gph[g][0], p01 = sp.gph[g][1], p10 = sp.gph[g][2], p11 = sp.gph[g][3];
      if (p00 < 8 && p11 < 8 && p01 == 8 && p10 == 8) sp.gcol[g] = (uint8_t)((((p11 - p00) & 3) == 0 ? COL_SAME : COL_S) | q << 3);
      else if (p00 == 8 && p11 == 8 && p01 < 8 && p10 < 8) sp.gcol[g] = (uint8_t)((((p10 - p01) & 3) == 0 ? COL_SAME : COL_S) | q << 3);
      else if (p00 < 8 && p01 == p00 && p10 == p00 && p11 == ((p00 + 4) & 7)) sp.gcol[g] = (uint8_t)(COL_H | q << 3);
    } else if (sp.gkind[g] == GK_PERM && hs.gnq[g] == 2) {
      for (int c = 0; c < 2; c++) {      // local control c, target 1 - c
        bool cx = true;
        for (int l = 0; l < 4; l++) cx = cx && sp.gperm[g][l] == (l ^ (((l >> c) & 1) << (1 - c)));
        if (cx) sp.gcol[g] = (uint8_t)(COL_CX | hs.gq[g][c] << 3 | hs.gq[g][1 - c] << 5);
      }
    }
  }
  for (int q = 0; q < 3; q++) {
    sp.qcut[q] = QC_NONE;
    for (int i = 0; i < sp.ncuts && sp.ncuts <= 4; i++)
      if (q < NQ && sp.rad[i] > 1 && (sp.cutmask[i] == 1 << q || sp.cutmask[i] == (N - 1) - (1 << q))) sp.qcut[q] = (uint8_t)(2 * i);
  }
  sp.cuts3 = NQ == 3 && sp.ncuts == 3 && sp.qcut[0] != QC_NONE && sp.qcut[1] != QC_NONE && sp.qcut[2] != QC_NONE &&
             sp.rad[0] == 3 && sp.rad[1] == 3 && sp.rad[2] == 3;
  gi.assign((size_t)GMAX * 64, int4{0, 0, 0, 0});
  for (int g = 0; g < hs.G; g++)
    for (int i = 0; i < LMAX * LMAX; i++) {
      const Zw z = hs.ginv[g][i];
      gi[(size_t)g * 64 + i] = int4{(int)z.a, (int)z.b, (int)z.c, (int)z.d};
    }
  gl.assign(2 * E, longlong2{});
  for (int r = 0; r < N; r++)
    for (int c = 0; c < N; c++) {
      gl[2 * (r * N + c)] = make_longlong2(r == c ? 1 : 0, 0);
      gl[2 * (r * N + c) + 1] = make_longlong2(0, 0);
    }
  sp.unit = !hs.states && unitary(hs.root.data(), N, hs.rk);
  for (int g = 0; g < hs.G; g++) sp.unit = sp.unit && unitary(hs.ginv[g].data(), 1 << hs.gnq[g], hs.gik[g]);
  sp.states = hs.states;
  sp.m = hs.states ? hs.m : N;
  if (hs.states) {                     // the goal: the reference's rows over sqrt2^gk, compared exactly
    sp.goal_id = 0;
    sp.gk = hs.gk;
    for (int e = 0; e < E; e++) {
      const Zw z = hs.goal[e];
      gl[2 * e] = make_longlong2(z.a, z.b);
      gl[2 * e + 1] = make_longlong2(z.c, z.d);
    }
  }
  return sp;
}

template <int NQ>
DevSpec Engine::Impl::prepare(const HostSpec &hs, const SymGroup &grp, int depth, bool nogoal) {
  std::vector<int4> gi;
  std::vector<longlong2> gl;
  DevSpec sp = devspec_host<NQ>(hs, grp, depth, nogoal, gi, gl);
  SpecDev *sd = nullptr;                   // spec tables: uploaded once per parsed spec (small LRU)
  for (auto &x : specs) if (x.uid == hs.uid) sd = &x;
  if (!sd) {
    sd = &specs[0];
    for (auto &x : specs) if (x.used < sd->used) sd = &x;
    sd->ginv.ensure(gi.size() * sizeof(int4)); sd->bad2.ensure(hs.bad2.size() + 1);
    sd->bad3.ensure(hs.bad3.size() * 4 + 4); sd->cxt.ensure(std::max<size_t>(1, hs.cxtable.size()) * 4);
    sd->goal.ensure(gl.size() * sizeof(longlong2));
    ck(cudaMemcpyAsync(sd->ginv.p, gi.data(), gi.size() * sizeof(int4), cudaMemcpyHostToDevice, s), "h2d");
    ck(cudaMemcpyAsync(sd->bad2.p, hs.bad2.data(), hs.bad2.size(), cudaMemcpyHostToDevice, s), "h2d");
    ck(cudaMemcpyAsync(sd->bad3.p, hs.bad3.data(), hs.bad3.size() * 4, cudaMemcpyHostToDevice, s), "h2d");
    if (!hs.cxtable.empty())
      ck(cudaMemcpyAsync(sd->cxt.p, hs.cxtable.data(), hs.cxtable.size() * 4, cudaMemcpyHostToDevice, s), "h2d");
    ck(cudaMemcpyAsync(sd->goal.p, gl.data(), gl.size() * sizeof(longlong2), cudaMemcpyHostToDevice, s), "h2d");
    sd->ginfo.ensure(std::max<size_t>(1, hs.ginfo.size()) * 4);
    if (!hs.ginfo.empty())
      ck(cudaMemcpyAsync(sd->ginfo.p, hs.ginfo.data(), hs.ginfo.size() * 4, cudaMemcpyHostToDevice, s), "h2d");
    ck(cudaStreamSynchronize(s), "spec upload");   // the host vectors above go out of scope
    h2d += (long long)(gi.size() * sizeof(int4) + hs.bad2.size() + hs.bad3.size() * 4 + hs.cxtable.size() * 4 +
                       gl.size() * sizeof(longlong2));
    sd->uid = hs.uid;
  }
  sd->used = ++use_clock;
  sp.ginv = sd->ginv.as<int4>(); sp.bad2 = sd->bad2.as<uint8_t>(); sp.bad3 = sd->bad3.as<uint32_t>();
  sp.cxtable = sd->cxt.as<int>(); sp.goal = sd->goal.as<longlong2>(); sp.ginfo = sd->ginfo.as<int>();

  return sp;
}

template <int NQ>
int Engine::Impl::run(const HostSpec &hs, const Options &opt, const std::function<void(const LevelStats &)> &cb,
                      SearchResult &res) {
  constexpr int N = 1 << NQ, E = N * N;
  const int depth = opt.depth >= 0 ? opt.depth : hs.depth;
  const SymGroup grp = sym_group(hs, opt.sym && !hs.states);   // no symmetry classes for state targets
  res.nsym = grp.nsym;
  // depth 0: the target is the goal (the identity; for state targets the goal rows) (cheese.cu:1794-1801)
  {
    bool done = hs.tk == (hs.states ? hs.gk : 0);
    for (int r = 0; r < N && done; r++)
      for (int c = 0; c < N && done; c++) {
        const Zw x = hs.target[r * N + c];
        done = hs.states ? zeq(x, hs.goal[r * N + c]) : r == c ? (x.a == 1 && !x.b && !x.c && !x.d) : zzero(x);
      }
    if (done && !opt.nogoal) { res.depth0 = true; return RC_CIRCUIT; }
  }
  DevSpec sp = prepare<NQ>(hs, grp, depth, opt.nogoal);

  // storage: int32 limbs unless the target itself needs more (then int64 from the start)
  bool wide = opt.store64 == 1;
  for (const Zw &z : hs.target) if (!fits32(z.a) || !fits32(z.b) || !fits32(z.c) || !fits32(z.d)) wide = true;
  // root node
  fMeta.ensure(sizeof(NodeMeta));
  if (!wide) {
    std::vector<Z4<int32_t>> t32(E);
    for (int i = 0; i < E; i++) t32[i] = {(int32_t)hs.root[i].a, (int32_t)hs.root[i].b, (int32_t)hs.root[i].c, (int32_t)hs.root[i].d};
    fR.ensure(E * sizeof(Z4<int32_t>));
    ck(cudaMemcpyAsync(fR.p, t32.data(), E * sizeof(Z4<int32_t>), cudaMemcpyHostToDevice, s), "h2d");
    h2d += E * sizeof(Z4<int32_t>);
    k_root<NQ, int32_t><<<1, 32, 0, s>>>(sp, fR.as<Z4<int32_t>>(), fMeta.as<NodeMeta>(), hs.rk);
  } else {
    fR.ensure(E * sizeof(Z4<int64_t>));
    ck(cudaMemcpyAsync(fR.p, hs.root.data(), E * sizeof(Zw), cudaMemcpyHostToDevice, s), "h2d");
    h2d += E * sizeof(Zw);
    k_root<NQ, int64_t><<<1, 32, 0, s>>>(sp, fR.as<Z4<int64_t>>(), fMeta.as<NodeMeta>(), hs.rk);
  }
  launches++;
  ck(cudaGetLastError(), "root kernel");
  ck(cudaStreamSynchronize(s), "root");
  int t = 1;
  int rc;
  front_m = 1;
  if (!wide) {
    rc = levels<NQ, int32_t>(hs, sp, opt, depth, t, cb, res);
    if (rc == -2) {   // a limb left int32: widen the current frontier and redo level t with int64 limbs
      DBuf w;
      w.ensure((size_t)front_m * E * sizeof(Z4<int64_t>));
      const size_t ne = (size_t)front_m * E;
      k_widen<<<(unsigned)std::min<size_t>((ne + 255) / 256, (size_t)nsm * 32), 256, 0, s>>>(fR.as<Z4<int32_t>>(),
                                                                                          w.as<Z4<int64_t>>(), ne);
      launches++;
      ck(cudaStreamSynchronize(s), "widen");
      std::swap(fR.p, w.p); std::swap(fR.cap, w.cap);
      w.release();
      wide = true;
      rc = levels<NQ, int64_t>(hs, sp, opt, depth, t, cb, res);
    }
  } else {
    rc = levels<NQ, int64_t>(hs, sp, opt, depth, t, cb, res);
  }
  res.store64 = wide;
  return rc;
}

template <int NQ, typename ST>
void Engine::Impl::eval_bounds(const HostSpec &hs, int count, const int64_t *ent, const int *ks, int *out4) {
  constexpr int E = (1 << NQ) * (1 << NQ);
  const SymGroup grp = sym_group(hs, false);
  const DevSpec sp = prepare<NQ>(hs, grp, hs.depth, false);
  std::vector<Z4<ST>> r((size_t)count * E);
  for (size_t i = 0; i < r.size(); i++)
    r[i] = Z4<ST>{(ST)ent[4 * i], (ST)ent[4 * i + 1], (ST)ent[4 * i + 2], (ST)ent[4 * i + 3]};
  DBuf dR, dK, dO;
  dR.ensure(r.size() * sizeof(Z4<ST>)); dK.ensure((size_t)count * 4 + 4); dO.ensure((size_t)count * 16 + 16);
  ck(cudaMemcpyAsync(dR.p, r.data(), r.size() * sizeof(Z4<ST>), cudaMemcpyHostToDevice, s), "h2d");
  ck(cudaMemcpyAsync(dK.p, ks, (size_t)count * 4, cudaMemcpyHostToDevice, s), "h2d");
  const int grid = std::max(1, std::min((count + EXP_WARPS - 1) / EXP_WARPS, nsm * 8));
  k_eval_bounds<NQ, ST><<<grid, EXP_WARPS * 32, 0, s>>>(sp, dR.as<Z4<ST>>(), dK.as<int>(), count, dO.as<int4>());
  launches++;
  ck(cudaGetLastError(), "bounds kernel");
  ck(cudaMemcpyAsync(out4, dO.p, (size_t)count * 16, cudaMemcpyDeviceToHost, s), "d2h");
  ck(cudaStreamSynchronize(s), "bounds");
  dR.release(); dK.release(); dO.release();
}

int Engine::eval_bounds(const HostSpec &hs, int count, const int64_t *ent, const int *ks, int *out4, std::string &err) {
  try {
    ck(cudaSetDevice(dev_), "cudaSetDevice");
    const size_t E = (size_t)1 << (2 * hs.n);
    bool wide = false;
    for (size_t i = 0; i < (size_t)count * E * 4; i++) if (!fits32(ent[i])) wide = true;
    switch (hs.n * 2 + wide) {
      case 2: impl_->eval_bounds<1, int32_t>(hs, count, ent, ks, out4); break;
      case 3: impl_->eval_bounds<1, int64_t>(hs, count, ent, ks, out4); break;
      case 4: impl_->eval_bounds<2, int32_t>(hs, count, ent, ks, out4); break;
      case 5: impl_->eval_bounds<2, int64_t>(hs, count, ent, ks, out4); break;
      case 6: impl_->eval_bounds<3, int32_t>(hs, count, ent, ks, out4); break;
      case 7: impl_->eval_bounds<3, int64_t>(hs, count, ent, ks, out4); break;
      default: err = "n not built"; return RC_USAGE;
    }
  } catch (const CudaError &e) {
    err = e.what();
    return RC_CUDA;
  }
  return 0;
}

// ---------------- bound evaluation without device allocation ----------------
// For callers that cannot allocate device memory: the spec's gate-matrix, CX and goal tables are staged in a
// file-scope device array instead of engine buffers; the residuals, exponents and bounds stay in the caller's
// device buffers. The array lives on every device that loads this library until the process exits.
namespace {
constexpr size_t NA_GINV = (size_t)GMAX * 64 * sizeof(int4);           // 64 gates x 8 x 8 local matrix
constexpr size_t NA_CXT = (size_t)NOALLOC_MAX_CXTABLE * sizeof(int);
constexpr size_t NA_GOAL = (size_t)64 * 2 * sizeof(longlong2);
static_assert(NA_GINV + NA_CXT + NA_GOAL <= NOALLOC_SCRATCH_BYTES, "no-alloc scratch too small");
static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_SCRATCH_BYTES];
std::mutex g_noalloc_mu;
void *g_noalloc_addr[256];                // per device: the array's device address (set up on first use)

template <int NQ>
void eval_bounds_noalloc_nq(const HostSpec &hs, unsigned char *base, int count, const int64_t *d_entries,
                            const int *d_k, int *d_bounds, cudaStream_t st) {
  const SymGroup grp = sym_group(hs, false);
  std::vector<int4> gi;
  std::vector<longlong2> gl;
  DevSpec sp = devspec_host<NQ>(hs, grp, hs.depth, false, gi, gl);
  // every table is rewritten in full by each call (nothing carries over from the previous call's contents)
  ck(cudaMemcpyAsync(base, gi.data(), NA_GINV, cudaMemcpyHostToDevice, st), "h2d");
  std::vector<int> cx(NOALLOC_MAX_CXTABLE, 0);
  std::copy(hs.cxtable.begin(), hs.cxtable.end(), cx.begin());
  ck(cudaMemcpyAsync(base + NA_GINV, cx.data(), NA_CXT, cudaMemcpyHostToDevice, st), "h2d");
  std::vector<longlong2> g64(64 * 2, longlong2{});
  std::copy(gl.begin(), gl.end(), g64.begin());
  ck(cudaMemcpyAsync(base + NA_GINV + NA_CXT, g64.data(), NA_GOAL, cudaMemcpyHostToDevice, st), "h2d");
  ck(cudaStreamSynchronize(st), "table staging");   // the host tables above go out of scope
  sp.ginv = (const int4 *)base;
  sp.cxtable = (const int *)(base + NA_GINV);
  sp.goal = (const longlong2 *)(base + NA_GINV + NA_CXT);
  sp.bad2 = nullptr;
  sp.bad3 = nullptr;
  int nsm = 148;
  int dev = 0;
  ck(cudaGetDevice(&dev), "cudaGetDevice");
  ck(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev), "SM count");
  const int grid = std::max(1, std::min((count + EXP_WARPS - 1) / EXP_WARPS, nsm * 8));
  k_eval_bounds<NQ, int64_t><<<grid, EXP_WARPS * 32, 0, st>>>(sp, (const Z4<int64_t> *)d_entries, d_k, count,
                                                              (int4 *)d_bounds);
  ck(cudaGetLastError(), "bounds kernel");
}
}  // namespace

int eval_bounds_noalloc(const HostSpec &hs, int count, const int64_t *d_entries, const int *d_k, int *d_bounds,
                        void *stream, std::string &err) {
  if (count < 0) { err = "count < 0"; return RC_USAGE; }
  if (count == 0) return 0;
  if (!d_entries || !d_k || !d_bounds) { err = "null device buffer"; return RC_USAGE; }
  if (((uintptr_t)d_entries & 15) || ((uintptr_t)d_bounds & 15) || ((uintptr_t)d_k & 3)) {
    err = "device buffers must be 16-byte aligned (entries, bounds) and 4-byte aligned (exponents)";
    return RC_USAGE;
  }
  if (hs.n < 1 || hs.n > NQMAX) { err = "n = " + std::to_string(hs.n) + " not built"; return RC_USAGE; }
  if (hs.cxtable.size() > (size_t)NOALLOC_MAX_CXTABLE) {
    err = "CX table of " + std::to_string(hs.cxtable.size()) + " entries exceeds the " +
          std::to_string(NOALLOC_MAX_CXTABLE) + " this entry point stages without allocating";
    return RC_USAGE;
  }
  try {
    int dev = 0;
    ck(cudaGetDevice(&dev), "cudaGetDevice");
    if (dev < 0 || dev >= 256) { err = "device index out of range"; return RC_USAGE; }
    unsigned char *base;
    {
      std::lock_guard<std::mutex> lk(g_noalloc_mu);
      if (!g_noalloc_addr[dev]) {          // once per device, with that device current
        void *p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) { err = std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e); return RC_CUDA; }
        g_noalloc_addr[dev] = p;
      }
      base = (unsigned char *)g_noalloc_addr[dev];
    }
    cudaStream_t st = (cudaStream_t)stream;
    switch (hs.n) {
      case 1: eval_bounds_noalloc_nq<1>(hs, base, count, d_entries, d_k, d_bounds, st); break;
      case 2: eval_bounds_noalloc_nq<2>(hs, base, count, d_entries, d_k, d_bounds, st); break;
      default: eval_bounds_noalloc_nq<3>(hs, base, count, d_entries, d_k, d_bounds, st); break;
    }
  } catch (const CudaError &e) {
    err = e.what();
    return RC_CUDA;
  }
  return 0;
}

Engine::Engine(int device) : impl_(new Impl(device)), dev_(device) {}
Engine::~Engine() { delete impl_; }
size_t Engine::trim() {
  cudaSetDevice(dev_);
  cudaStreamSynchronize(impl_->s);
  return impl_->trim();
}
void *Engine::stream() const { return impl_->s; }

double Engine::int32_peak() {
  ck(cudaSetDevice(dev_), "cudaSetDevice");
  DBuf o;
  o.ensure(64);
  const int iters = 1 << 14, blocks = impl_->nsm * 8, threads = 256;
  float best = 1e30f;
  for (int rep = 0; rep < 6; rep++) {
    ck(cudaEventRecord(impl_->ev[0], impl_->s), "event");
    k_imad_probe<<<blocks, threads, 0, impl_->s>>>(iters, 0x2545f491u, o.as<uint32_t>());
    ck(cudaEventRecord(impl_->ev[1], impl_->s), "event");
    ck(cudaEventSynchronize(impl_->ev[1]), "probe");
    float ms = 0;
    cudaEventElapsedTime(&ms, impl_->ev[0], impl_->ev[1]);
    if (rep > 0 && ms < best) best = ms;
  }
  o.release();
  const double imads = (double)blocks * threads * iters * 8;
  return 2.0 * imads / (best * 1e-3);
}

int Engine::sort_pairs(uint64_t *keys, uint32_t *vals, size_t n, int lo, int hi, float *ms, std::string &err) {
  if (lo < 0 || hi > 64 || lo > hi || (hi - lo) % 8) { err = "bit range [lo, hi) must be whole bytes within 64"; return RC_USAGE; }
  try {
    ck(cudaSetDevice(dev_), "cudaSetDevice");
    Impl &I = *impl_;
    I.k1.ensure(n * 8 + 8); I.v1.ensure(n * 4 + 4);
    I.hist.ensure(sort_hist_words(n) * 4);
    I.part.ensure(scan_partials_words(sort_hist_words(n)) * 4);
    SortScratch sc{I.hist.as<uint32_t>(), I.part.as<uint32_t>(), I.hist.cap / 4, I.part.cap / 4};
    sc.flags = I.sort_flags();
    ck(cudaEventRecord(I.ev[0], I.s), "event");
    int nl = 0;
    const bool f = radix_sort(keys, vals, I.k1.as<uint64_t>(), I.v1.as<uint32_t>(), n, lo, hi, sc, I.s, &nl);
    I.launches += nl;
    ck(cudaEventRecord(I.ev[1], I.s), "event");
    if (f) {
      ck(cudaMemcpyAsync(keys, I.k1.p, n * 8, cudaMemcpyDeviceToDevice, I.s), "d2d");
      ck(cudaMemcpyAsync(vals, I.v1.p, n * 4, cudaMemcpyDeviceToDevice, I.s), "d2d");
    }
    ck(cudaGetLastError(), "sort");
    const uint32_t flags = sort_failed(sc, I.s);
    float t = 0;
    ck(cudaEventElapsedTime(&t, I.ev[0], I.ev[1]), "event");
    if (ms) *ms = t;
    if (flags & 2u) { err = "the keys changed while they were sorted (order the buffers before the call)"; return RC_CUDA; }
    if (flags & 1u) err = "a look-back wait gave up (the result is exact; the predecessors were counted directly)";
  } catch (const CudaError &e) {
    err = e.what();
    return RC_CUDA;
  }
  return 0;
}

int Engine::search(const HostSpec &hs, const Options &opt, const std::function<void(const LevelStats &)> &cb,
                   SearchResult &res) {
  res = SearchResult{};
  const double t0 = now_s();
  const long long l0 = impl_->launches, e0 = impl_->expand_launches, h0 = impl_->h2d, d0 = impl_->d2h;
  int rc;
  try {
    ck(cudaSetDevice(dev_), "cudaSetDevice");
    if (opt.mitm && hs.states) {
      res.nsym = 1;
      res.error = "--mitm: unitary targets only";
      rc = RC_USAGE;
    } else if (opt.mitm) {
      switch (hs.n) {
        case 1: rc = impl_->run_mitm<1>(hs, opt, cb, res); break;
        case 2: rc = impl_->run_mitm<2>(hs, opt, cb, res); break;
        case 3: rc = impl_->run_mitm<3>(hs, opt, cb, res); break;
        default: res.error = "n = " + std::to_string(hs.n) + " not built"; rc = RC_USAGE;
      }
    } else if (opt.table_k > 0 && !hs.states) {
      switch (hs.n) {
        case 1: rc = impl_->run_table<1>(hs, opt, cb, res); break;
        case 2: rc = impl_->run_table<2>(hs, opt, cb, res); break;
        case 3: rc = impl_->run_table<3>(hs, opt, cb, res); break;
        default: res.error = "n = " + std::to_string(hs.n) + " not built"; rc = RC_USAGE;
      }
    } else {
      switch (hs.n) {
        case 1: rc = impl_->run<1>(hs, opt, cb, res); break;
        case 2: rc = impl_->run<2>(hs, opt, cb, res); break;
        case 3: rc = impl_->run<3>(hs, opt, cb, res); break;
        default: res.error = "n = " + std::to_string(hs.n) + " not built"; rc = RC_USAGE;
      }
    }
  } catch (const CudaError &e) {
    res.error = e.what();
    rc = RC_CUDA;
  }
  res.launches = impl_->launches - l0;
  res.expand_launches = impl_->expand_launches - e0;
  res.h2d_bytes = impl_->h2d - h0;
  res.d2h_bytes = impl_->d2h - d0;
  res.total_ms = (now_s() - t0) * 1e3;
  res.rc = rc;
  return rc;
}

// ---------------- batched search (continuous batching over many jobs of one qubit count) ----------------
namespace {

__global__ void k_jst_init(DevStats *jst, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    DevStats z;
    memset(&z, 0, sizeof z);
    z.first_found = ~0ULL;
    jst[i] = z;
  }
}

// the roots of newly admitted jobs: one warp each (the bounds of k_root with the job's spec)
template <int NQ>
__global__ void k_root_batch(const DevSpec *specs, const uint32_t *rjob, const int *rtk, int nroots,
                             const Z4<int32_t> *R, NodeMeta *meta) {
  constexpr int E = (1 << NQ) * (1 << NQ);
  __shared__ Z4<int32_t> S[E];
  const int i = blockIdx.x, lane = threadIdx.x;
  if (i >= nroots) return;
  const DevSpec &sp = specs[rjob[i]];
  const int tk = rtk[i];
  for (int e = lane; e < E; e += 32) S[e] = R[(size_t)i * E + e];
  __syncwarp();
  int T = 0, c2 = 0, needs = 0;
  Cheap ch{false, 0, 0};
  if (sp.standard || sp.lite) T = ptm_bound<NQ, int32_t>(S, tk, lane);
  if (sp.standard) {
    c2 = warp_cx_bound<NQ, int32_t>(S, sp, lane, 0, 0, needs);
    ch = warp_cheap<NQ, int32_t>(S, tk, sp, lane, false, true, (1 << NQ) - 1, 0);
  }
  if (lane == 0) {
    NodeMeta m;
    m.k = (int16_t)tk; m.T = (uint8_t)(T > 255 ? 255 : T); m.c2 = (uint8_t)c2; m.g1 = m.g2 = 0xff;
    m.hsn = (uint8_t)((ch.hs == 2 ? 1 : 0) | (ch.ntriv << 1));
    m.needs = (uint8_t)needs;
    m.cols = 0;
    meta[i] = m;
  }
}

// survivors of jobs still running -> (key, slot) pairs; the job is mixed into the key so runs stay within a job
__global__ void k_bsort_init(const uint64_t *h1, const uint64_t *sidx, size_t n, const uint32_t *fjob,
                             const uint8_t *jact, uint64_t *keys, uint32_t *vals, unsigned long long *cnt) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const size_t nit = (n + stride - 1) / stride;
  const int lane = threadIdx.x & 31;
  for (size_t it = 0; it < nit; it++) {
    const size_t i = it * stride + blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    uint32_t job = 0;
    bool act = false;
    if (i < n) { job = fjob[sidx[i] / BATCH_GS]; act = jact[job] != 0; }
    const unsigned bal = __ballot_sync(FULL, act);
    if (!bal) continue;
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(cnt, (unsigned long long)__popc(bal));
    base = __shfl_sync(FULL, base, 0);
    if (act) {
      const unsigned long long pos = base + __popc(bal & ((1u << lane) - 1));
      keys[pos] = h1[i] + (uint64_t)(job + 1) * 0x9e3779b97f4a7c15ULL;
      vals[pos] = (uint32_t)i;
    }
  }
}

__global__ void k_bcount(const uint64_t *kidx, size_t nk, const uint32_t *fjob, unsigned long long *jdist) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nk; i += (size_t)gridDim.x * blockDim.x) {
    // the indices are in order, so a warp's 32 are mostly one job's: one addition per job in the warp (2.6 -> 0.3 ms
    // over a batch of 96 jobs)
    const uint32_t job = fjob[kidx[i] / BATCH_GS];
    const unsigned peers = __match_any_sync(__activemask(), job);
    if ((int)(threadIdx.x & 31) == __ffs((int)peers) - 1) atomicAdd(&jdist[job], (unsigned long long)__popc(peers));
  }
}
// circuits of jobs that found the goal: child o at step s, at job level t; walked back through the tree of steps
// s - 1 .. s0 (the job's first step). A node carried over a step its job waited has gate 0xff there.
__global__ void k_walk(const unsigned long long *fo, const int *ft, const int *fs, const int *fs0, int nf,
                       const uint32_t *const *tpar, const uint8_t *const *tgat, int *out, int *bad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nf) return;
  const unsigned long long o = fo[i];
  const int t = ft[i], s = fs[i], s0 = fs0[i];
  int *c = out + (size_t)i * MAXDEPTH_WALK;
  int pos = t - 1;
  c[pos] = (int)(o % BATCH_GS);
  unsigned long long p = o / BATCH_GS;
  for (int st = s - 1; st >= s0 && pos > 0; st--) {
    const uint8_t g = tgat[st][p];
    p = tpar[st][p];
    if (g != 0xff) c[--pos] = g;
  }
  if (pos != 0) atomicOr(bad, 1);
}

// nodes of jobs that wait this step: carried to the next frontier unchanged (tree: same node, no gate)
template <typename ST>
__global__ void k_carry(long long p0, long long n, int E, const Z4<ST> *R, const NodeMeta *meta, const uint32_t *fjob,
                        Z4<ST> *R2, NodeMeta *meta2, uint32_t *fjob2, uint32_t *par, uint8_t *gat) {
  const size_t tot = (size_t)n * E;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < tot; i += (size_t)gridDim.x * blockDim.x) {
    const size_t j = i / E;
    R2[i] = R[(size_t)p0 * E + i];
    if (i % E == 0) { meta2[j] = meta[p0 + j]; fjob2[j] = fjob[p0 + j]; par[j] = (uint32_t)(p0 + j); gat[j] = 0xff; }
  }
}

// device addresses of one spec's tables (inverse gates, window rules, CX table, goal), shared by equal specs
struct SpecTables { const int4 *ginv; const uint8_t *bad2; const uint32_t *bad3; const int *cxt; const longlong2 *goal; };

uint64_t bytes_hash(uint64_t h, const void *p, size_t n) {
  const unsigned char *b = (const unsigned char *)p;
  for (size_t i = 0; i < n; i++) { h ^= b[i]; h *= 1099511628211ULL; }
  return h;
}

}  // namespace

struct BatchSession::Impl {
  virtual ~Impl() {}
  virtual int nq() const = 0;
  virtual int submit(const HostSpec &hs, const Options &opt) = 0;
  virtual int step() = 0;
  virtual int running() const = 0;
  virtual const BatchJob &job(int id) const = 0;
  virtual int jobs() const = 0;
  virtual long long frontier() const = 0;
  virtual long long launches() const = 0;
  virtual long long steps() const = 0;
  virtual size_t device_bytes() const = 0;
  virtual size_t projected_bytes() const = 0;
  virtual void set_budget(size_t bytes) = 0;
  virtual long long waits() const = 0;
  BatchTuning tune;
};

namespace {

template <int NQ>
struct BatchImpl : BatchSession::Impl {
  static constexpr int N = 1 << NQ, E = N * N;
  using ST = int32_t;
  struct Job {
    HostSpec hs;
    Options opt;
    int depth = 0;
    DevSpec sp;
    int t = 1;                       // the level this job runs at its next step
    long long seg = 0;               // its nodes in the frontier
    double rate = 1.0;               // survivors per child at its previous level
    double drate = 1.0;              // distinct per survivor at its previous level
    bool queued = true, running = false;
    BatchJob out;
  };
  Engine &eng;
  cudaStream_t s;
  int nsm = 148;
  std::vector<Job> J;
  std::vector<int> queue;            // submitted, not yet admitted
  std::map<uint64_t, SpecTables> tables;
  std::vector<DBuf> arenas;          // the spec tables of each admission, one device block each, kept for the session
  DBuf dspecs, jt, jst, jact, jdist;
  // the large buffers grow in place (frontiers, survivors, T queue, dedupe scratch): no copies, no frees
  VBuf fR, fMeta, fJob, fR2, fMeta2, fJob2;
  VBuf sH1, sH2, sIdx, sMeta;              // survivors: 40-byte records
  DBuf stats;
  DBuf bgoal, jgoal;                       // the goal pass: counters + candidate list, per-job results
  VBuf tq, tqleft;                         // deferred T evaluations; TBoundArgs::left
  VBuf k0, k1, v0, v1, work, tmp, kidx, kslot;
  DBuf hist, part, cnt;
  DBuf rJob, rTk, tptr, wbuf;
  std::vector<DBuf> tpar, tgat;      // tree of every step
  std::vector<DBuf> spare_par, spare_gat;   // tree buffers of released steps, for later steps
  long long m = 0;                   // frontier nodes
  long long tree_lo = 0;             // tree levels below this step are released
  long long nlaunch = 0, nstep = 0;
  int nrun = 0;
  size_t spec_cap = 0;

  BatchImpl(Engine &e) : eng(e), s((cudaStream_t)e.stream()) {
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, e.device());
    stats.ensure(sizeof(DevStats));
    cnt.ensure(64);
    size_t fr = 0, tot = 0;
    if (cudaMemGetInfo(&fr, &tot) == cudaSuccess) budget = (size_t)(0.8 * (double)fr);
  }
  size_t budget = (size_t)64 << 30;  // device bytes a step may plan for (frontiers + survivors)
  void set_budget(size_t b) override { budget = b; }
  long long nwait = 0;               // job-steps spent waiting for memory
  long long waits() const override { return nwait; }
  ~BatchImpl() override {
    cudaSetDevice(eng.device());
    cudaStreamSynchronize(s);          // unmapping does not wait for the device
    for (DBuf *b : {&dspecs, &jt, &jst, &jact, &jdist, &stats, &hist, &part, &cnt, &rJob, &rTk, &tptr, &wbuf, &bgoal,
                    &jgoal})
      b->release();
    for (VBuf *b : {&fR, &fMeta, &fJob, &fR2, &fMeta2, &fJob2, &sH1, &sH2, &sIdx, &sMeta, &tq, &tqleft, &k0, &k1, &v0, &v1,
                    &work, &tmp, &kidx, &kslot})
      b->release();
    for (auto &b : tpar) b.release();
    for (auto &b : spare_par) b.release();
    for (auto &b : spare_gat) b.release();
    for (auto &b : tgat) b.release();
    for (auto &b : arenas) b.release();
  }
  int nq() const override { return NQ; }
  int running() const override { return nrun + (int)queue.size(); }
  const BatchJob &job(int id) const override { return J.at(id).out; }
  int jobs() const override { return (int)J.size(); }
  long long frontier() const override { return m; }
  long long launches() const override { return nlaunch; }
  long long steps() const override { return nstep; }
  size_t device_bytes() const override {
    size_t b = 0;
    for (const DBuf *x : {&dspecs, &jt, &jst, &jact, &jdist, &hist, &part})
      b += x->cap;
    for (const VBuf *x : {&fR, &fMeta, &fJob, &fR2, &fMeta2, &fJob2, &sH1, &sH2, &sIdx, &sMeta, &tq, &tqleft, &k0, &k1, &v0, &v1,
                          &work, &tmp, &kidx, &kslot})
      b += x->cap;
    for (auto &x : tpar) b += x.cap;
    for (auto &x : tgat) b += x.cap;
    for (auto &x : spare_par) b += x.cap;
    for (auto &x : spare_gat) b += x.cap;
    for (auto &x : arenas) b += x.cap;
    return b;
  }

  // device bytes of a frontier node with its tree entry, and of a survivor record with its dedupe sort entries
  static constexpr size_t NODE_BYTES = E * sizeof(Z4<ST>) + sizeof(NodeMeta) + 4 + 5;
  static constexpr size_t SURV_BYTES = 48 + 48;
  static constexpr unsigned long long SOLO_CHILDREN = 1ull << 22;
  // expected nodes of the job's next frontier: its children at the previous level's survivor and distinct rates,
  // with a quarter more survivors and 1024 nodes to spare (every child at the first level)
  double next_nodes(const Job &j) const {
    const double all = j.t < j.depth ? (double)j.seg * j.hs.G : 0.0;
    return std::min(all, (1.25 * j.rate * all + 1024.0) * j.drate);
  }
  size_t projected_bytes() const override {   // this frontier, the next one, and one chunk's survivor room
    double b = (double)m * NODE_BYTES, want = 0;
    for (const Job &j : J)
      if (j.running && j.t < j.depth) {
        const double all = (double)j.seg * j.hs.G;
        b += next_nodes(j) * NODE_BYTES;
        want += std::min(all, 1.5 * j.rate * all + 4096.0);
      }
    return (size_t)(b + std::min(want, (double)(tune.chunk_bytes / SURV_BYTES)) * SURV_BYTES);
  }

  int submit(const HostSpec &hs, const Options &opt) override {
    Job j;
    j.hs = hs;
    j.opt = opt;
    j.depth = opt.depth >= 0 ? opt.depth : hs.depth;
    J.push_back(std::move(j));
    queue.push_back((int)J.size() - 1);
    return (int)J.size() - 1;
  }

  void finish(Job &j, int rc) {
    j.out.done = true;
    j.out.res.rc = rc;
    j.out.finished_step = (int)nstep;
    if (j.running) nrun--;
    j.running = false;
  }
  void run_plain(Job &j) {
    j.out.levels.clear();
    SearchResult r;
    eng.search(j.hs, j.opt, [&](const LevelStats &L) { j.out.levels.push_back(L); }, r);
    j.out.res = r;
    j.out.plain = true;
    j.out.done = true;
    j.out.finished_step = (int)nstep;
  }

  // Host staging of one admission: every new spec's tables, then the admitted jobs' device specs, root residuals and
  // (job, T exponent) pairs, each section 256-byte aligned, moved to the device by one copy. Pageable copies wait for
  // the stream, so one copy per admission instead of several per job.
  struct Stage {
    std::vector<unsigned char> b;
    size_t put(const void *p, size_t n) {
      const size_t o = (b.size() + 255) & ~(size_t)255;
      b.resize(o + std::max<size_t>(n, 4), 0);
      if (n) std::memcpy(b.data() + o, p, n);
      return o;
    }
  };

  // the spec's device specialisation; its tables come from an earlier admission when an equal spec had them, else
  // they are staged (offsets into the staging block, made device addresses once the block is on the device)
  void stage_spec(Job &j, Stage &st, std::map<uint64_t, std::array<size_t, 5>> &fresh, std::vector<std::pair<int, uint64_t>> &fix,
                  int id) {
    const SymGroup grp = sym_group(j.hs, j.opt.sym);
    j.out.res.nsym = grp.nsym;
    std::vector<int4> gi;
    std::vector<longlong2> gl;
    j.sp = devspec_host<NQ>(j.hs, grp, j.depth, false, gi, gl);
    uint64_t h = 1469598103934665603ULL;
    h = bytes_hash(h, gi.data(), gi.size() * sizeof(int4));
    h = bytes_hash(h, j.hs.bad2.data(), j.hs.bad2.size());
    h = bytes_hash(h, j.hs.bad3.data(), j.hs.bad3.size() * 4);
    h = bytes_hash(h, j.hs.cxtable.data(), j.hs.cxtable.size() * 4);
    h = bytes_hash(h, gl.data(), gl.size() * sizeof(longlong2));
    auto it = tables.find(h);
    if (it != tables.end()) {
      const SpecTables &t = it->second;
      j.sp.ginv = t.ginv; j.sp.bad2 = t.bad2; j.sp.bad3 = t.bad3; j.sp.cxtable = t.cxt; j.sp.goal = t.goal;
      return;
    }
    if (!fresh.count(h))
      fresh[h] = {st.put(gi.data(), gi.size() * sizeof(int4)), st.put(j.hs.bad2.data(), j.hs.bad2.size()),
                  st.put(j.hs.bad3.data(), j.hs.bad3.size() * 4), st.put(j.hs.cxtable.data(), j.hs.cxtable.size() * 4),
                  st.put(gl.data(), gl.size() * sizeof(longlong2))};
    fix.push_back({id, h});
  }

  // admit the queued jobs: depth-0 and unsupported ones finish here, the others append their root to the frontier
  void admit() {
    std::vector<int> roots;
    Stage st;
    std::map<uint64_t, std::array<size_t, 5>> fresh;
    std::vector<std::pair<int, uint64_t>> fix;
    for (int id : queue) {
      Job &j = J[id];
      j.queued = false;
      j.out.joined_step = (int)nstep;
      bool ident = j.hs.tk == 0;
      for (int r = 0; r < N && ident; r++)
        for (int c = 0; c < N && ident; c++) {
          const Zw x = j.hs.target[r * N + c];
          ident = r == c ? (x.a == 1 && !x.b && !x.c && !x.d) : zzero(x);
        }
      if (ident && !j.opt.nogoal) { j.out.res.depth0 = true; j.out.res.nsym = sym_group(j.hs, j.opt.sym).nsym; finish(j, RC_CIRCUIT); continue; }
      bool wide = j.opt.store64 == 1;
      auto f32 = [](int64_t v) { return v >= INT32_MIN && v <= INT32_MAX; };
      for (const Zw &z : j.hs.target) if (!f32(z.a) || !f32(z.b) || !f32(z.c) || !f32(z.d)) wide = true;
      if (wide || !j.opt.dedupe || j.opt.nogoal || j.depth < 1 || j.depth > MAXDEPTH_WALK) { run_plain(j); continue; }
      stage_spec(j, st, fresh, fix, id);
      roots.push_back(id);
    }
    const int qlo = queue.empty() ? 0 : queue.front(), qhi = queue.empty() ? -1 : queue.back();
    queue.clear();
    // device specs: one per job id
    if (J.size() > spec_cap) {
      spec_cap = std::max<size_t>(J.size(), spec_cap * 2);
      DBuf nd;
      nd.ensure(spec_cap * sizeof(DevSpec));
      if (dspecs.p) ck(cudaMemcpyAsync(nd.p, dspecs.p, dspecs.cap < spec_cap * sizeof(DevSpec) ? dspecs.cap : spec_cap * sizeof(DevSpec), cudaMemcpyDeviceToDevice, s), "d2d");
      ck(cudaStreamSynchronize(s), "specs");
      dspecs.release();
      dspecs = nd;
      nd.p = nullptr;
    }
    if (roots.empty()) return;
    // the staged tables get their device block first: the job specs staged after them hold its addresses
    st.b.resize((st.b.size() + 255) & ~(size_t)255, 0);
    const size_t tables_end = st.b.size();
    DBuf arena;
    if (tables_end) {
      arena.ensure(tables_end);
      const char *base = arena.as<char>();
      for (auto &kv : fresh)
        tables[kv.first] = SpecTables{(const int4 *)(base + kv.second[0]), (const uint8_t *)(base + kv.second[1]),
                                      (const uint32_t *)(base + kv.second[2]), (const int *)(base + kv.second[3]),
                                      (const longlong2 *)(base + kv.second[4])};
      for (auto &f : fix) {
        const SpecTables &t = tables[f.second];
        DevSpec &sp = J[f.first].sp;
        sp.ginv = t.ginv; sp.bad2 = t.bad2; sp.bad3 = t.bad3; sp.cxtable = t.cxt; sp.goal = t.goal;
      }
    }
    // queued ids are consecutive and newer than every admitted job: their specs are one range of the spec array
    // (jobs that finished above get a zeroed entry they never read)
    std::vector<DevSpec> sps((size_t)(qhi - qlo + 1));
    std::memset((void *)sps.data(), 0, sps.size() * sizeof(DevSpec));
    const long long nr = (long long)roots.size();
    std::vector<Z4<int32_t>> rr(roots.size() * E);
    std::vector<uint32_t> rjk(2 * roots.size());
    for (size_t i = 0; i < roots.size(); i++) {
      Job &j = J[roots[i]];
      for (int e = 0; e < E; e++)
        rr[i * E + e] = {(int32_t)j.hs.root[e].a, (int32_t)j.hs.root[e].b, (int32_t)j.hs.root[e].c,
                         (int32_t)j.hs.root[e].d};
      rjk[i] = (uint32_t)roots[i];
      rjk[roots.size() + i] = (uint32_t)j.hs.rk;
      sps[roots[i] - qlo] = j.sp;
      j.t = 1;
      j.seg = 1;
      j.running = true;
      nrun++;
    }
    const size_t o_sp = st.put(sps.data(), sps.size() * sizeof(DevSpec));
    const size_t o_rr = st.put(rr.data(), rr.size() * sizeof(Z4<int32_t>));
    const size_t o_rj = st.put(rjk.data(), rjk.size() * 4);
    // grow the frontier (contents kept); new tables go to a device block kept for the session, the rest of the staged
    // bytes to a work buffer, from which the specs and the roots' residuals are copied into place
    grow_keep(fR, (size_t)(m + nr) * E * sizeof(Z4<ST>), (size_t)m * E * sizeof(Z4<ST>));
    grow_keep(fMeta, (size_t)(m + nr) * sizeof(NodeMeta), (size_t)m * sizeof(NodeMeta));
    grow_keep(fJob, (size_t)(m + nr) * 4, (size_t)m * 4);
    if (tables_end) {
      ck(cudaMemcpyAsync(arena.p, st.b.data(), tables_end, cudaMemcpyHostToDevice, s), "h2d");
      arenas.push_back(arena);
      arena.p = nullptr;
    }
    wbuf.ensure(st.b.size() - tables_end);
    ck(cudaMemcpyAsync(wbuf.p, st.b.data() + tables_end, st.b.size() - tables_end, cudaMemcpyHostToDevice, s), "h2d");
    const char *w = wbuf.as<char>() - tables_end;     // staging offsets past the tables, as device addresses
    ck(cudaMemcpyAsync(dspecs.as<DevSpec>() + qlo, w + o_sp, sps.size() * sizeof(DevSpec), cudaMemcpyDeviceToDevice, s),
       "d2d");
    ck(cudaMemcpyAsync(fR.as<Z4<ST>>() + m * E, w + o_rr, rr.size() * sizeof(Z4<int32_t>), cudaMemcpyDeviceToDevice, s),
       "d2d");
    const uint32_t *rj = (const uint32_t *)(w + o_rj);
    ck(cudaMemcpyAsync(fJob.as<uint32_t>() + m, rj, nr * 4, cudaMemcpyDeviceToDevice, s), "d2d");
    k_root_batch<NQ><<<(unsigned)nr, 32, 0, s>>>(dspecs.as<DevSpec>(), rj, (const int *)(rj + nr), (int)nr,
                                                 fR.as<Z4<ST>>() + m * E, fMeta.as<NodeMeta>() + m);
    nlaunch++;
    ck(cudaGetLastError(), "root kernel");
    ck(cudaStreamSynchronize(s), "admit");
    m += nr;
  }

  void grow_keep(VBuf &b, size_t bytes, size_t) { b.ensure(bytes); }   // grows in place: contents stay
  // grow b to `bytes`, keeping its first `keep` bytes (half again as much room below 1 GB, a tenth above)
  void grow_keep(DBuf &b, size_t bytes, size_t keep) {
    if (bytes <= b.cap) return;
    DBuf nb;
    nb.ensure(bytes + (bytes < ((size_t)1 << 30) ? bytes / 2 : bytes / 10));
    if (keep) ck(cudaMemcpyAsync(nb.p, b.p, keep, cudaMemcpyDeviceToDevice, s), "d2d");
    ck(cudaStreamSynchronize(s), "grow");
    b.release();
    b = nb;
    nb.p = nullptr;
  }

  // One level of every running job. The frontier holds the jobs in id order, each contiguous; it is processed in
  // chunks of whole jobs whose children fit the survivor budget: expand, then (found / overflowed jobs leave)
  // dedupe over the chunk's survivors and append its distinct children to the next frontier and the tree.
  int step() override {
    ck(cudaSetDevice(eng.device()), "cudaSetDevice");
    if (!queue.empty()) admit();
    if (m == 0) { nstep++; return running(); }
    const double t0 = now_s();
    const int nj = (int)J.size();
    std::vector<int> ht(nj, 0);
    for (int i = 0; i < nj; i++) ht[i] = J[i].t;
    jt.ensure(nj * 4); jst.ensure(nj * sizeof(DevStats)); jact.ensure(nj + 4); jdist.ensure(nj * 8);
    ck(cudaMemcpyAsync(jt.p, ht.data(), nj * 4, cudaMemcpyHostToDevice, s), "h2d");
    k_jst_init<<<(nj + 255) / 256, 256, 0, s>>>(jst.as<DevStats>(), nj);
    nlaunch++;
    const size_t rec = SURV_BYTES, node = NODE_BYTES;
    const unsigned long long cap_limit = std::max<unsigned long long>(1 << 16, tune.chunk_bytes / rec);
    // the plan, in frontier (= id) order: chunks of advancing jobs whose expected survivors fit the survivor
    // budget, and runs of waiting jobs carried over unchanged. A job advances while the step's planned memory (this
    // frontier, the next one at each job's last survivor and distinct rates, the survivor room of one chunk, which
    // every chunk reuses) stays under the session budget; the first job always advances.
    struct Op { bool carry; long long p0, p1; unsigned long long cap, all; std::vector<int> jobs; bool solo = false; };
    std::vector<Op> ops;
    size_t step_budget = budget;
    if ((size_t)m * node * 8 > budget / 4) {              // a large step: never plan past what the device has left
      size_t fr = 0, tot = 0;
      if (cudaMemGetInfo(&fr, &tot) == cudaSuccess) {
        const size_t mine = fR2.cap + fMeta2.cap + fJob2.cap + sH1.cap + sH2.cap + sIdx.cap + sMeta.cap + k0.cap +
                            k1.cap + v0.cap + v1.cap + kidx.cap + kslot.cap + work.cap + tmp.cap;
        step_budget = std::min(step_budget, (size_t)(0.9 * (double)(fr + mine)));
      }
    }
    {
      size_t planned = (size_t)m * node;
      unsigned long long want_all = 0;
      bool any_adv = false;
      Op c{false, 0, 0, 0, 0, {}};
      long long off = 0;
      for (int i = 0; i < nj; i++) {
        Job &j = J[i];
        if (!j.running || j.seg == 0) continue;
        const unsigned long long all = j.t < j.depth ? (unsigned long long)j.seg * j.hs.G : 0;
        const unsigned long long want = all ? std::min<unsigned long long>(all, (unsigned long long)(1.5 * j.rate * (double)all) + 4096) : 0;
        const size_t cost = (size_t)next_nodes(j) * node;
        const size_t room = (size_t)std::min(cap_limit, want_all + want) * rec;
        const bool adv = !any_adv || planned + cost + room <= step_budget;
        planned += adv ? cost : (size_t)j.seg * node;
        if (adv) want_all += want;
        any_adv |= adv;
        // a job of at least SOLO_CHILDREN children fills the GPU by itself: it gets a chunk of its own (the one-job
        // level kernel); smaller jobs share chunks
        const bool solo = adv && all >= SOLO_CHILDREN;
        if (!c.jobs.empty() && (c.carry == adv || (adv && (c.cap + want > cap_limit || solo || c.solo)))) {
          ops.push_back(c);
          c = Op{!adv, off, off, 0, 0, {}};
        }
        c.carry = !adv;
        c.solo = solo;
        c.jobs.push_back(i);
        if (adv) { c.cap += want; c.all += all; }
        off += j.seg;
        c.p1 = off;
      }
      if (!c.jobs.empty()) ops.push_back(c);
      if (off != m) throw std::logic_error("batch frontier out of step with its jobs");
      for (Op &o : ops) if (!o.carry) o.cap = std::min(o.all, std::max<unsigned long long>(o.cap, 1 << 20));
    }
    if ((long long)tpar.size() <= nstep) { tpar.resize(nstep + 1); tgat.resize(nstep + 1); }
    {
      size_t est = 0;                                     // next frontier: carried nodes + expected distinct children
      for (const Op &o : ops) {
        if (o.carry) { est += (size_t)(o.p1 - o.p0); continue; }
        for (int i : o.jobs) est += (size_t)next_nodes(J[i]);
      }
      // (the next frontier itself grows in place chunk by chunk; the tree is sized ahead, its growth copies)
      if (!tpar[nstep].p && !spare_par.empty()) {        // tree buffers of released levels are reused
        tpar[nstep] = spare_par.back(); spare_par.pop_back();
        tgat[nstep] = spare_gat.back(); spare_gat.pop_back();
      }
      tpar[nstep].ensure(est * 4 + 4); tgat[nstep].ensure(est + 4);
    }
    std::vector<DevStats> hj(nj);
    std::vector<uint8_t> act(nj, 0);
    std::vector<unsigned long long> dist(nj, 0);
    std::vector<int> overflow_ids;
    size_t total_distinct = 0;
    DevStats *dst = stats.as<DevStats>();
    for (const Op &ch : ops) {
      if (ch.carry) {                                     // waiting jobs: nodes carried over unchanged
        const long long n = ch.p1 - ch.p0;
        const size_t o0 = total_distinct, o1 = total_distinct + (size_t)n;
        grow_keep(tpar[nstep], o1 * 4 + 4, o0 * 4);
        grow_keep(tgat[nstep], o1 + 4, o0);
        grow_keep(fR2, o1 * E * sizeof(Z4<ST>) + 16, o0 * E * sizeof(Z4<ST>));
        grow_keep(fMeta2, o1 * sizeof(NodeMeta) + 16, o0 * sizeof(NodeMeta));
        grow_keep(fJob2, o1 * 4 + 4, o0 * 4);
        const size_t tot = (size_t)n * E;
        const unsigned gg = (unsigned)std::max<size_t>(1, std::min<size_t>((tot + 255) / 256, (size_t)nsm * 32));
        k_carry<ST><<<gg, 256, 0, s>>>(ch.p0, n, E, fR.as<Z4<ST>>(), fMeta.as<NodeMeta>(), fJob.as<uint32_t>(),
                                       fR2.as<Z4<ST>>() + o0 * E, fMeta2.as<NodeMeta>() + o0, fJob2.as<uint32_t>() + o0,
                                       tpar[nstep].as<uint32_t>() + o0, tgat[nstep].as<uint8_t>() + o0);
        nlaunch++;
        nwait += (long long)ch.jobs.size();
        ck(cudaGetLastError(), "carry");
        total_distinct = o1;
        continue;
      }
      const long long cm = ch.p1 - ch.p0;
      const int jlo = ch.jobs.front(), jn = ch.jobs.back() - jlo + 1;
      unsigned long long cap = std::min<unsigned long long>(ch.cap, cap_limit);
      unsigned long long tqcap = 1024;                  // deferred T evaluations: one per non-Clifford child at most
      for (int i : ch.jobs) {
        int ncl = 0;
        for (int g = 0; g < J[i].hs.G; g++) ncl += !(J[i].hs.gflags[g] & GF_CLIFFORD);
        tqcap += (unsigned long long)J[i].seg * (unsigned long long)std::max(1, ncl);
      }
      TboundForms forms{false, false};                  // those that any of the chunk's jobs needs
      for (int i : ch.jobs) {
        const TboundForms f = tbound_forms<NQ, ST>(J[i].hs, J[i].sp, J[i].t, J[i].sp.depth);
        forms.packed |= f.packed;
        forms.general |= f.general;
      }
      DevStats h{};
      // goal pass over the chunk: jobs whose goal it finds skip their found level in the level kernels
      bgoal.ensure(sizeof(GoalShort) + (size_t)GOAL_LIST * 4 + 64);
      jgoal.ensure((size_t)nj * sizeof(ulonglong2) + 16);
      GoalShort *gsd = bgoal.as<GoalShort>();
      ulonglong2 *jg = jgoal.as<ulonglong2>();
      {
        k_level_init<<<1, 256, 0, s>>>(gsd, nullptr, jg + jlo, jn);   // (no copies from pageable memory)
        nlaunch++;
        const unsigned gc = (unsigned)std::max<long long>(1, std::min<long long>((cm + 255) / 256, (long long)nsm * 8));
        k_goal_candidates_batch<<<gc, 256, 0, s>>>(fMeta.as<NodeMeta>(), fJob.as<uint32_t>(), dspecs.as<DevSpec>(),
                                                   ch.p0, ch.p1, (uint32_t *)(gsd + 1), gsd);
        k_goal_level_batch<NQ, ST><<<(unsigned)nsm * 2, EXP_WARPS * 32, 0, s>>>(
            dspecs.as<DevSpec>(), fJob.as<uint32_t>(), fR.as<Z4<ST>>(), fMeta.as<NodeMeta>(), (uint32_t *)(gsd + 1), gsd,
            jg);
        nlaunch += 2;
        ck(cudaGetLastError(), "goal pass");
      }
      GoalShort hgs{};
      std::vector<ulonglong2> hjg(jn);
      for (int attempt = 0; attempt < 2; attempt++) {
        tq.ensure(tqcap * sizeof(TQEntry));
        if (forms.packed && forms.general) tqleft.ensure(tqcap * 4);
        if (cap) {
          sH1.ensure(cap * 8); sH2.ensure(cap * 8); sIdx.ensure(cap * 8);
          sMeta.ensure(cap * sizeof(NodeMeta));
        }
        ck(cudaMemsetAsync(dst, 0, sizeof(DevStats), s), "memset");
        if (attempt) {                                   // the chunk's jobs start over (ids jlo..jhi)
          k_jst_init<<<(jn + 255) / 256, 256, 0, s>>>(jst.as<DevStats>() + jlo, jn);
          nlaunch++;
        }
        BatchArgs<ST> a;
        a.m = ch.p1; a.p0 = ch.p0;
        a.R = fR.as<Z4<ST>>(); a.meta = fMeta.as<NodeMeta>(); a.fjob = fJob.as<uint32_t>();
        a.specs = dspecs.as<DevSpec>(); a.jt = jt.as<int>(); a.jst = jst.as<DevStats>(); a.st = dst; a.cap = cap;
        a.sh1 = sH1.as<uint64_t>(); a.sh2 = sH2.as<uint64_t>(); a.sidx = sIdx.as<uint64_t>();
        a.smeta = sMeta.as<NodeMeta>();
        a.tq = tq.as<TQEntry>(); a.tqcap = tqcap;
        a.gshort = gsd; a.jgoal = jg;
        const long long want = (cm + EXP_WARPS - 1) / EXP_WARPS;
        const long long grid = std::max<long long>(1, std::min<long long>(want, (long long)nsm * tune.expand_blocks_per_sm));
        if (ch.jobs.size() == 1) {               // the plain level's two parts
          k_expand_solo<NQ, ST, 1><<<(unsigned)grid, EXP_WARPS * 32, 0, s>>>(J[jlo].sp, a, jlo);
          k_expand_solo<NQ, ST, 2><<<(unsigned)grid, EXP_WARPS * 32, 0, s>>>(J[jlo].sp, a, jlo);
          nlaunch++;
        } else {
          k_expand_batch<NQ, ST><<<(unsigned)grid, EXP_WARPS * 32, 0, s>>>(a);
        }
        TBoundArgs<ST> tb;
        tb.R = fR.as<Z4<ST>>(); tb.meta = fMeta.as<NodeMeta>(); tb.tq = tq.as<TQEntry>(); tb.tqcap = tqcap;
        tb.GS = BATCH_GS; tb.rem = 0; tb.keep = 0; tb.fjob = fJob.as<uint32_t>(); tb.specs = dspecs.as<DevSpec>();
        tb.jt = jt.as<int>(); tb.jst = jst.as<DevStats>(); tb.st = dst; tb.cap = cap; tb.sh1 = sH1.as<uint64_t>();
        tb.sh2 = sH2.as<uint64_t>(); tb.sidx = sIdx.as<uint64_t>(); tb.smeta = sMeta.as<NodeMeta>();
        const unsigned tgrid = (unsigned)(nsm * tune.tbound_blocks_per_sm);
        int ntb;
        if (ch.jobs.size() == 1) {               // one job: the plain kernel, its spec a parameter (its tallies go
          const Job &jj = J[jlo];                 // to the chunk's block and are added to the job's below)
          tb.fjob = nullptr; tb.specs = nullptr; tb.jt = nullptr; tb.jst = nullptr;
          tb.rem = jj.sp.depth - jj.t; tb.keep = jj.t < jj.sp.depth;
          ntb = launch_tbound<NQ, ST, false>(jj.sp, tb, forms.general ? tqleft.as<uint32_t>() : nullptr, forms, tgrid, s);
        } else {
          ntb = launch_tbound<NQ, ST, true>(DevSpec{}, tb, forms.general ? tqleft.as<uint32_t>() : nullptr, forms, tgrid, s);
        }
        nlaunch += 1 + ntb;
        ck(cudaGetLastError(), "batched expand");
        // the chunk's counters, the jobs' statistics and the goal pass's results, read back with one wait
        ck(cudaMemcpyAsync(&h, dst, sizeof(DevStats), cudaMemcpyDeviceToHost, s), "d2h");
        ck(cudaMemcpyAsync(hj.data() + jlo, jst.as<DevStats>() + jlo, jn * sizeof(DevStats), cudaMemcpyDeviceToHost, s),
           "d2h");
        ck(cudaMemcpyAsync(&hgs, gsd, sizeof hgs, cudaMemcpyDeviceToHost, s), "d2h");
        ck(cudaMemcpyAsync(hjg.data(), jg + jlo, jn * sizeof(ulonglong2), cudaMemcpyDeviceToHost, s), "d2h");
        ck(cudaStreamSynchronize(s), "batched expand");
        if (!h.surv_overflow && h.n_tq <= tqcap) break;
        cap = std::max<unsigned long long>(cap, h.n_surv);  // every survivor and entry was counted: exact room
        tqcap = std::max<unsigned long long>(tqcap, h.n_tq);
      }
      if (h.surv_overflow || h.n_tq > tqcap) throw std::runtime_error("survivor or T queue overflow");
      if (h.n_left && !forms.general) throw std::logic_error("T bounds left over");
      if (ch.jobs.size() == 1) {                 // the one-job T kernel's tallies, kept in the chunk's block
        DevStats &d = hj[jlo];
        d.dead += h.dead; d.alive += h.alive; d.t_evals += h.t_evals;
        if (h.ovf) d.ovf = 1;
      }
      if (!hgs.ovf && hgs.count <= GOAL_LIST)            // jobs found by the goal pass (their level kernels skipped)
        for (int i : ch.jobs)
          if (hjg[i - jlo].x) { hj[i].found = hjg[i - jlo].x; hj[i].first_found = hjg[i - jlo].y; }
      std::vector<int> found_ids;
      size_t nsort = 0;
      for (int i : ch.jobs) {
        Job &j = J[i];
        if (hj[i].ovf) { overflow_ids.push_back(i); continue; }
        if (hj[i].found) { found_ids.push_back(i); continue; }
        act[i] = 1;
        if (j.t < j.depth) nsort += hj[i].alive;
      }
      if (!found_ids.empty()) walk(found_ids, hj);
      if (!nsort) continue;
      // dedupe of the chunk's running jobs' survivors
      std::vector<uint8_t> cact(nj, 0);
      for (int i : ch.jobs) cact[i] = act[i];
      ck(cudaMemcpyAsync(jact.p, cact.data(), nj, cudaMemcpyHostToDevice, s), "h2d");
      const size_t ns = (size_t)h.n_surv;
      k0.ensure(nsort * 8); k1.ensure(nsort * 8); v0.ensure(nsort * 4); v1.ensure(nsort * 4);
      kidx.ensure(nsort * 8); kslot.ensure(nsort * 4); work.ensure(nsort * sizeof(uint2)); tmp.ensure(nsort * 4);
      hist.ensure(sort_hist_words(nsort) * 4);
      part.ensure(scan_partials_words(sort_hist_words(nsort)) * 4);
      SortScratch sc{hist.as<uint32_t>(), part.as<uint32_t>(), hist.cap / 4, part.cap / 4};
      ck(cudaMemsetAsync(cnt.p, 0, 8, s), "memset");
      const unsigned gb = (unsigned)std::max<size_t>(1, std::min<size_t>((ns + 255) / 256, (size_t)nsm * 16));
      k_bsort_init<<<gb, 256, 0, s>>>(sH1.as<uint64_t>(), sIdx.as<uint64_t>(), ns, fJob.as<uint32_t>(),
                                      jact.as<uint8_t>(), k0.as<uint64_t>(), v0.as<uint32_t>(),
                                      cnt.as<unsigned long long>());
      nlaunch++;
      int ln = 0;
      const bool f = radix_sort(k0.as<uint64_t>(), v0.as<uint32_t>(), k1.as<uint64_t>(), v1.as<uint32_t>(), nsort, 32,
                                64, sc, s, &ln);
      nlaunch += ln;
      const uint64_t *sk = f ? k1.as<uint64_t>() : k0.as<uint64_t>();
      const uint32_t *sv = f ? v1.as<uint32_t>() : v0.as<uint32_t>();
      ck(cudaMemsetAsync(dst, 0, sizeof(DevStats), s), "memset");
      const unsigned gs = (unsigned)std::max<size_t>(1, std::min<size_t>((nsort + 255) / 256, (size_t)nsm * 16));
      k_runs<<<gs, 256, 0, s>>>(sk, sv, nsort, sIdx.as<uint64_t>(), kidx.as<uint64_t>(), kslot.as<uint32_t>(),
                                work.as<uint2>(), dst);
      // a one-job chunk passes its job's spec as the kernels' parameter (a shared copy, as in the plain level)
      const bool one = ch.jobs.size() == 1;
      const DevSpec one_sp = one ? J[jlo].sp : DevSpec{};
      k_resolve<NQ, ST><<<(unsigned)nsm * 8, RES_WARPS * 32, 0, s>>>(
          one_sp, one ? nullptr : dspecs.as<DevSpec>(), one ? nullptr : fJob.as<uint32_t>(), BATCH_GS, fR.as<Z4<ST>>(),
          fMeta.as<NodeMeta>(),
          work.as<uint2>(), sv, sH1.as<uint64_t>(), sH2.as<uint64_t>(), sIdx.as<uint64_t>(), sMeta.as<NodeMeta>(),
          tmp.as<uint32_t>(), kidx.as<uint64_t>(), kslot.as<uint32_t>(), dst);
      nlaunch += 2;
      ck(cudaGetLastError(), "batched dedupe");
      ck(cudaMemcpyAsync(&h, dst, sizeof(DevStats), cudaMemcpyDeviceToHost, s), "d2h");
      ck(cudaStreamSynchronize(s), "batched dedupe");
      const size_t distinct = (size_t)h.n_kept;
      ck(cudaMemsetAsync(jdist.p, 0, nj * 8, s), "memset");
      k_bcount<<<(unsigned)std::max<size_t>(1, std::min<size_t>((distinct + 255) / 256, (size_t)nsm * 16)), 256, 0, s>>>(
          kidx.as<uint64_t>(), distinct, fJob.as<uint32_t>(), jdist.as<unsigned long long>());
      nlaunch++;
      std::vector<unsigned long long> cd(nj, 0);
      ck(cudaMemcpyAsync(cd.data(), jdist.p, nj * 8, cudaMemcpyDeviceToHost, s), "d2h");
      // the chunk's distinct children in child-index order, appended to the next frontier and this step's tree
      int bits = 1;
      while (bits < 64 && ((unsigned long long)ch.p1 * BATCH_GS) >> bits) bits++;
      const int hi = ((bits + 7) / 8) * 8;
      ln = 0;
      const bool f2 = radix_sort(kidx.as<uint64_t>(), kslot.as<uint32_t>(), k1.as<uint64_t>(), v1.as<uint32_t>(),
                                 distinct, 0, hi, sc, s, &ln);
      nlaunch += ln;
      const uint64_t *ki = f2 ? k1.as<uint64_t>() : kidx.as<uint64_t>();
      const uint32_t *vi = f2 ? v1.as<uint32_t>() : kslot.as<uint32_t>();
      const size_t o0 = total_distinct, o1 = total_distinct + distinct;
      grow_keep(tpar[nstep], o1 * 4 + 4, o0 * 4);
      grow_keep(tgat[nstep], o1 + 4, o0);
      grow_keep(fR2, o1 * E * sizeof(Z4<ST>) + 16, o0 * E * sizeof(Z4<ST>));
      grow_keep(fMeta2, o1 * sizeof(NodeMeta) + 16, o0 * sizeof(NodeMeta));
      grow_keep(fJob2, o1 * 4 + 4, o0 * 4);
      const unsigned gg = (unsigned)std::max<size_t>(1, std::min<size_t>((distinct + RES_WARPS - 1) / RES_WARPS,
                                                                         (size_t)nsm * 16));
      k_materialize<NQ, ST><<<gg, RES_WARPS * 32, 0, s>>>(
          one_sp, one ? nullptr : dspecs.as<DevSpec>(), fJob.as<uint32_t>(), BATCH_GS, fR.as<Z4<ST>>(), fMeta.as<NodeMeta>(), ki, vi,
          distinct, sMeta.as<NodeMeta>(), fR2.as<Z4<ST>>() + o0 * E, fMeta2.as<NodeMeta>() + o0,
          tpar[nstep].as<uint32_t>() + o0, tgat[nstep].as<uint8_t>() + o0, fJob2.as<uint32_t>() + o0);
      nlaunch++;
      ck(cudaGetLastError(), "batched gather");   // the next chunk's work queues behind the gather (no wait here)
      for (int i : ch.jobs) dist[i] = cd[i];
      total_distinct = o1;
    }
    ck(cudaStreamSynchronize(s), "batched gather");
    std::swap(fR, fR2); std::swap(fMeta, fMeta2); std::swap(fJob, fJob2);
    // level lines of the running jobs
    const double secs = now_s() - t0;
    for (int i = 0; i < nj; i++) {
      Job &j = J[i];
      if (!j.running || !act[i]) continue;
      const DevStats &d = hj[i];
      LevelStats L;
      L.t = j.t; L.parents = j.seg; L.prefixes = j.seg * j.hs.G - (long long)d.w2; L.cut_w3 = (long long)d.w3;
      L.cut_lb = (long long)d.dead; L.survivors = (long long)d.alive;
      L.distinct = j.t < j.depth ? (long long)dist[i] : 0;
      L.proved_unsat = L.distinct == 0;
      L.seconds = secs;
      if (j.seg * j.hs.G > 0) j.rate = (double)d.alive / ((double)j.seg * j.hs.G);
      if (d.alive > 0 && j.t < j.depth) j.drate = std::min(1.0, (double)dist[i] / (double)d.alive);
      j.out.levels.push_back(L);
      j.out.res.prefixes += L.prefixes;
      account(j, d);
      j.out.res.levels = j.t;
      if (L.distinct == 0) { j.seg = 0; finish(j, RC_PROOF); continue; }
      j.seg = L.distinct;
      j.t++;
    }
    m = (long long)total_distinct;
    nstep++;
    // jobs whose int32 limbs overflowed: rerun alone (the plain path promotes them to int64)
    for (int id : overflow_ids) {
      Job &j = J[id];
      if (j.running) nrun--;
      j.running = false;
      j.seg = 0;
      run_plain(j);
    }
    // tree levels older than every running job's first step: no walk reads them again; their buffers go to the
  // spare lists (freeing device memory synchronises the device and can take milliseconds)
    long long oldest = nstep;
    for (const Job &j : J) if (j.running) oldest = std::min<long long>(oldest, j.out.joined_step);
    for (; tree_lo < oldest && tree_lo < (long long)tpar.size(); tree_lo++) {
      if (!tpar[tree_lo].p) continue;
      spare_par.push_back(tpar[tree_lo]); spare_gat.push_back(tgat[tree_lo]);
      tpar[tree_lo] = DBuf(); tgat[tree_lo] = DBuf();
    }
    return running();
  }

  // circuits of the jobs that found the goal at this step: one thread per job walks the tree back
  void walk(const std::vector<int> &found_ids, const std::vector<DevStats> &hj) {
    const int nf = (int)found_ids.size();
    std::vector<unsigned long long> fo(nf);
    std::vector<int> ft(nf), fs(nf), fs0(nf);
    for (int i = 0; i < nf; i++) {
      fo[i] = hj[found_ids[i]].first_found; ft[i] = J[found_ids[i]].t; fs[i] = (int)nstep;
      fs0[i] = J[found_ids[i]].out.joined_step;
    }
    std::vector<const uint32_t *> pp(nstep + 1, nullptr);
    std::vector<const uint8_t *> gp(nstep + 1, nullptr);
    for (long long st2 = 0; st2 < nstep && st2 < (long long)tpar.size(); st2++) { pp[st2] = tpar[st2].as<uint32_t>(); gp[st2] = tgat[st2].as<uint8_t>(); }
    const size_t pb = pp.size() * sizeof(void *);
    tptr.ensure(2 * pb + (size_t)nf * (8 + 4 + 4 + 4) + (size_t)nf * MAXDEPTH_WALK * 4 + 64);
    char *base = (char *)tptr.p;
    ck(cudaMemcpyAsync(base, pp.data(), pb, cudaMemcpyHostToDevice, s), "h2d");
    ck(cudaMemcpyAsync(base + pb, gp.data(), pb, cudaMemcpyHostToDevice, s), "h2d");
    char *q = base + 2 * pb;
    unsigned long long *dfo = (unsigned long long *)q; q += (size_t)nf * 8;
    int *dft = (int *)q; q += (size_t)nf * 4;
    int *dfs = (int *)q; q += (size_t)nf * 4;
    int *dfs0 = (int *)q; q += (size_t)nf * 4;
    int *dout = (int *)q;
    ck(cudaMemcpyAsync(dfo, fo.data(), nf * 8, cudaMemcpyHostToDevice, s), "h2d");
    ck(cudaMemcpyAsync(dft, ft.data(), nf * 4, cudaMemcpyHostToDevice, s), "h2d");
    ck(cudaMemcpyAsync(dfs, fs.data(), nf * 4, cudaMemcpyHostToDevice, s), "h2d");
    ck(cudaMemcpyAsync(dfs0, fs0.data(), nf * 4, cudaMemcpyHostToDevice, s), "h2d");
    ck(cudaMemsetAsync(cnt.p, 0, 4, s), "memset");
    k_walk<<<(nf + 63) / 64, 64, 0, s>>>(dfo, dft, dfs, dfs0, nf, (const uint32_t *const *)base,
                                         (const uint8_t *const *)(base + pb), dout, cnt.as<int>());
    nlaunch++;
    std::vector<int> circ((size_t)nf * MAXDEPTH_WALK);
    int bad = 0;
    ck(cudaMemcpyAsync(circ.data(), dout, circ.size() * 4, cudaMemcpyDeviceToHost, s), "d2h");
    ck(cudaMemcpyAsync(&bad, cnt.p, 4, cudaMemcpyDeviceToHost, s), "d2h");
    ck(cudaStreamSynchronize(s), "walk");
    if (bad) throw std::logic_error("batch tree walk ended early");
    for (int i = 0; i < nf; i++) {
      Job &j = J[found_ids[i]];
      j.out.res.circuit.assign(circ.begin() + (size_t)i * MAXDEPTH_WALK, circ.begin() + (size_t)i * MAXDEPTH_WALK + j.t);
      j.out.res.n_found = (long long)hj[found_ids[i]].found;
      j.out.res.levels = j.t;
      account(j, hj[found_ids[i]]);
      j.seg = 0;
      finish(j, RC_CIRCUIT);
    }
  }
  void account(Job &j, const DevStats &d) {
    j.out.res.t_evals += (long long)d.t_evals;
    j.out.res.children += (long long)d.children;
    j.out.res.children_full += (long long)d.full;
  }
};

}  // namespace

BatchSession::BatchSession(Engine &engine, int nq) {
  switch (nq) {
    case 1: impl_ = new BatchImpl<1>(engine); break;
    case 2: impl_ = new BatchImpl<2>(engine); break;
    case 3: impl_ = new BatchImpl<3>(engine); break;
    default: throw std::invalid_argument("qubit count must be 1, 2 or 3");
  }
}
BatchSession::~BatchSession() { delete impl_; }
int BatchSession::nq() const { return impl_->nq(); }
int BatchSession::submit(const HostSpec &hs, const Options &opt) { return impl_->submit(hs, opt); }
int BatchSession::step() { return impl_->step(); }
int BatchSession::running() const { return impl_->running(); }
const BatchJob &BatchSession::job(int id) const { return impl_->job(id); }
int BatchSession::jobs() const { return impl_->jobs(); }
long long BatchSession::frontier() const { return impl_->frontier(); }
long long BatchSession::launches() const { return impl_->launches(); }
long long BatchSession::steps() const { return impl_->steps(); }
size_t BatchSession::device_bytes() const { return impl_->device_bytes(); }
size_t BatchSession::projected_bytes() const { return impl_->projected_bytes(); }
void BatchSession::set_memory_budget(size_t bytes) { impl_->set_budget(bytes); }
void BatchSession::set_tuning(const BatchTuning &t) { impl_->tune = t; }
BatchTuning BatchSession::tuning() const { return impl_->tune; }

BatchTuning autotune_batch(Engine &engine, int nq, const std::vector<const HostSpec *> &probe, const Options &opt,
                           std::vector<TuneTrial> *trials) {
  // the search space, committed here: chunk budget (bytes of survivor records per chunk of jobs), expand blocks per
  // SM, deferred-T blocks per SM; the defaults first in each list
  static const size_t chunk_space[] = {(size_t)8 << 30, (size_t)1 << 30, (size_t)2 << 30, (size_t)4 << 30};
  static const int expand_space[] = {16, 4, 8, 32};
  static const int tbound_space[] = {4, 1, 2, 8};
  // every trial on one session, so that all of them run with its buffers already grown and its spec tables on the
  // device (the probe jobs are submitted again for each trial)
  BatchSession b(engine, nq);
  auto run = [&](const BatchTuning &t) {
    b.set_tuning(t);
    const double t0 = now_s();
    for (const HostSpec *hs : probe) b.submit(*hs, opt);
    while (b.step() > 0) {}
    const double sec = now_s() - t0;
    if (trials) trials->push_back({t, sec});
    return sec;
  };
  BatchTuning best;
  run(best);                                      // warm-up
  if (trials) trials->clear();
  double best_s = run(best);
  for (int dim = 0; dim < 3; dim++) {
    for (int i = 1; i < 4; i++) {
      BatchTuning t = best;
      if (dim == 0) t.chunk_bytes = chunk_space[i];
      else if (dim == 1) t.expand_blocks_per_sm = expand_space[i];
      else t.tbound_blocks_per_sm = tbound_space[i];
      const double sec = run(t);
      if (sec < best_s) { best_s = sec; best = t; }
    }
  }
  return best;
}
long long BatchSession::waits() const { return impl_->waits(); }

}  // namespace cz
