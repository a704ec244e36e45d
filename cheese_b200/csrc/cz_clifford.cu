// sm_100a kernels and host loop of the Clifford-table path (the reference's src/clifford.cu, "cliffopt").
//
// Reference semantics: breadth-first search over the n-qubit Clifford group from the identity with generators
// H, S, Sdg, X, Z on every qubit and CX on every ordered pair (clifford.cu:148-166, 247-276), giving the minimal
// gate count of every element; a beam search over the placements K of every T gate, K Z_q' K^-1 = +-Z_q, with
// the cost of a partial placement the summed minimal lengths of the segments fixed so far (:168-201, 281-330);
// every segment read back as an optimal word by walking the distances down (:343-372).
//
// B200 design:
//  * the table is direct-addressed by a perfect rank of the group element (cz_tableau.h): a 92.9 MB byte array of
//    distances at n = 3 that stays in L2 while it is probed. No keys, no probing chains, and no element array: the
//    element of a rank is computed back from the rank (unrank) for candidate enumeration and uniform draws;
//  * BFS: one thread per symplectic part, whose reached sign vectors are one 64-bit mask (n = 3); a generator carries
//    the whole mask, its bits permuted by XOR with the signs it adds;
//  * beam step: dist(X) = dist(X^-1) (the generator set is closed under inverses), and X^-1 is the placement composed
//    with the inverse of the beam state's left part, a 4^n-entry row lookup table held in shared memory. The 4^n sign
//    vectors of a placement share one composition and one rank; rows of 4^n costs are screened by their least one, and
//    only the placements up to the beam's threshold are listed and sorted;
//  * read-back: one warp per segment, a lane per generator, ballot picks the first generator one step closer.
// Candidates are ordered by their tableau value (the reference leaves their order to an atomic counter).
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cctype>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <stdexcept>

#include "cz_buf.h"
#include "cz_clifford.h"
#include "cz_sort.cuh"
#include "cz_tableau.h"

namespace cz {

namespace {

constexpr int CL_T = 256;
constexpr int HB = 2048;            // cost histogram bins
constexpr int MAXBEAM = 255;
constexpr int WORDMAX = 32;         // longest optimal word read back (13 at n = 3)

struct GateSet {
  int ng;
  int8_t k[32], a[32], b[32];
};
GateSet gate_set(int n) {           // clifford.cu:148-153 order: per qubit h, s, sdg, x, z; then cx over ordered pairs
  GateSet g{};
  for (int q = 0; q < n; q++)
    for (int k : {CG_H, CG_S, CG_SDG, CG_X, CG_Z}) { g.k[g.ng] = (int8_t)k; g.a[g.ng] = (int8_t)q; g.b[g.ng] = 0; g.ng++; }
  for (int a = 0; a < n; a++)
    for (int b = 0; b < n; b++)
      if (a != b) { g.k[g.ng] = CG_CX; g.a[g.ng] = (int8_t)a; g.b[g.ng] = (int8_t)b; g.ng++; }
  return g;
}

// generator j of the n-qubit set in the order of gate_set, computed (no table): per qubit h, s, sdg, x, z, then
// cx over ordered pairs
template <int N>
struct Gen {
  static constexpr int NG = 5 * N + N * (N - 1);
  __host__ __device__ __forceinline__ static void get(int j, int &k, int &a, int &b) {
    if (j < 5 * N) { k = j % 5; a = j / 5; b = 0; return; }
    const int i = j - 5 * N, bb = N > 1 ? i % (N - 1) : 0;
    k = CG_CX;
    a = N > 1 ? i / (N - 1) : 0;
    b = bb + (bb >= a ? 1 : 0);
  }
};

struct ClCudaError : std::runtime_error { using std::runtime_error::runtime_error; };
void clk(cudaError_t e, const char *what) {
  if (e != cudaSuccess) {
    cudaGetLastError();            // a failed allocation must not be reported again by the next launch check
    throw ClCudaError(std::string("CUDA error after ") + what + ": " + cudaGetErrorString(e));
  }
}
double cl_now() { return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count(); }

struct ClMemory {
  static void *get(size_t n) {
    void *p = nullptr;
    clk(cudaMalloc(&p, n), "cudaMalloc");
    return p;
  }
  static void put(void *p) { clk(cudaFree(p), "free"); }
  static void drop(void *p) { cudaFree(p); }
};
using CBuf = GrowBuf<ClMemory>;

// ---------------- kernels ----------------
// The group is the symplectic parts S (1,451,520 at n = 3) times the 4^n sign vectors, and rank = 4^n rank(S) + signs.
// A generator maps (S, s) to (S', s ^ c) with c depending on S alone, so the elements of one S that a BFS level reached
// are one 4^n-bit mask, and a generator carries the whole mask at once: its bits permuted by XOR with c.
template <int N> struct Sym {
  static constexpr int NS = 1 << (2 * N);            // sign vectors
  static constexpr uint32_t ORDER = (uint32_t)(clifford_order(N) / NS);
};
// bit s of F moved to bit s ^ c
template <int N> __device__ __forceinline__ uint64_t xor_bits(uint64_t F, uint32_t c) {
  constexpr uint64_t M[6] = {0x5555555555555555ULL, 0x3333333333333333ULL, 0x0f0f0f0f0f0f0f0fULL,
                             0x00ff00ff00ff00ffULL, 0x0000ffff0000ffffULL, 0x00000000ffffffffULL};
#pragma unroll
  for (int b = 0; b < 2 * N; b++) {
    const uint64_t G = ((F & M[b]) << (1 << b)) | ((F >> (1 << b)) & M[b]);
    F = (c >> b) & 1u ? G : F;
  }
  return F;
}
template <int N> __device__ __forceinline__ uint32_t sign_vector(uint64_t X) {
  uint32_t c = 0;
#pragma unroll
  for (int i = 0; i < 2 * N; i++) c |= ((uint32_t)(X >> (i * Tb<N>::RB + Tb<N>::SB)) & 1u) << i;
  return c;
}
// the symplectic parts as tableaux without signs, by rank
template <int N> __global__ void k_cl_parts(uint64_t *part) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < Sym<N>::ORDER; i += gridDim.x * blockDim.x)
    part[i] = Tb<N>::unrank(i << (2 * N));
}
// one BFS level, one thread per symplectic part: the generators applied to its frontier mask, the images not seen yet
// added to the next masks. X and Z keep the part (no rank), S and Sdg share theirs: 12 ranks for 21 generators.
// Bound by issue (the ranks): the 14 levels take 3.0 ms, and 0.3 ms for k_cl_level; with one thread per group element
// (92.9 M elements, 21 ranks each) they took 68.2 ms.
template <int N>
__global__ void __launch_bounds__(CL_T) k_cl_bfs(const uint64_t *part, const uint64_t *front, const uint64_t *seen,
                                                 uint64_t *next, int *ovf) {
  using T = Tb<N>;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < Sym<N>::ORDER; i += gridDim.x * blockDim.x) {
    const uint64_t F = front[i];
    if (!F) continue;
    const uint64_t X = part[i];
    auto reach = [&](uint32_t r, uint32_t c) {
      const uint64_t m = xor_bits<N>(F, c) & ~seen[r];
      if (m) atomicOr((unsigned long long *)&next[r], (unsigned long long)m);
    };
    uint32_t rs = 0;
#pragma unroll
    for (int j = 0; j < Gen<N>::NG; j++) {
      int gk, ga, gb;
      Gen<N>::get(j, gk, ga, gb);
      const uint64_t C = T::gate(X, gk, ga, gb);
      const uint32_t c = sign_vector<N>(C);
      if (gk == CG_X || gk == CG_Z) { reach(i, c); continue; }
      if (gk != CG_SDG) {                            // (Sdg follows S on the same qubit)
        rs = T::rank(C);
        if (rs == T::BAD) { atomicOr(ovf, 2); continue; }
        rs >>= 2 * N;
      }
      if (rs < Sym<N>::ORDER) reach(rs, c);
    }
  }
}
// the level's end: the next masks become the frontier and are marked seen, their elements' distances written (a warp
// writes the rows of its 32 parts one after another, coalesced) and counted
template <int N>
__global__ void __launch_bounds__(CL_T) k_cl_level(uint64_t *front, uint64_t *seen, uint64_t *next, uint8_t *dist, uint8_t d,
                                                   unsigned long long *count) {
  constexpr int NS = Sym<N>::NS;
  __shared__ unsigned total;
  if (threadIdx.x == 0) total = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  unsigned mine = 0;
  for (uint32_t i0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; i0 < Sym<N>::ORDER; i0 += gridDim.x * blockDim.x) {
    const uint32_t i = i0 + lane;
    uint64_t m = 0;
    if (i < Sym<N>::ORDER) {
      m = next[i];
      front[i] = m;
      if (m) { next[i] = 0; seen[i] |= m; }
    }
    mine += (unsigned)__popcll(m);
    for (unsigned todo = __ballot_sync(0xffffffffu, m != 0); todo; todo &= todo - 1) {
      const int k = __ffs((int)todo) - 1;
      const uint64_t mk = __shfl_sync(0xffffffffu, m, k);
      for (int e = lane; e < NS; e += 32)
        if ((mk >> e) & 1) dist[(size_t)(i0 + k) * NS + e] = d;
    }
  }
  mine = __reduce_add_sync(0xffffffffu, mine);
  if (lane == 0 && mine) atomicAdd(&total, mine);
  __syncthreads();
  if (threadIdx.x == 0 && total) atomicAdd(count, (unsigned long long)total);
}

// placements of a T on qubit q: every K with K Z_q' K^-1 = +-Z_q for some q' (clifford.cu:170-183). The condition does
// not see K's signs, so the placements are kept as symplectic parts (as tableaux without signs), 4^n placements each.
template <int N> __device__ __forceinline__ int placed_qubit(uint64_t K, int q) {   // q', or -1
  int qp = -1;
  for (int i = 0; i < N; i++)
    if ((Tb<N>::row(K, N + i) & Tb<N>::SYM) == (1u << (N + q))) qp = i;
  return qp;
}
template <int N>
__global__ void k_cl_cands(const uint64_t *part, uint64_t *lists, uint32_t capq, uint32_t *cnt, int *ovf) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < Sym<N>::ORDER; i += gridDim.x * blockDim.x) {
    const uint64_t K = part[i];
    for (int q = 0; q < N; q++)
      if (placed_qubit<N>(K, q) >= 0) {
        const uint32_t pos = atomicAdd(&cnt[q], 1u);
        if (pos < capq) lists[(size_t)q * capq + pos] = K;
        else atomicOr(ovf, 1);
      }
  }
}
// per symplectic part the least distance over its sign vectors
template <int N> __global__ void k_cl_least(const uint8_t *dist, uint8_t *least) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < Sym<N>::ORDER; i += gridDim.x * blockDim.x) {
    uint32_t m = 0xffffffffu;
    const uint32_t *row = (const uint32_t *)(dist + (size_t)i * Sym<N>::NS);
#pragma unroll
    for (int w = 0; w < Sym<N>::NS / 4; w++) m = __vminu4(m, row[w]);
    m = __vminu4(m, m >> 16);
    least[i] = (uint8_t)min(m & 0xffu, (m >> 8) & 0xffu);
  }
}

// Beam step, first pass: one row per (state b, flip f, symplectic part g of the placements), the 4^n placements of the
// part. With K's sign vector s, the rank of the composed tableau is at ^ s: composition adds K's signs to the table's,
// and the flip (row X_q' times Z_q' times the T's sign, which cancels Z_q's) only adds a constant. So one composition and
// one rank serve 4^n evaluations; the row's least cost comes from the part's least distance. Row i = (b * 2 + f) * ng + g
// gets at[i] and rcost[i], and the least costs a histogram relative to cmin. A step with 16 states (2.2 M rows standing
// for 142 M placements) takes 65 us, and 15 us to list the kept ones; one rank per placement took 3.0 ms, and 0.4 ms to
// select.
constexpr int BADCOST = 999;        // of a placement outside the table (the reference's)
template <int N>
__global__ void __launch_bounds__(CL_T) k_cl_beam(const uint64_t *parts, uint32_t ng, int nb, int q, const uint8_t *tabs,
                                                  const int *bcost, int dagger, int cmin, const uint8_t *least,
                                                  uint32_t *at, uint16_t *rcost, unsigned *hist) {
  using T = Tb<N>;
  constexpr int TS = 1 << (2 * N);
  __shared__ uint8_t stab[MAXBEAM * TS];
  __shared__ int sbc[MAXBEAM];
  __shared__ unsigned sh[HB];
  for (int i = threadIdx.x; i < nb * TS; i += blockDim.x) stab[i] = tabs[i];
  for (int i = threadIdx.x; i < nb; i += blockDim.x) sbc[i] = bcost[i];
  for (int i = threadIdx.x; i < HB; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  const uint32_t rows = (uint32_t)nb * 2 * ng, stride = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < rows; i += stride) {
    const uint32_t g = i % ng, bf = i / ng;
    const int b = (int)(bf >> 1);
    uint64_t K = parts[g];
    if (bf & 1) {
      // the flipped placement's K o g^-1 (g = Sdg if the T is a dagger after the sign, else S): row X_qp -> +-Y_qp image
      const int qp = placed_qubit<N>(K, q);
      K = T::with_row(K, qp, T::image(K, 1u << qp, 1u << qp) ^ ((dagger ? 0u : 1u) << T::SB));
    }
    const uint32_t r = T::rank(T::compose_tab(K, stab + b * TS));
    const int v = sbc[b] + (r == T::BAD ? BADCOST : (int)least[r >> (2 * N)]);
    at[i] = r;
    rcost[i] = (uint16_t)v;
    atomicAdd(&sh[min(v - cmin, HB - 1)], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < HB; i += blockDim.x)
    if (sh[i]) atomicAdd(&hist[i], sh[i]);
}
// second pass: the placements of cost <= thr as keys cost - cmin | b | K | f, in the order the beam keeps them in (cost,
// then state, placement by tableau value, flip); *cnt counts all of them, the first cap are stored
template <int N> constexpr int KEY_BITS = Tb<N>::RB * Tb<N>::ROWS + 1;      // of (K, f)
template <int N>
__global__ void __launch_bounds__(CL_T) k_cl_emit(const uint64_t *parts, uint32_t ng, uint32_t rows, const int *bcost,
                                                  int cmin, int thr, const uint8_t *dist, const uint32_t *at,
                                                  const uint16_t *rcost, uint64_t *keys, unsigned long long cap,
                                                  unsigned long long *cnt) {
  using T = Tb<N>;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < rows; i += gridDim.x * blockDim.x) {
    if ((int)rcost[i] > thr) continue;
    const uint32_t g = i % ng, bf = i / ng, r = at[i];
    const int base = bcost[bf >> 1];
    for (uint32_t sv = 0; sv < (uint32_t)Sym<N>::NS; sv++) {
      const int v = base + (r == T::BAD ? BADCOST : (int)dist[r ^ sv]);
      if (v > thr) continue;
      uint64_t K = parts[g];
#pragma unroll
      for (int j = 0; j < 2 * N; j++) K |= (uint64_t)((sv >> j) & 1u) << (j * T::RB + T::SB);
      const unsigned long long pos = atomicAdd(cnt, 1ULL);
      if (pos < cap)
        keys[pos] = ((uint64_t)(v - cmin) << (KEY_BITS<N> + 8)) | ((uint64_t)(bf >> 1) << KEY_BITS<N>) | (K << 1) | (bf & 1);
    }
  }
}
// histogram of the costs >= base (bins relative to base)
__global__ void k_cl_hist(const uint16_t *cost, unsigned long long tot, int base, unsigned *hist) {
  __shared__ unsigned sh[HB];
  for (int i = threadIdx.x; i < HB; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < tot;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const int v = cost[i];
    if (v >= base) atomicAdd(&sh[min(v - base, HB - 1)], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < HB; i += blockDim.x)
    if (sh[i]) atomicAdd(&hist[i], sh[i]);
}

template <int N>
__global__ void k_cl_dist(const uint64_t *tab, size_t n, const uint8_t *dist, int *out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t r = Tb<N>::rank(tab[i]);
    out[i] = r == Tb<N>::BAD ? -1 : (dist[r] == 0xff ? -1 : (int)dist[r]);
  }
}
template <int N>
__global__ void k_cl_elem(const uint64_t *idx, size_t n, unsigned long long order, uint64_t *out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    out[i] = idx[i] < order ? Tb<N>::unrank((uint32_t)idx[i]) : 0;
}
// one warp per segment: the optimal word of X, generators indexed into gs (clifford.cu:352-371)
template <int N>
__global__ void k_cl_word(const uint64_t *X0, int nseg, const uint8_t *dist, int8_t *out, int *len) {
  using T = Tb<N>;
  const int w = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (w >= nseg) return;
  uint64_t X = X0[w];
  const uint32_t r0 = T::rank(X);
  int d = r0 == T::BAD || dist[r0] == 0xff ? -1 : (int)dist[r0];
  if (d < 0 || d > WORDMAX) { if (lane == 0) len[w] = -1; return; }
  if (lane == 0) len[w] = d;
  for (int pos = d - 1; pos >= 0; pos--) {
    uint64_t pre = 0;
    bool ok = false;
    if (lane < Gen<N>::NG) {
      int gk, ga, gb;
      Gen<N>::get(lane, gk, ga, gb);
      pre = T::gate(X, T::inverse_kind(gk), ga, gb);
      const uint32_t r = T::rank(pre);
      ok = r != T::BAD && dist[r] == pos;
    }
    const unsigned bal = __ballot_sync(0xffffffffu, ok);
    if (!bal) { if (lane == 0) len[w] = -2; return; }
    const int g = __ffs((int)bal) - 1;
    X = __shfl_sync(0xffffffffu, pre, g);
    if (lane == 0) out[w * WORDMAX + pos] = (int8_t)g;
  }
}

// host-side tableau ops at runtime n
uint64_t h_identity(int n) { return n == 1 ? Tb<1>::identity() : n == 2 ? Tb<2>::identity() : Tb<3>::identity(); }
uint64_t h_gate(int n, uint64_t T, int k, int a, int b) {
  return n == 1 ? Tb<1>::gate(T, k, a, b) : n == 2 ? Tb<2>::gate(T, k, a, b) : Tb<3>::gate(T, k, a, b);
}
uint64_t h_compose(int n, uint64_t A, uint64_t B) {
  return n == 1 ? Tb<1>::compose(A, B) : n == 2 ? Tb<2>::compose(A, B) : Tb<3>::compose(A, B);
}
uint64_t h_inverse(int n, uint64_t A) { return n == 1 ? Tb<1>::inverse(A) : n == 2 ? Tb<2>::inverse(A) : Tb<3>::inverse(A); }
void h_image_table(int n, uint64_t B, uint8_t *tab) {
  if (n == 1) Tb<1>::image_table(B, tab); else if (n == 2) Tb<2>::image_table(B, tab); else Tb<3>::image_table(B, tab);
}

}  // namespace

struct CTable {
  int n = 0;
  long long order = 0;
  CBuf dist, least;                          // by rank; per symplectic part
  CBuf cand[3];                              // per qubit: the symplectic parts of its placements
  uint32_t ncand[3] = {0, 0, 0};
  CliffTableInfo info;
  void release() { dist.release(); least.release(); for (CBuf &c : cand) c.release(); }
};

class CliffordContext {
 public:
  int dev;
  cudaStream_t s;
  int nsm = 148;
  std::map<int, CTable *> tables;
  CBuf ovf, cnt, at, cost, hist, keys, keys2, vals, vals2, shist, part, tabs, bc, pk, tmp, out, len;
  long long launches = 0;
  CliffordContext(int d, void *stream) : dev(d), s((cudaStream_t)stream) {
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  }
  ~CliffordContext() {
    cudaSetDevice(dev);
    for (auto &kv : tables) { kv.second->release(); delete kv.second; }
    for (CBuf *b : {&ovf, &cnt, &at, &cost, &hist, &keys, &keys2, &vals, &vals2, &shist, &part, &tabs, &bc, &pk, &tmp,
                    &out, &len})
      b->release();
  }
  size_t trim() {                              // work buffers back to the device; resident tables stay
    size_t n = 0;
    for (CBuf *b : {&cnt, &at, &cost, &hist, &keys, &keys2, &vals, &vals2, &shist, &part, &tabs, &bc, &pk, &tmp, &out,
                    &len}) {
      n += b->cap;
      b->release();
    }
    return n;
  }
  unsigned grid(unsigned long long n, int per = 8) const {
    return (unsigned)std::max<unsigned long long>(1, std::min<unsigned long long>((n + CL_T - 1) / CL_T,
                                                                                   (unsigned long long)nsm * per));
  }
  void sync(const char *what) { clk(cudaStreamSynchronize(s), what); }

  CTable *table(int n, CliffTableInfo &info);
  template <int N> void build(CTable &t);
  struct Placed { int b, f, cost; uint64_t K; int qp, neg; };   // a kept placement: state, flip, cost, K and its q', sign
  template <int N> std::vector<Placed> beam_step(CTable &t, int q, int dagger, const std::vector<uint64_t> &left,
                                                 const std::vector<int> &bcost, int beam);
  std::vector<int> dist_of(CTable &t, const std::vector<uint64_t> &x);
  void words(CTable &t, const std::vector<uint64_t> &x, std::vector<std::vector<int>> &w);
};

template <int N>
void CliffordContext::build(CTable &t) {
  using T = Tb<N>;
  const double t0 = cl_now();
  const unsigned long long order = (unsigned long long)clifford_order(N);
  t.n = N;
  t.order = (long long)order;
  t.dist.ensure(order);
  const size_t masks = (size_t)Sym<N>::ORDER * 8;
  CBuf part, seen, fa, fb;
  part.ensure(masks); seen.ensure(masks); fa.ensure(masks); fb.ensure(masks);
  ovf.ensure(4); cnt.ensure(64);
  clk(cudaMemsetAsync(t.dist.p, 0xff, order, s), "memset");
  for (CBuf *m : {&seen, &fa, &fb}) clk(cudaMemsetAsync(m->p, 0, masks, s), "memset");
  clk(cudaMemsetAsync(ovf.p, 0, 4, s), "memset");
  const uint32_t r0 = T::rank(T::identity());
  const uint8_t zero = 0;
  const uint64_t bit = 1ULL << (r0 & (Sym<N>::NS - 1));
  clk(cudaMemcpyAsync(t.dist.as<uint8_t>() + r0, &zero, 1, cudaMemcpyHostToDevice, s), "h2d");
  clk(cudaMemcpyAsync(seen.as<uint64_t>() + (r0 >> (2 * N)), &bit, 8, cudaMemcpyHostToDevice, s), "h2d");
  clk(cudaMemcpyAsync(fa.as<uint64_t>() + (r0 >> (2 * N)), &bit, 8, cudaMemcpyHostToDevice, s), "h2d");
  const unsigned gp = grid(Sym<N>::ORDER, 16);
  k_cl_parts<N><<<gp, CL_T, 0, s>>>(part.as<uint64_t>());
  launches++;
  CliffTableInfo &inf = t.info;
  inf = CliffTableInfo{};
  inf.n = N;
  inf.order = (long long)order;
  unsigned long long nf = 1, total = 1;
  for (int d = 1; nf; d++) {
    clk(cudaMemsetAsync(cnt.p, 0, 8, s), "memset");
    k_cl_bfs<N><<<gp, CL_T, 0, s>>>(part.as<uint64_t>(), fa.as<uint64_t>(), seen.as<uint64_t>(), fb.as<uint64_t>(),
                                    ovf.as<int>());
    k_cl_level<N><<<gp, CL_T, 0, s>>>(fa.as<uint64_t>(), seen.as<uint64_t>(), fb.as<uint64_t>(), t.dist.as<uint8_t>(),
                                      (uint8_t)d, cnt.as<unsigned long long>());
    launches += 2;
    clk(cudaGetLastError(), "bfs");
    unsigned long long nn = 0;
    int of = 0;
    clk(cudaMemcpyAsync(&nn, cnt.p, 8, cudaMemcpyDeviceToHost, s), "d2h");
    clk(cudaMemcpyAsync(&of, ovf.p, 4, cudaMemcpyDeviceToHost, s), "d2h");
    sync("bfs");
    if (of) throw std::overflow_error("invalid tableau in the BFS");
    nf = nn;
    total += nf;
    if (nf) { if (d < 32) inf.per_distance[d] = (long long)nf; inf.max_distance = d; }
  }
  inf.per_distance[0] = 1;
  inf.elements = (long long)total;
  for (CBuf *m : {&seen, &fa, &fb}) m->release();
  if (total != order) { part.release(); throw std::logic_error("group order mismatch"); }
  t.least.ensure(Sym<N>::ORDER);
  k_cl_least<N><<<gp, CL_T, 0, s>>>(t.dist.as<uint8_t>(), t.least.as<uint8_t>());
  // the placements' parts per qubit: Z_q comes from one of n rows, each with one of 4^n - 1 images
  const uint32_t capq = Sym<N>::ORDER / ((1u << (2 * N)) - 1) * N;
  CBuf lists;
  lists.ensure((size_t)capq * N * 8);
  clk(cudaMemsetAsync(cnt.p, 0, 64, s), "memset");
  k_cl_cands<N><<<gp, CL_T, 0, s>>>(part.as<uint64_t>(), lists.as<uint64_t>(), capq, cnt.as<uint32_t>(), ovf.as<int>());
  launches += 2;
  clk(cudaGetLastError(), "candidates");
  int of = 0;
  clk(cudaMemcpyAsync(t.ncand, cnt.p, 12, cudaMemcpyDeviceToHost, s), "d2h");
  clk(cudaMemcpyAsync(&of, ovf.p, 4, cudaMemcpyDeviceToHost, s), "d2h");
  sync("candidates");
  part.release();
  if (of) { lists.release(); throw std::overflow_error("candidate buffer too small"); }
  for (int q = 0; q < N; q++) {
    t.cand[q].ensure((size_t)t.ncand[q] * 8 + 8);
    clk(cudaMemcpyAsync(t.cand[q].p, lists.as<uint64_t>() + (size_t)q * capq, (size_t)t.ncand[q] * 8,
                        cudaMemcpyDeviceToDevice, s), "d2d");
  }
  sync("candidates");
  lists.release();
  inf.built = true;
  inf.seconds = cl_now() - t0;
}

CTable *CliffordContext::table(int n, CliffTableInfo &info) {
  auto it = tables.find(n);
  if (it != tables.end()) {
    info = it->second->info;
    info.built = false;
    info.seconds = 0;
    return it->second;
  }
  clk(cudaSetDevice(dev), "cudaSetDevice");
  CTable *t = new CTable;
  try {
    if (n == 1) build<1>(*t); else if (n == 2) build<2>(*t); else build<3>(*t);
  } catch (...) {
    t->release();
    delete t;
    throw;
  }
  tables[n] = t;
  info = t->info;
  return t;
}

std::vector<int> CliffordContext::dist_of(CTable &t, const std::vector<uint64_t> &x) {
  std::vector<int> r(x.size());
  if (x.empty()) return r;
  tmp.ensure(x.size() * 8); out.ensure(x.size() * 4);
  clk(cudaMemcpyAsync(tmp.p, x.data(), x.size() * 8, cudaMemcpyHostToDevice, s), "h2d");
  if (t.n == 1) k_cl_dist<1><<<grid(x.size()), CL_T, 0, s>>>(tmp.as<uint64_t>(), x.size(), t.dist.as<uint8_t>(), out.as<int>());
  else if (t.n == 2) k_cl_dist<2><<<grid(x.size()), CL_T, 0, s>>>(tmp.as<uint64_t>(), x.size(), t.dist.as<uint8_t>(), out.as<int>());
  else k_cl_dist<3><<<grid(x.size()), CL_T, 0, s>>>(tmp.as<uint64_t>(), x.size(), t.dist.as<uint8_t>(), out.as<int>());
  launches++;
  clk(cudaGetLastError(), "dist");
  clk(cudaMemcpyAsync(r.data(), out.p, x.size() * 4, cudaMemcpyDeviceToHost, s), "d2h");
  sync("dist");
  return r;
}

void CliffordContext::words(CTable &t, const std::vector<uint64_t> &x, std::vector<std::vector<int>> &w) {
  const int m = (int)x.size();
  w.assign(m, {});
  if (!m) return;
  tmp.ensure(m * 8); out.ensure((size_t)m * WORDMAX); len.ensure(m * 4);
  clk(cudaMemcpyAsync(tmp.p, x.data(), m * 8, cudaMemcpyHostToDevice, s), "h2d");
  const unsigned blocks = (unsigned)((m * 32 + CL_T - 1) / CL_T);
  if (t.n == 1) k_cl_word<1><<<blocks, CL_T, 0, s>>>(tmp.as<uint64_t>(), m, t.dist.as<uint8_t>(), out.as<int8_t>(), len.as<int>());
  else if (t.n == 2) k_cl_word<2><<<blocks, CL_T, 0, s>>>(tmp.as<uint64_t>(), m, t.dist.as<uint8_t>(), out.as<int8_t>(), len.as<int>());
  else k_cl_word<3><<<blocks, CL_T, 0, s>>>(tmp.as<uint64_t>(), m, t.dist.as<uint8_t>(), out.as<int8_t>(), len.as<int>());
  launches++;
  clk(cudaGetLastError(), "read-back");
  std::vector<int8_t> ho((size_t)m * WORDMAX);
  std::vector<int> hl(m);
  clk(cudaMemcpyAsync(ho.data(), out.p, ho.size(), cudaMemcpyDeviceToHost, s), "d2h");
  clk(cudaMemcpyAsync(hl.data(), len.p, m * 4, cudaMemcpyDeviceToHost, s), "d2h");
  sync("read-back");
  for (int i = 0; i < m; i++) {
    if (hl[i] == -1) throw std::logic_error("segment not in the table");
    if (hl[i] < 0) throw std::logic_error("path reconstruction failed");
    for (int j = 0; j < hl[i]; j++) w[i].push_back(ho[(size_t)i * WORDMAX + j]);
  }
}

// one beam step over the placements of a T gate on qubit q: the kept ones, by (cost, state, placement, flip)
template <int N>
std::vector<CliffordContext::Placed> CliffordContext::beam_step(CTable &t, int q, int dagger, const std::vector<uint64_t> &left,
                                                                const std::vector<int> &bcost, int beam) {
  using T = Tb<N>;
  constexpr int TS = 1 << (2 * N);
  const int nb = (int)left.size();
  const uint32_t ng = t.ncand[q], rows = (uint32_t)nb * 2 * ng;
  std::vector<uint8_t> ht((size_t)nb * TS);
  for (int b = 0; b < nb; b++) T::image_table(T::inverse(left[b]), ht.data() + (size_t)b * TS);
  int cmin = 1 << 30, cmax = 0;
  for (int v : bcost) { cmin = std::min(cmin, v); cmax = std::max(cmax, v); }
  if (cmax + BADCOST > 65535) throw std::range_error("beam cost out of range");
  tabs.ensure(ht.size()); bc.ensure(nb * 4); hist.ensure(HB * 4); cost.ensure((size_t)rows * 2 + 2); at.ensure((size_t)rows * 4 + 4);
  cnt.ensure(64);
  clk(cudaMemcpyAsync(tabs.p, ht.data(), ht.size(), cudaMemcpyHostToDevice, s), "h2d");
  clk(cudaMemcpyAsync(bc.p, bcost.data(), nb * 4, cudaMemcpyHostToDevice, s), "h2d");
  clk(cudaMemsetAsync(hist.p, 0, HB * 4, s), "memset");
  k_cl_beam<N><<<grid(rows, 16), CL_T, 0, s>>>(t.cand[q].as<uint64_t>(), ng, nb, q, tabs.as<uint8_t>(), bc.as<int>(), dagger,
                                                cmin, t.least.as<uint8_t>(), at.as<uint32_t>(), cost.as<uint16_t>(),
                                                hist.as<unsigned>());
  launches++;
  clk(cudaGetLastError(), "beam step");
  // a threshold with at least `keep` placements at or below it: the cost of the keep-th smallest row's best (every row
  // has a placement of its least cost), or every row when there are fewer
  const unsigned long long keep = std::min<unsigned long long>((unsigned long long)beam, (unsigned long long)rows * Sym<N>::NS);
  const unsigned long long krows = std::min<unsigned long long>(keep, rows);
  unsigned long long nlow = 0;
  int base = cmin, thr = -1;
  std::vector<unsigned> hh(HB);
  for (;;) {
    clk(cudaMemcpyAsync(hh.data(), hist.p, HB * 4, cudaMemcpyDeviceToHost, s), "d2h");
    sync("histogram");
    unsigned long long cum = nlow;
    int k = 0;
    for (; k < HB - 1; k++) {
      if (cum + hh[k] >= krows) break;
      cum += hh[k];
    }
    if (k < HB - 1) { thr = base + k; break; }
    nlow = cum;                      // everything below base + HB - 1 is kept: zoom into the overflow bin
    base += HB - 1;
    clk(cudaMemsetAsync(hist.p, 0, HB * 4, s), "memset");
    k_cl_hist<<<grid(rows, 16), CL_T, 0, s>>>(cost.as<uint16_t>(), rows, base, hist.as<unsigned>());
    launches++;
  }
  if (keep > krows) thr = cmax + BADCOST;            // fewer rows than the beam keeps: all their placements
  // every placement up to the threshold (few: the tail of the costs is thin), sorted; a second round when they are more
  // than the room
  int kb = 0;
  while ((thr - cmin) >> kb) kb++;
  const int bits = KEY_BITS<N> + 8 + kb;
  if (bits > 64) throw std::range_error("beam cost out of range");
  unsigned long long room = std::max<unsigned long long>(keys.cap / 8, 1ULL << 16), m = 0;
  for (;;) {
    keys.ensure(room * 8);
    room = keys.cap / 8;
    clk(cudaMemsetAsync(cnt.p, 0, 8, s), "memset");
    k_cl_emit<N><<<grid(rows, 16), CL_T, 0, s>>>(t.cand[q].as<uint64_t>(), ng, rows, bc.as<int>(), cmin, thr,
                                                 t.dist.as<uint8_t>(), at.as<uint32_t>(), cost.as<uint16_t>(),
                                                 keys.as<uint64_t>(), room, cnt.as<unsigned long long>());
    launches++;
    clk(cudaGetLastError(), "beam placements");
    clk(cudaMemcpyAsync(&m, cnt.p, 8, cudaMemcpyDeviceToHost, s), "d2h");
    sync("beam placements");
    if (m <= room) break;
    room = m;
  }
  if (m < keep) throw std::logic_error("beam selection count mismatch");
  keys2.ensure(m * 8 + 8); vals.ensure(m * 4 + 4); vals2.ensure(m * 4 + 4);
  shist.ensure(sort_hist_words(m) * 4 + 4); part.ensure(scan_partials_words(sort_hist_words(m)) * 4 + 4);
  SortScratch sc{shist.as<uint32_t>(), part.as<uint32_t>(), shist.cap / 4, part.cap / 4};
  int ln = 0;
  const bool fl = radix_sort(keys.as<uint64_t>(), vals.as<uint32_t>(), keys2.as<uint64_t>(), vals2.as<uint32_t>(), (size_t)m, 0,
                             (bits + 7) / 8 * 8, sc, s, &ln);
  launches += ln;
  std::vector<uint64_t> hk(keep);
  clk(cudaMemcpyAsync(hk.data(), fl ? keys2.p : keys.p, keep * 8, cudaMemcpyDeviceToHost, s), "d2h");
  sync("beam selection");
  std::vector<Placed> out;
  for (uint64_t k : hk) {
    Placed p;
    p.f = (int)(k & 1);
    p.K = (k >> 1) & ((1ULL << (KEY_BITS<N> - 1)) - 1);
    p.b = (int)((k >> KEY_BITS<N>) & 0xff);
    p.cost = cmin + (int)(k >> (KEY_BITS<N> + 8));
    p.qp = p.neg = 0;
    for (int i = 0; i < N; i++) {
      const uint32_t w = T::row(p.K, N + i);
      if ((w & T::SYM) == (1u << (N + q))) { p.qp = i; p.neg = (int)(w >> T::SB); }
    }
    out.push_back(p);
  }
  return out;
}

// ---------------- jobs ----------------
int parse_cliff_job(const char *text, size_t len, CliffJob &J, std::string &err) {
  J = CliffJob{};
  const char *p = text, *end = text + len;
  auto tok = [&](std::string &o) {
    while (p < end && std::isspace((unsigned char)*p)) p++;
    if (p >= end) return false;
    const char *b = p;
    while (p < end && !std::isspace((unsigned char)*p)) p++;
    o.assign(b, p);
    return true;
  };
  bool bad = false;
  auto num = [&]() -> long {
    std::string t;
    if (bad || !tok(t)) { bad = true; return 0; }
    char *e;
    const long v = std::strtol(t.c_str(), &e, 10);
    if (e == t.c_str() || *e) bad = true;
    return v;
  };
  J.n = (int)num();
  const long t = num();
  if (bad || J.n < 1 || J.n > 3 || t < 0 || t > 1000000) { err = "bad job file"; return 2; }
  J.tq.resize(t); J.td.resize(t);
  for (long i = 0; i < t && !bad; i++) {
    J.tq[i] = (int)num(); J.td[i] = (int)num();
    if (J.tq[i] < 0 || J.tq[i] >= J.n || J.td[i] < 0 || J.td[i] > 1) bad = true;
  }
  J.seg.resize(t + 1);
  for (long j = 0; j <= t && !bad; j++) {
    const long m = num();
    if (m < 0 || m > 100000000) { bad = true; break; }
    for (long i = 0; i < m && !bad; i++) {
      std::string nm;
      if (!tok(nm)) { bad = true; break; }
      int k;
      if (nm == "h") k = CG_H; else if (nm == "s") k = CG_S; else if (nm == "sdg") k = CG_SDG;
      else if (nm == "x") k = CG_X; else if (nm == "z") k = CG_Z; else if (nm == "y") k = CG_Y;
      else if (nm == "cx") k = CG_CX;
      else { err = "unknown Clifford gate " + nm; return 2; }
      const int a = (int)num();
      const int b = k == CG_CX ? (int)num() : 0;
      if (a < 0 || a >= J.n || (k == CG_CX && (b < 0 || b >= J.n || b == a))) bad = true;
      J.seg[j].push_back(k); J.seg[j].push_back(a); J.seg[j].push_back(b);
    }
  }
  if (bad) { err = "bad job file"; return 2; }
  return 0;
}

CliffordContext *clifford_context_create(int device, void *stream) { return new CliffordContext(device, stream); }
void clifford_context_destroy(CliffordContext *c) { delete c; }
size_t clifford_context_trim(CliffordContext *c) {
  cudaSetDevice(c->dev);
  cudaStreamSynchronize(c->s);
  return c->trim();
}

int clifford_table(CliffordContext *c, int n, CliffTableInfo &info, std::string &err) {
  if (n < 1 || n > 3) { err = "n must be 1, 2 or 3"; return 3; }
  try {
    c->table(n, info);
    return 0;
  } catch (const std::logic_error &e) {
    err = e.what();
    return 4;
  } catch (const std::overflow_error &e) {
    err = e.what();
    return 4;
  } catch (const std::exception &e) {
    err = e.what();
    return 5;
  }
}

int cliffopt_run(CliffordContext *c, const CliffJob &J, int beam,
                 const std::function<void(int, const CliffStep &)> &on_step, CliffOptResult &res) {
  res = CliffOptResult{};
  const double t0 = cl_now();
  const long long l0 = c->launches;
  beam = std::max(1, std::min(MAXBEAM, beam));
  try {
    clk(cudaSetDevice(c->dev), "cudaSetDevice");
    const int n = J.n, t = (int)J.tq.size();
    CTable &tab = *c->table(n, res.table);
    std::vector<uint64_t> D(t + 1);
    for (int j = 0; j <= t; j++) {
      uint64_t X = h_identity(n);
      for (size_t i = 0; i < J.seg[j].size(); i += 3) X = h_gate(n, X, J.seg[j][i], J.seg[j][i + 1], J.seg[j][i + 2]);
      D[j] = X;
    }
    struct Pick { int parent, flip; uint64_t K; int qp, neg; };
    std::vector<std::vector<Pick>> hist(t);
    std::vector<uint64_t> Kprev{0};
    std::vector<int> bcost{0};
    for (int j = 0; j < t; j++) {
      const int q = J.tq[j];
      std::vector<uint64_t> left(Kprev.size());
      for (size_t b = 0; b < Kprev.size(); b++) left[b] = j == 0 ? D[j] : h_compose(n, Kprev[b], D[j]);
      const std::vector<CliffordContext::Placed> kept =
          n == 1 ? c->beam_step<1>(tab, q, J.td[j], left, bcost, beam)
                 : n == 2 ? c->beam_step<2>(tab, q, J.td[j], left, bcost, beam) : c->beam_step<3>(tab, q, J.td[j], left, bcost, beam);
      if (kept.empty()) throw std::logic_error("no placement candidates");
      Kprev.clear();
      bcost.clear();
      for (const auto &p : kept) {
        hist[j].push_back(Pick{p.b, p.f, p.K, p.qp, p.neg});
        Kprev.push_back(p.K);
        bcost.push_back(p.cost);
      }
      if (on_step) on_step(j, CliffStep{(long long)tab.ncand[q] << (2 * n), bcost[0]});
    }
    int best = 0;
    if (t > 0) {
      std::vector<uint64_t> fin(Kprev.size());
      for (size_t b = 0; b < Kprev.size(); b++) fin[b] = h_compose(n, Kprev[b], D[t]);
      const std::vector<int> fd = c->dist_of(tab, fin);
      int bestv = 1 << 30;
      for (size_t b = 0; b < fin.size(); b++) {
        const int v = bcost[b] + (fd[b] < 0 ? 999 : fd[b]);
        if (v < bestv) { bestv = v; best = (int)b; }
      }
    }
    std::vector<Pick> K(t);
    for (int j = t - 1, b = best; j >= 0; j--) { K[j] = hist[j][b]; b = hist[j][b].parent; }
    std::vector<uint64_t> Kinv(t);
    std::vector<int> dag(t);
    for (int j = 0; j < t; j++) {                       // the placed T: dagger after the sign and the flip
      const int d0 = J.td[j] ^ K[j].neg;
      Kinv[j] = h_inverse(n, K[j].K);
      if (K[j].flip) Kinv[j] = h_gate(n, Kinv[j], d0 ? CG_SDG : CG_S, K[j].qp, 0);
      dag[j] = d0 ^ K[j].flip;
    }
    std::vector<uint64_t> segs(t + 1);
    for (int j = 0; j <= t; j++) {
      uint64_t X = j > 0 ? h_compose(n, K[j - 1].K, D[j]) : D[j];
      if (j < t) X = h_compose(n, X, Kinv[j]);
      segs[j] = X;
    }
    std::vector<std::vector<int>> w;
    c->words(tab, segs, w);
    const GateSet gs = gate_set(n);
    static const char *nm[] = {"h", "s", "sdg", "x", "z", "cx", "y"};
    std::string txt;
    char line[64];
    int total = 0, before = 0;
    for (int j = 0; j <= t; j++) {
      total += (int)w[j].size();
      before += (int)(J.seg[j].size() / 3);
      for (int g : w[j]) {
        if (gs.k[g] == CG_CX) std::snprintf(line, sizeof line, "cx %d %d\n", gs.a[g], gs.b[g]);
        else std::snprintf(line, sizeof line, "%s %d\n", nm[gs.k[g]], gs.a[g]);
        txt += line;
      }
      if (j < t) { std::snprintf(line, sizeof line, "%s %d\n", dag[j] ? "tdg" : "t", K[j].qp); txt += line; }
    }
    res.clifford_gates = total;
    res.before = before;
    res.t_gates = t;
    res.text = std::move(txt);
    res.rc = 0;
  } catch (const std::range_error &e) {
    res.error = e.what();
    res.rc = 3;
  } catch (const std::logic_error &e) {
    res.error = e.what();
    res.rc = 4;
  } catch (const std::overflow_error &e) {
    res.error = e.what();
    res.rc = 4;
  } catch (const std::exception &e) {
    res.error = e.what();
    res.rc = 5;
  }
  res.launches = c->launches - l0;
  res.seconds = cl_now() - t0;
  return res.rc;
}

int clifford_dist(CliffordContext *c, int n, const uint64_t *tabp, size_t count, int *outp, std::string &err) {
  CliffTableInfo info;
  const int rc = clifford_table(c, n, info, err);
  if (rc) return rc;
  try {
    CTable &t = *c->tables[n];
    const std::vector<int> d = c->dist_of(t, std::vector<uint64_t>(tabp, tabp + count));
    std::copy(d.begin(), d.end(), outp);
    return 0;
  } catch (const std::exception &e) {
    err = e.what();
    return 5;
  }
}

int clifford_words(CliffordContext *c, int n, const uint64_t *tabp, size_t count,
                   std::vector<std::vector<int>> &words, std::string &err) {
  CliffTableInfo info;
  const int rc = clifford_table(c, n, info, err);
  if (rc) return rc;
  try {
    std::vector<std::vector<int>> w;
    c->words(*c->tables[n], std::vector<uint64_t>(tabp, tabp + count), w);
    const GateSet gs = gate_set(n);
    words.assign(count, {});
    for (size_t i = 0; i < count; i++)
      for (int g : w[i]) { words[i].push_back(gs.k[g]); words[i].push_back(gs.a[g]); words[i].push_back(gs.b[g]); }
    return 0;
  } catch (const std::logic_error &e) {
    err = e.what();
    return 4;
  } catch (const std::exception &e) {
    err = e.what();
    return 5;
  }
}

int clifford_element(CliffordContext *c, int n, const uint64_t *index, size_t count, uint64_t *tabp, std::string &err) {
  CliffTableInfo info;
  const int rc = clifford_table(c, n, info, err);
  if (rc) return rc;
  if (!count) return 0;
  try {
    CTable &t = *c->tables[n];
    c->tmp.ensure(count * 8); c->pk.ensure(count * 8);
    clk(cudaMemcpyAsync(c->tmp.p, index, count * 8, cudaMemcpyHostToDevice, c->s), "h2d");
    const unsigned g = c->grid(count);
    if (n == 1) k_cl_elem<1><<<g, CL_T, 0, c->s>>>(c->tmp.as<uint64_t>(), count, t.order, c->pk.as<uint64_t>());
    else if (n == 2) k_cl_elem<2><<<g, CL_T, 0, c->s>>>(c->tmp.as<uint64_t>(), count, t.order, c->pk.as<uint64_t>());
    else k_cl_elem<3><<<g, CL_T, 0, c->s>>>(c->tmp.as<uint64_t>(), count, t.order, c->pk.as<uint64_t>());
    c->launches++;
    clk(cudaGetLastError(), "element");
    clk(cudaMemcpyAsync(tabp, c->pk.p, count * 8, cudaMemcpyDeviceToHost, c->s), "d2h");
    c->sync("element");
    return 0;
  } catch (const std::exception &e) {
    err = e.what();
    return 5;
  }
}

}  // namespace cz
