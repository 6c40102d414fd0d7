// Device-side data layout and the per-(cell, angle) arithmetic shared by the
// apply, block, sweep and adjoint kernels.
//
// HBM layout. Phase-space vectors keep UBOLT's row order (angle fastest), so
// a cell's n_basis * n_angles values are one contiguous run. Geometry is
// split into a per-CELL part - the face codes (neighbour or boundary side),
// the mirror slot of each interior face, a geometry-class id - and a
// per-CLASS part holding everything derived from shape: outward area
// normals, face matrices, basis gradients, face basis values, volume. Cells
// whose class data are bitwise equal share a class, so a uniform box reads
// a few dozen classes from L1/L2 instead of kilobytes of geometry per cell.
#pragma once

#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>

namespace ubolt {

constexpr int kMaxNb = 4;
constexpr int kMaxFaces = 6;

// Face code per (cell, slot): >= 0 the neighbour cell; -1 - side on the
// boundary, side = 2 * axis + (0 low | 1 high).
__host__ __device__ inline bool FaceInterior(int32_t code) { return code >= 0; }
__host__ __device__ inline int FaceSide(int32_t code) { return -1 - code; }

// n elements of `elem` bytes rounded up to a whole number of 16-byte units
__host__ __device__ constexpr int Pad16(int n, int elem) { return (n + 16 / elem - 1) / (16 / elem) * (16 / elem); }

// A geometry class packed as one record of 16-byte units, so a thread reads
// a face's parts with a few vector loads: per face f a slab [nA_f (3, padded
// to 4) | face_own_f (nb x nb) | face_up_f (nb x nb)], then [grad phi (nb x
// 3) | 1 / V] (the matrices and gradients only for nb > 1), each part padded
// to 16 bytes. Offsets in elements of `elem` bytes.
struct RecordLayout {
   int nb, fm, fs, tail, size;
   __host__ __device__ constexpr RecordLayout(int nb_, int F, int elem)
       : nb(nb_), fm(nb_ > 1 ? Pad16(nb_ * nb_, elem) : 0), fs(4 + 2 * (nb_ > 1 ? Pad16(nb_ * nb_, elem) : 0)),
         tail(F * (4 + 2 * (nb_ > 1 ? Pad16(nb_ * nb_, elem) : 0))),
         size(F * (4 + 2 * (nb_ > 1 ? Pad16(nb_ * nb_, elem) : 0)) + Pad16((nb_ > 1 ? 3 * nb_ : 0) + 1, elem))
   {
   }
   __host__ __device__ constexpr int nA(int f) const { return f * fs; }
   __host__ __device__ constexpr int fown(int f) const { return f * fs + 4; }
   __host__ __device__ constexpr int fup(int f) const { return f * fs + 4 + fm; }
   __host__ __device__ constexpr int bgrad() const { return tail; }
   __host__ __device__ constexpr int ivol() const { return tail + (nb > 1 ? 3 * nb : 0); }
};

template <typename T>
struct DevGeom {
   int32_t dim, nb, F, A;
   int64_t n_cells;
   T sum_weights;
   T inv_sum_weights;
   // Per class
   const T *nA;       // [class][F][3]
   const T *fown;     // [class][F][nb][nb]
   const T *fup;      // [class][F][nb][nb]
   const T *bgrad;    // [class][nb][3]
   const T *fbv;      // [class][F][nb]
   const T *inv_vol;  // [class]
   const T *rec;      // [class][RecordLayout(nb, F, sizeof(T)).size]: the same data packed per class
   // Per cell
   const int32_t *cls;     // [cell]
   const int32_t *code;    // [cell][F]
   const int8_t *mirror;   // [cell][F]: the neighbour's slot for the same face, -1 on the boundary
   // Quadrature
   const T *omega;         // [A][3]
   const T *w;             // [A]
   const int32_t *refl;    // [3][A]
   int32_t side_bc[6];     // UBOLT_BC_* per side
   const int32_t *opp;     // [A] the opposite ordinate (every cosine negated)
   const T *volume;        // [cell] cell volume
   // Group cross sections (per cell)
   const T *sigma_t;
   const T *sigma_s;
};

// An asynchronous global -> shared copy of one 4-, 8- or 16-byte word, both
// addresses aligned to its size
template <int BYTES>
__device__ __forceinline__ void CpAsync(void *smem_dst, const void *src)
{
   const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
   asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(src), "n"(BYTES) : "memory");
}
// An L2 policy that evicts a line first: for data read once per launch
// (streamed through, not to displace what other warps are about to read)
__device__ __forceinline__ uint64_t EvictFirstPolicy()
{
   uint64_t p;
   asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
   return p;
}
// A load with an L2 cache policy
__device__ __forceinline__ double LoadHint(const double *p, uint64_t policy)
{
   double v;
   asm volatile("ld.global.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(p), "l"(policy));
   return v;
}
__device__ __forceinline__ float LoadHint(const float *p, uint64_t policy)
{
   float v;
   asm volatile("ld.global.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(policy));
   return v;
}
__device__ __forceinline__ void CpAsyncWaitAll() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void CpAsyncCommit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// Wait until at most N of this thread's committed groups are still in flight
template <int N>
__device__ __forceinline__ void CpAsyncWaitGroup() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ uint32_t SmemAddr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void MbarInit(uint64_t *bar, uint32_t count)
{
   asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(SmemAddr(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void MbarInitFence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

__device__ __forceinline__ void MbarExpectTx(uint64_t *bar, uint32_t bytes)
{
   asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(SmemAddr(bar)), "r"(bytes) : "memory");
}

// One contiguous global -> shared copy completing on `bar` (both addresses
// 16-byte aligned, bytes a multiple of 16)
__device__ __forceinline__ void BulkLoad(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
   asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                    SmemAddr(dst)),
                "l"(src), "r"(bytes), "r"(SmemAddr(bar))
                : "memory");
}

__device__ __forceinline__ bool MbarTryWait(uint64_t *bar, uint32_t parity)
{
   uint32_t ok;
   asm volatile(
       "{\n\t.reg .pred p;\n\t"
       "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
       "selp.u32 %0, 1, 0, p;\n\t}"
       : "=r"(ok)
       : "r"(SmemAddr(bar)), "r"(parity)
       : "memory");
   return ok != 0;
}

// At most limit + 1 polls of the phase
__device__ __forceinline__ bool MbarWaitBounded(uint64_t *bar, uint32_t parity, uint32_t limit)
{
   for (uint32_t k = 0; k <= limit; k++)
      if (MbarTryWait(bar, parity)) return true;
   return false;
}

// N consecutive values from an address aligned to 16 bytes (N * sizeof(T)
// a multiple of 16), to 8 bytes (8), or element-aligned
template <typename T, int N>
__device__ __forceinline__ void LoadRun(const T *__restrict__ p, T v[N])
{
   constexpr int B = (int)sizeof(T) * N;
   if constexpr (B % 16 == 0) {
#pragma unroll
      for (int u = 0; u < B / 16; u++) {
         const int4 w = __ldg(reinterpret_cast<const int4 *>(p) + u);
         memcpy(&v[u * (16 / (int)sizeof(T))], &w, 16);
      }
   } else if constexpr (B == 8 && sizeof(T) == 4) {
      const int2 w = __ldg(reinterpret_cast<const int2 *>(p));
      memcpy(v, &w, 8);
   } else {
#pragma unroll
      for (int i = 0; i < N; i++) v[i] = __ldg(p + i);
   }
}

template <typename T, int N>
__device__ __forceinline__ void StoreRun(T *__restrict__ p, const T v[N])
{
   constexpr int B = (int)sizeof(T) * N;
   if constexpr (B % 16 == 0) {
#pragma unroll
      for (int u = 0; u < B / 16; u++) {
         int4 w;
         memcpy(&w, &v[u * (16 / (int)sizeof(T))], 16);
         __stcs(reinterpret_cast<int4 *>(p) + u, w);
      }
   } else {
#pragma unroll
      for (int i = 0; i < N; i++) p[i] = v[i];
   }
}

// N consecutive values from shared memory, 16-byte aligned when N *
// sizeof(T) is a multiple of 16
template <typename T, int N>
__device__ __forceinline__ void LoadShared(const T *p, T v[N])
{
   if constexpr ((int)sizeof(T) * N % 16 == 0) {
#pragma unroll
      for (int u = 0; u < (int)sizeof(T) * N / 16; u++) {
         const int4 w = reinterpret_cast<const int4 *>(p)[u];
         memcpy(&v[u * (16 / (int)sizeof(T))], &w, 16);
      }
   } else {
#pragma unroll
      for (int i = 0; i < N; i++) v[i] = p[i];
   }
}

template <typename T>
__device__ __forceinline__ T Dot3(const T *__restrict__ om, const T *__restrict__ n)
{
   // Omega . nA in the reference's term order (FaceFlux, plex_commonk.hpp:314-317)
   return om[0] * n[0] + om[1] * n[1] + om[2] * n[2];
}
template <typename T>
__device__ __forceinline__ T Dot3(T ox, T oy, T oz, const T *__restrict__ n)
{
   return ox * n[0] + oy * n[1] + oz * n[2];
}

// The (cell, angle) element block of streaming + removal:
//   B(i, j) = sum_{f: s_f > 0} s_f face_own_f(i, j) - [j == 0, i > 0] Omega . grad phi_i + sigma_t delta_ij
// DG0: B = (sum_{s > 0} s) / V + sigma_t (DG0OutflowDiagonal then removal,
// termsk.kokkos.cxx:183-196, 451-470). DG1: StreamingTermDG1::assemble_add,
// termsk.kokkos.cxx:314-389.
template <typename T, int NB, int F>
__device__ __forceinline__ void BuildBlock(const DevGeom<T> &g, int32_t cl, const T om[3], T sigma_t, T B[NB][NB])
{
   if constexpr (NB == 1) {
      T outflow = T(0);
#pragma unroll
      for (int f = 0; f < F; f++) {
         const T s = Dot3(om, g.nA + ((int64_t)cl * F + f) * 3);
         if (s > T(0)) outflow += s;
      }
      B[0][0] = outflow * g.inv_vol[cl] + sigma_t;
   } else {
#pragma unroll
      for (int i = 0; i < NB; i++)
#pragma unroll
         for (int j = 0; j < NB; j++) B[i][j] = T(0);
#pragma unroll
      for (int f = 0; f < F; f++) {
         const T s = Dot3(om, g.nA + ((int64_t)cl * F + f) * 3);
         if (s > T(0)) {
            const T *M = g.fown + ((int64_t)cl * F + f) * NB * NB;
#pragma unroll
            for (int i = 0; i < NB; i++)
#pragma unroll
               for (int j = 0; j < NB; j++) B[i][j] += s * M[i * NB + j];
         }
      }
#pragma unroll
      for (int i = 1; i < NB; i++) B[i][0] -= Dot3(om, g.bgrad + ((int64_t)cl * NB + i) * 3);
#pragma unroll
      for (int i = 0; i < NB; i++) B[i][i] += sigma_t;
   }
}

// Solve B y = r in place by Gaussian elimination with partial pivoting.
// Returns false for a singular block (a zero pivot), leaving r unchanged.
template <typename T, int NB>
__device__ __forceinline__ bool SolveBlock(T B[NB][NB], T r[NB])
{
   if constexpr (NB == 1) {
      if (B[0][0] == T(0)) return false;
      r[0] = r[0] / B[0][0];
      return true;
   } else {
#pragma unroll
      for (int k = 0; k < NB; k++) {
         int piv = k;
         T best = fabs(B[k][k]);
#pragma unroll
         for (int i = k + 1; i < NB; i++) {
            const T v = fabs(B[i][k]);
            if (v > best) { best = v; piv = i; }
         }
         if (best == T(0)) return false;
         if (piv != k) {
#pragma unroll
            for (int i = k + 1; i < NB; i++)
               if (i == piv) {
#pragma unroll
                  for (int j = 0; j < NB; j++) { const T t = B[k][j]; B[k][j] = B[i][j]; B[i][j] = t; }
                  const T t = r[k]; r[k] = r[i]; r[i] = t;
               }
         }
         const T inv = T(1) / B[k][k];
#pragma unroll
         for (int i = k + 1; i < NB; i++) {
            const T f = B[i][k] * inv;
#pragma unroll
            for (int j = k + 1; j < NB; j++) B[i][j] -= f * B[k][j];
            r[i] -= f * r[k];
         }
      }
#pragma unroll
      for (int k = NB - 1; k >= 0; k--) {
         T s = r[k];
#pragma unroll
         for (int j = k + 1; j < NB; j++) s -= B[k][j] * r[j];
         r[k] = s / B[k][k];
      }
      return true;
   }
}

// The explicit inverse by Gauss-Jordan with partial pivoting, [B | I] ->
// [I | B^{-1}], in InvertBlocksKernel's order (block_inversek.kokkos.cxx:83-150).
// B is destroyed. False on a zero pivot, with W left partial.
template <typename T, int NB>
__device__ __forceinline__ bool InvertBlock(T m[NB][NB], T w[NB][NB])
{
#pragma unroll
   for (int i = 0; i < NB; i++)
#pragma unroll
      for (int j = 0; j < NB; j++) w[i][j] = (i == j) ? T(1) : T(0);
#pragma unroll
   for (int k = 0; k < NB; k++) {
      int piv = k;
      T best = fabs(m[k][k]);
#pragma unroll
      for (int i = k + 1; i < NB; i++) {
         const T v = fabs(m[i][k]);
         if (v > best) { best = v; piv = i; }
      }
      if (best == T(0)) return false;
      if (piv != k) {
#pragma unroll
         for (int i = 0; i < NB; i++)
            if (i == piv && i != k) {
#pragma unroll
               for (int j = 0; j < NB; j++) {
                  T t = m[k][j]; m[k][j] = m[i][j]; m[i][j] = t;
                  t = w[k][j]; w[k][j] = w[i][j]; w[i][j] = t;
               }
            }
      }
      const T inv_piv = T(1) / m[k][k];
#pragma unroll
      for (int j = 0; j < NB; j++) { m[k][j] *= inv_piv; w[k][j] *= inv_piv; }
#pragma unroll
      for (int i = 0; i < NB; i++) {
         if (i == k) continue;
         const T f = m[i][k];
         if (f == T(0)) continue;
#pragma unroll
         for (int j = 0; j < NB; j++) { m[i][j] -= f * m[k][j]; w[i][j] -= f * w[k][j]; }
      }
   }
   return true;
}

template <typename T, int NB>
__device__ __forceinline__ void Transpose(T B[NB][NB])
{
#pragma unroll
   for (int i = 0; i < NB; i++)
#pragma unroll
      for (int j = i + 1; j < NB; j++) { const T t = B[i][j]; B[i][j] = B[j][i]; B[j][i] = t; }
}

// Threads per block for the (cell, angle)-flattened kernels: whole cells per
// block, about 256 threads.
__host__ inline int CellsPerBlock(int A)
{
   int k = (256 + A / 2) / A;
   return k < 1 ? 1 : k;
}

// The explicit inverse as InvertBlock's, without a branch: the largest entry of
// a column comes up by conditional row swaps, which leave every row's
// arithmetic as it is. False on a zero pivot, with w not to be used.
template <typename T, int NB>
__device__ __forceinline__ bool InvertBlockSelect(T m[NB][NB], T w[NB][NB])
{
   bool ok = true;
#pragma unroll
   for (int i = 0; i < NB; i++)
#pragma unroll
      for (int j = 0; j < NB; j++) w[i][j] = (i == j) ? T(1) : T(0);
#pragma unroll
   for (int k = 0; k < NB; k++) {
#pragma unroll
      for (int i = k + 1; i < NB; i++) {
         const bool up = fabs(m[i][k]) > fabs(m[k][k]);
#pragma unroll
         for (int j = 0; j < NB; j++) {
            const T a = m[k][j], b = m[i][j], c = w[k][j], e = w[i][j];
            m[k][j] = up ? b : a;
            m[i][j] = up ? a : b;
            w[k][j] = up ? e : c;
            w[i][j] = up ? c : e;
         }
      }
      ok &= m[k][k] != T(0);
      const T inv_piv = T(1) / m[k][k];
#pragma unroll
      for (int j = 0; j < NB; j++) { m[k][j] *= inv_piv; w[k][j] *= inv_piv; }
#pragma unroll
      for (int i = 0; i < NB; i++) {
         if (i == k) continue;
         const T f = m[i][k];
#pragma unroll
         for (int j = 0; j < NB; j++) { m[i][j] -= f * m[k][j]; w[i][j] -= f * w[k][j]; }
      }
   }
   return ok;
}

// The factors of one (cell, ordinate) for the sweep, from the cell's class
// record (in shared or global memory): W = B^{-1} of its streaming + removal
// block, and G_s = W (s_f face_up_f) for each gathered face f of `mask` in face
// order (slot s < S; unused slots zero); element (s, ii, j) goes to
// Gout[s * gs + ii * gr + j * gj]. A singular block gives zero factors. With
// the records in shared memory (SHARED) no lane branches on its own; from
// global memory, where the lanes' cells lie on lines of their own and the
// loads are what costs, a face's matrix is read only where it counts.
template <typename T, int NB, int F, bool SHARED>
__device__ __forceinline__ void CellFactors(const T *rec, T sigma_t, const T om[3], uint32_t mask, int S, T W[NB][NB],
                                            T *Gout, size_t gs, size_t gr, size_t gj)
{
   constexpr RecordLayout L(NB, F, (int)sizeof(T));
   constexpr int kFm = L.fm > 0 ? L.fm : 1, kTail = L.size - L.tail;
   T B[NB][NB], tail[kTail];
   LoadShared<T, kTail>(rec + L.tail, tail);
#pragma unroll
   for (int i = 0; i < NB; i++)
#pragma unroll
      for (int j = 0; j < NB; j++) B[i][j] = T(0);
#pragma unroll
   for (int f = 0; f < F; f++) {
      T n[4];
      LoadShared<T, 4>(rec + L.nA(f), n);
      const T s = fmax(Dot3(om, n), T(0));
      if constexpr (NB == 1) {
         B[0][0] += s;
      } else if (SHARED || s > T(0)) {
         T m[kFm];
         LoadShared<T, kFm>(rec + L.fown(f), m);
#pragma unroll
         for (int i = 0; i < NB; i++)
#pragma unroll
            for (int j = 0; j < NB; j++) B[i][j] += s * m[i * NB + j];
      }
   }
   if constexpr (NB == 1) {
      B[0][0] = B[0][0] * tail[0] + sigma_t;
   } else {
#pragma unroll
      for (int i = 1; i < NB; i++) B[i][0] -= Dot3(om, tail + 3 * i);
#pragma unroll
      for (int i = 0; i < NB; i++) B[i][i] += sigma_t;
   }
   const bool ok = InvertBlockSelect<T, NB>(B, W);
#pragma unroll
   for (int ii = 0; ii < NB; ii++)
#pragma unroll
      for (int j = 0; j < NB; j++) W[ii][j] = ok ? W[ii][j] : T(0);
   uint32_t left = (mask | (mask >> 8)) & 0xffu;
#pragma unroll 1
   for (int slot = 0; slot < S; slot++) {
      const bool used = left != 0;
      const int f = used ? __ffs(left) - 1 : 0;
      left &= left - 1;
      T n[4];
      LoadShared<T, 4>(rec + L.nA(f), n);
      const T sf = used ? Dot3(om, n) : T(0);
      T *Gf = Gout + (size_t)slot * gs;
      if constexpr (NB == 1) {
         Gf[0] = used ? W[0][0] * (sf * tail[0]) : T(0);
      } else {
         T m[kFm];
         LoadShared<T, kFm>(rec + L.fup(f), m);
#pragma unroll
         for (int k = 0; k < NB * NB; k++) m[k] = used ? sf * m[k] : T(0);
#pragma unroll
         for (int ii = 0; ii < NB; ii++)
#pragma unroll
            for (int j = 0; j < NB; j++) {
               T u = T(0);
#pragma unroll
               for (int kk = 0; kk < NB; kk++) u += W[ii][kk] * m[kk * NB + j];
               Gf[(size_t)ii * gr + (size_t)j * gj] = u;
            }
      }
   }
}

// A grid barrier's arrival and wait, by one thread of a block of a cooperative
// launch: the block's writes so far are released, `target` arrivals waited for
// (the blocks' number times the barriers so far), the others' writes acquired.
// Bounded, at most limit + 1 polls; false: gave up. The fence empties the SM's L1.
constexpr uint32_t kGridSpins = 1u << 24;
__device__ __forceinline__ bool GridArrive(unsigned *count, unsigned target, uint32_t limit = kGridSpins)
{
   asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
   unsigned v;
   uint32_t tries = 0;
   do {
      asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
   } while ((int)(v - target) < 0 && tries++ < limit);
   __threadfence();
   return (int)(v - target) >= 0;
}

// Node-run kernels. A node's A ordinates are one contiguous run of psi. A
// warp takes kLpn = 8 lanes per node, four nodes at a time; lane `sub` of a
// node strides its run by 8, so every load or store of the warp covers four
// runs of 8 consecutive values (whole sectors), and a node's eight partial
// sums meet in 3 shuffle steps. All lanes of a warp run the same iterations.
constexpr int kLpn = 8;

__device__ __forceinline__ double GroupSum(double v)
{
   v += __shfl_xor_sync(0xffffffffu, v, 4);
   v += __shfl_xor_sync(0xffffffffu, v, 2);
   v += __shfl_xor_sync(0xffffffffu, v, 1);
   return v;
}

// Blocks of 256 threads for a grid-stride loop over groups of four runs
__host__ inline int RunGrid(int64_t n_runs)
{
   const int64_t want = (n_runs + 31) / 32;
   return (int)(want < 1 ? 1 : (want > 148 * 16 ? 148 * 16 : want));
}

}  // namespace ubolt
