// Element blocks of streaming + removal, never stored: each (cell, angle)
// block is rebuilt from the class geometry and sigma_t and solved in
// registers. ElementBlockInverse (src/block_inversek.kokkos.cxx) stores
// n_cells * A * nb^2 inverted blocks instead - 86 GB at 128^3 hexes, S8, FP64 -
// and reads them on every apply.
#include "cg.h"
#include "ctx.h"

#include <algorithm>

namespace ubolt {

// What a block solve needs of a class, in shared memory: per face the normal
// (padded to 4) and face_own, then the gradients and 1 / V, every part on a
// 16-byte boundary (the class record without face_up)
template <typename T, int NB, int F>
struct OwnRecord {
   static constexpr RecordLayout L = RecordLayout(NB, F, (int)sizeof(T));
   static constexpr int kUnit = 16 / (int)sizeof(T);
   static constexpr int kFace = 4 + L.fm, kTail = F * kFace;
   static constexpr int kFaceUnits = kFace / kUnit, kUnits = (kTail + L.size - L.tail) / kUnit;
   // The stride between records, odd in 16-byte units: lanes of different
   // cells then read different banks
   static constexpr int kSize = (kUnits | 1) * kUnit;
   // Unit u's place in the class record
   static __device__ __forceinline__ int Source(int u)
   {
      constexpr RecordLayout R(NB, F, (int)sizeof(T));
      const int f = u / kFaceUnits;
      return f < F ? R.nA(f) + (u - f * kFaceUnits) * kUnit : R.tail + (u - F * kFaceUnits) * kUnit;
   }
};

// B r = x solved in place by Gaussian elimination with partial pivoting,
// without a branch: the largest entry of a column is brought up by
// conditional row swaps (each row is eliminated by the same arithmetic
// wherever it stands). A zero pivot (a singular block) gives zero, as its
// zeroed inverse does in the reference.
template <typename T, int NB>
__device__ __forceinline__ void SolveBlockSelect(T B[NB][NB], T r[NB])
{
   bool singular = false;
#pragma unroll
   for (int k = 0; k < NB; k++) {
#pragma unroll
      for (int i = k + 1; i < NB; i++) {
         const bool up = fabs(B[i][k]) > fabs(B[k][k]);
#pragma unroll
         for (int j = k; j < NB; j++) {
            const T a = B[k][j], b = B[i][j];
            B[k][j] = up ? b : a;
            B[i][j] = up ? a : b;
         }
         const T a = r[k], b = r[i];
         r[k] = up ? b : a;
         r[i] = up ? a : b;
      }
      singular |= B[k][k] == T(0);
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
   if (singular)
#pragma unroll
      for (int k = 0; k < NB; k++) r[k] = T(0);
}

// Most threads of a block (see BlockApplyShape)
constexpr int kBlockThreads = 160;
// Blocks of that many per SM the registers should leave room for: all that fit
// without heavy spills (256^2 triangles, FP64, in blocks of 128: 97 us at five,
// 87 at six, 82 at eight; blocks of 256 threads 123)
template <typename T, int NB>
constexpr int BlockApplyMinBlocks() { return NB == 1 ? 9 : sizeof(T) == 8 && NB == 4 ? 3 : 6; }

// y = B^{-1} x (or B^{-T} x). A block holds K whole cells, a thread one cell and AP consecutive ordinates at a time (one 16-byte run of
// each row). The cells' shape data are staged in shared memory by cp.async
// beside the loads of x. Bound by issue: about 230 instructions per (cell,
// ordinate), half of them FP64, none behind a branch that splits a warp. A
// thread per (cell, ordinate) with branches on the signs of the face terms and on
// the pivots, its shapes gathered through L1, and this kernel, S8, FP64 / FP32:
// 256^2 triangles 153 / 77 -> 86 / 49 us (0.45 / 0.39 of the copy bandwidth),
// 301 x 257 quadrilaterals 108 / 49 -> 58 / 36, 40^3 hexahedra 405 / 154 -> 188 /
// 86, 20^3 cubes of tetrahedra 273 / 107 -> 118 / 56.
template <typename T, int NB, int F, int AP, bool TRANS>
__global__ void __launch_bounds__(kBlockThreads, BlockApplyMinBlocks<T, NB>())
   BlockApplyKernel(const DevGeom<T> g, const T *__restrict__ x, T *__restrict__ y, int K)
{
   using Rec = OwnRecord<T, NB, F>;
   constexpr RecordLayout L(NB, F, (int)sizeof(T));
   constexpr int kFm = L.fm, kRecSize = L.size;
   extern __shared__ __align__(16) unsigned char smem_raw[];
   T *recs = reinterpret_cast<T *>(smem_raw);
   const int A = g.A, QA = A / AP;
   const int64_t c0 = (int64_t)blockIdx.x * K;
   const int kc = (int)min((int64_t)K, g.n_cells - c0);
   for (int e = threadIdx.x; e < kc * Rec::kUnits; e += (int)blockDim.x) {
      const int k = e / Rec::kUnits, u = e - k * Rec::kUnits;
      CpAsync<16>(recs + k * Rec::kSize + u * Rec::kUnit, g.rec + (int64_t)g.cls[c0 + k] * kRecSize + Rec::Source(u));
   }
   bool staged = false;
   for (int e0 = 0; e0 < kc * QA; e0 += (int)blockDim.x) {
      const int e = min(e0 + (int)threadIdx.x, kc * QA - 1);
      const int k = e / QA, a0 = (e - k * QA) * AP;
      const int64_t c = c0 + k;
      T v[NB][AP], om[3 * AP];
#pragma unroll
      for (int j = 0; j < NB; j++) LoadRun<T, AP>(x + (c * NB + j) * A + a0, v[j]);
      LoadRun<T, 3 * AP>(g.omega + 3 * a0, om);
      const T sigma = g.sigma_t[c];
      if (!staged) {
         CpAsyncWaitAll();
         __syncthreads();
         staged = true;
      }
      const T *rec = recs + k * Rec::kSize;
#pragma unroll
      for (int p = 0; p < AP; p++) {
         // One ordinate after the other: with the matrices read once for all
         // of them they are kept in registers, and spill
         asm volatile("" ::: "memory");
         const T o[3] = {om[3 * p], om[3 * p + 1], om[3 * p + 2]};
         T B[NB][NB], r[NB];
#pragma unroll
         for (int i = 0; i < NB; i++) {
            r[i] = v[i][p];
#pragma unroll
            for (int j = 0; j < NB; j++) B[i][j] = T(0);
         }
         if constexpr (NB == 1) {
            T out = T(0);
#pragma unroll
            for (int f = 0; f < F; f++) out += fmax(Dot3(o, rec + f * Rec::kFace), T(0));
            B[0][0] = out * rec[Rec::kTail] + sigma;
         } else {
#pragma unroll
            for (int f = 0; f < F; f++) {
               T n[4], m[kFm];
               LoadShared<T, 4>(rec + f * Rec::kFace, n);
               LoadShared<T, kFm>(rec + f * Rec::kFace + 4, m);
               const T s = fmax(Dot3(o, n), T(0));
#pragma unroll
               for (int i = 0; i < NB; i++)
#pragma unroll
                  for (int j = 0; j < NB; j++) B[i][j] += s * m[i * NB + j];
            }
#pragma unroll
            for (int i = 1; i < NB; i++) B[i][0] -= Dot3(o, rec + Rec::kTail + 3 * i);
#pragma unroll
            for (int i = 0; i < NB; i++) B[i][i] += sigma;
            if constexpr (TRANS) Transpose<T, NB>(B);
         }
         SolveBlockSelect<T, NB>(B, r);
#pragma unroll
         for (int i = 0; i < NB; i++) v[i][p] = r[i];
      }
      if (e0 + (int)threadIdx.x < kc * QA)
#pragma unroll
         for (int j = 0; j < NB; j++) StoreRun<T, AP>(y + (c * NB + j) * A + a0, v[j]);
   }
}

// The same, a thread per (cell, ordinate) that reads its cell's shape data
// itself (LaunchBlockApply says where)
template <typename T, int NB, int F, bool TRANS>
__global__ void __launch_bounds__(256) BlockApplyDirectKernel(const DevGeom<T> g, const T *__restrict__ x, T *__restrict__ y)
{
   const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
   if (tid >= g.n_cells * g.A) return;
   const int64_t c = tid / g.A;
   const int a = (int)(tid - c * g.A);
   const T om[3] = {g.omega[3 * a], g.omega[3 * a + 1], g.omega[3 * a + 2]};
   T B[NB][NB], r[NB];
   BuildBlock<T, NB, F>(g, g.cls[c], om, g.sigma_t[c], B);
   if constexpr (TRANS) Transpose<T, NB>(B);
#pragma unroll
   for (int j = 0; j < NB; j++) r[j] = x[(c * NB + j) * g.A + a];
   const bool ok = SolveBlock<T, NB>(B, r);
#pragma unroll
   for (int j = 0; j < NB; j++) y[(c * NB + j) * g.A + a] = ok ? r[j] : T(0);
}

// Singular-block census (ElementBlockInverse::setup's check,
// block_inversek.kokkos.cxx:291-296)
template <typename T, int NB, int F>
__global__ void BlockCountKernel(const DevGeom<T> g, unsigned long long *n_singular)
{
   const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
   bool bad = false;
   if (tid < g.n_cells * g.A) {
      const int64_t c = tid / g.A;
      const int a = (int)(tid - c * g.A);
      const T om[3] = {g.omega[3 * a], g.omega[3 * a + 1], g.omega[3 * a + 2]};
      T B[NB][NB], r[NB];
      BuildBlock<T, NB, F>(g, g.cls[c], om, g.sigma_t[c], B);
#pragma unroll
      for (int j = 0; j < NB; j++) r[j] = T(1);
      bad = !SolveBlock<T, NB>(B, r);
   }
   const unsigned m = __ballot_sync(0xffffffffu, bad);
   if ((threadIdx.x & 31) == 0 && m) atomicAdd(n_singular, (unsigned long long)__popc(m));
}

// The explicit inverse of every (cell, angle) block (InvertBlocksKernel,
// block_inversek.kokkos.cxx:83-150); a singular block is stored as zero.
template <typename T, int NB, int F>
__global__ void BlockInverseKernel(const DevGeom<T> g, T *__restrict__ inv)
{
   const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
   if (b >= g.n_cells * g.A) return;
   const int64_t c = b / g.A;
   const int a = (int)(b - c * g.A);
   const T om[3] = {g.omega[3 * a], g.omega[3 * a + 1], g.omega[3 * a + 2]};
   T m[NB][NB], w[NB][NB];
   BuildBlock<T, NB, F>(g, g.cls[c], om, g.sigma_t[c], m);
   const bool ok = InvertBlock<T, NB>(m, w);
#pragma unroll
   for (int i = 0; i < NB; i++)
#pragma unroll
      for (int j = 0; j < NB; j++) inv[(b * NB + i) * NB + j] = ok ? w[i][j] : T(0);
}

struct BlockShape {
   int cells, threads;
};

// Whole cells of QA threads each to a block: as many as 128 threads hold, up to
// 160 where that leaves a tenth fewer lanes idle (FP64 S16 on 256^2 DG0
// triangles, 72 threads a cell: 174 -> 130 us); a cell of more than 160 in
// rounds of equal length
static BlockShape BlockApplyShape(int QA)
{
   const auto warps = [](int n) { return (n + 31) / 32; };
   if (QA > kBlockThreads) {
      const int rounds = (QA + kBlockThreads - 1) / kBlockThreads;
      return {1, 32 * warps((QA + rounds - 1) / rounds)};
   }
   int K = std::max(1, 128 / QA);
   for (int k = K + 1; k * QA <= kBlockThreads; k++)
      if (10 * k * warps(K * QA) > 11 * K * warps(k * QA)) K = k;
   return {K, 32 * warps(K * QA)};
}

template <typename T, int NB, int F>
static int LaunchBlockApply(const DevGeom<T> &g, const T *x, T *y, bool trans, cudaStream_t s)
{
   // Ordinates per thread as one 16-byte run where they divide evenly, both
   // vectors are 16-byte aligned and a cell has three runs or more: with
   // fewer a block holds the shapes of so many cells that few fit an SM (S2,
   // two runs, FP64: 256^2 triangles 40 us in runs and 32 one by one)
   constexpr int AV = 16 / (int)sizeof(T);
   const bool vec = g.A % AV == 0 && g.A / AV >= 3 &&
                    (reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) % 16 == 0;
   // Without staging where that only delays: DG0 one by one, a division per
   // value (256^2 triangles S16 FP64 off a 16-byte boundary: 187 us staged,
   // 122), and DG1 triangles of four ordinates (S2), which use half of the
   // shape data staged for them (256^2: 25 us, 19)
   if constexpr (NB == 1 || F == 3)
      if (!vec && (NB == 1 || g.A <= 4)) {
         const int64_t n = g.n_cells * g.A;
         const unsigned grid = (unsigned)((n + 255) / 256);
         if (trans) BlockApplyDirectKernel<T, NB, F, true><<<grid, 256, 0, s>>>(g, x, y);
         else BlockApplyDirectKernel<T, NB, F, false><<<grid, 256, 0, s>>>(g, x, y);
         return CheckLaunch("block_apply");
      }
   const int QA = g.A / (vec ? AV : 1);
   const BlockShape shape = BlockApplyShape(QA);
   const int K = shape.cells, threads = shape.threads;
   const size_t smem = (size_t)K * OwnRecord<T, NB, F>::kSize * sizeof(T);
   auto kern = vec ? (trans ? BlockApplyKernel<T, NB, F, AV, true> : BlockApplyKernel<T, NB, F, AV, false>)
                   : (trans ? BlockApplyKernel<T, NB, F, 1, true> : BlockApplyKernel<T, NB, F, 1, false>);
   if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
   kern<<<(g.n_cells + K - 1) / K, threads, smem, s>>>(g, x, y, K);
   return CheckLaunch("block_apply");
}

template <typename T>
int BlockApply(ubolt_ctx *ctx, const T *x, T *y, bool trans, void *stream)
{
   int rc = CheckReady(ctx, true);
   if (rc) return rc;
   if (!x || !y || (const void *)x == (const void *)y)
      return SetError(UBOLT_ERR_ARG, "block apply: x and y must be distinct device arrays");
   if (ctx->cg) {
      if (trans) return RequireDg(ctx, "the transposed block apply");
      return CgJacobiApply<T>(ctx, x, y, stream);
   }
   UBOLT_DISPATCH(ctx->nb, ctx->F,
                  return (LaunchBlockApply<T, NB_, F_>(ctx->geom<T>(), x, y, trans, (cudaStream_t)stream)));
   return SetError(UBOLT_ERR_STATE, "no kernel for this shape");
}

template int BlockApply<double>(ubolt_ctx *, const double *, double *, bool, void *);
template int BlockApply<float>(ubolt_ctx *, const float *, float *, bool, void *);

}  // namespace ubolt

using namespace ubolt;

extern "C" int ubolt_block_apply(ubolt_ctx *ctx, const double *x, double *y, void *stream)
{
   return BlockApply<double>(ctx, x, y, false, stream);
}
extern "C" int ubolt_block_apply_f32(ubolt_ctx *ctx, const float *x, float *y, void *stream)
{
   return BlockApply<float>(ctx, x, y, false, stream);
}
extern "C" int ubolt_block_apply_transpose(ubolt_ctx *ctx, const double *x, double *y, void *stream)
{
   return BlockApply<double>(ctx, x, y, true, stream);
}

extern "C" int ubolt_block_setup(ubolt_ctx *ctx, int64_t *n_singular, void *stream)
{
   int rc = CheckReady(ctx, true);
   if (rc) return rc;
   if (ctx->cg) return CgJacobiSetup(ctx, n_singular, stream);
   unsigned long long *d = ctx->d_counters, h = 0;
   cudaStream_t s = (cudaStream_t)stream;
   cudaMemsetAsync(d, 0, sizeof *d, s);
   const int64_t n = ctx->n_cells * ctx->A;
   UBOLT_DISPATCH(ctx->nb, ctx->F, (BlockCountKernel<double, NB_, F_><<<(n + 255) / 256, 256, 0, s>>>(ctx->g64, d)));
   rc = CheckLaunch("block_setup");
   cudaMemcpyAsync(&h, d, sizeof h, cudaMemcpyDeviceToHost, s);
   if (!rc) rc = CudaCheck(cudaStreamSynchronize(s), "block_setup");
   if (n_singular) *n_singular = (int64_t)h;
   if (rc) return rc;
   if (h) return SetError(UBOLT_ERR_SINGULAR, "%llu of %lld element blocks are singular", h, (long long)n);
   return UBOLT_OK;
}

extern "C" int ubolt_block_inverse(ubolt_ctx *ctx, double *inv, void *stream)
{
   int rc = CheckReady(ctx, true);
   if (rc) return rc;
   if (!inv) return SetError(UBOLT_ERR_ARG, "block_inverse: NULL output");
   if ((rc = RequireDg(ctx, "block_inverse"))) return rc;
   const int64_t n = ctx->n_cells * ctx->A;
   cudaStream_t s = (cudaStream_t)stream;
   UBOLT_DISPATCH(ctx->nb, ctx->F, (BlockInverseKernel<double, NB_, F_><<<(n + 255) / 256, 256, 0, s>>>(ctx->g64, inv)));
   return CheckLaunch("block_inverse");
}
