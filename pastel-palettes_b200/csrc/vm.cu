// vm.cu — the persistent H-LU virtual machine for sm_100a, plus FP64 residual kernels.
//
// Replaces the reference's `kernel_dynamic` (Pastel-Palettes src/kernel.cu:1375-1526).
// The reference gives each thread block a fixed, statically scheduled instruction
// stream and makes blocks spin on per-instruction flags in global memory.  Here every
// CTA of a persistent grid takes the next READY task from a device queue (one queue, or one per
// priority class); finishing a task decrements its successors' dependency counters, and of those
// that reach zero the CTA runs the first and pushes the others.  Waits are bounded: a CTA that
// finds nothing for longer than its time limit (globaltimer) records PP_VM_TIMEOUT or PP_VM_IDLE and
// every CTA returns.
//
// Arithmetic contract (FP64 path): every matrix element receives its updates in the
// order the reference's routines apply them, one fma per product with the same
// operands, so dense results are bitwise identical to src/kernel.cu:
//   GETRF  kernel.cu:104-147   l = a_ri / a_ii;  a_rc = fma(a_ic, -l, a_rc), i ascending
//   TRSML  kernel.cu:150-182   b_rc = fma(b_ic, -l_ri, b_rc), i ascending
//   TRSMR  kernel.cu:185-226   x_ri = b_ri / u_ii; b_rc = fma(-x_ri, u_ic, b_rc)
//   TRSMRT kernel.cu:229-285   x_ic = v_ic * (1 / u_ii); v_rc = fma(-u_ir, x_ic, v_rc)
//   GEMM   kernel.cu:288-664   c_ij = fma(alpha a_ik, b_kj, c_ij), k ascending from beta c_ij
// Work distribution does not touch that order: an FP64 tensor-core product (dmma) gives the bits of
// the same chain of fma, and the routines feed it in ascending k.  Only products marked free-order
// (the solves', whose sums no contract fixes) are split over lanes and warps.
// Data other CTAs have written is loaded past L1 (ld.global.cg, cp.async.cg) or through it (8-byte
// cp.async, SHADOW's 32-byte loads): a task starts behind a gpu-scope acquire of its CTA, which
// invalidates that SM's L1.
//
// What an instruction costs inside the VM is often its code: its lines have been evicted by the tasks
// before, a scheduler holds two warps, a taken branch costs one about 30 cycles, and beside SMs that
// load the memory system a fetch costs several times as much.  So each routine is one compact
// piece of code, inlined once (a call spills more than it saves), loops are rolled where the body
// is long enough, and conditions on lanes are predicates, not branches.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>
#include <stdint.h>

#include "vm.cuh"

#define NT PP_VM_THREADS
#define TL PP_VM_TILE
#define VM_SMEM_BYTES 184320   /* 180 KB, one CTA per SM: ACCUM keeps its ny x k1 sketch on chip;
                                  the BF16 GEMM holds 3 stages of 48 KB + its epilogue's buffers */

namespace {

__device__ __forceinline__ double ldcg(const double* p) { return __ldcg(p); }

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int atom_add_relaxed(int* p, int v) {
  int old;
  asm volatile("atom.relaxed.gpu.global.add.s32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}
__device__ __forceinline__ int ld_relaxed(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// ------------------------------------------------------------------------- FP64 tensor-core product
// mma.sync.m8n8k4.f64 (FP64 has no tcgen05 kind; this is the FP64 tensor path of sm_100a).
// Fragments: A (8 x 4) lane l holds A[l/4][l%4]; B (4 x 8) holds B[l%4][l/4]; C (8 x 8) holds
// C[l/4][2(l%4) + {0,1}].  Measured on a B200: 64 fma per clock and SM (57 for the scalar fma),
// 26 cycles from accumulator to accumulator, and the same bits as the four fma in ascending k
// (128 000 random outputs of mixed magnitude), so a chain of them keeps the arithmetic contract
// above; the bitwise tests against the oracle hold that.
__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// asynchronous copies into shared memory; bytes past `valid` are written as zeros.  The 16-byte
// form bypasses L1; the 8-byte form (odd strides or offsets) allocates there, which the VM's
// acquire before each task makes safe: it invalidates this SM's L1.
__device__ __forceinline__ void cp_async16(uint32_t dst, const double* src, uint32_t valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const double* src, uint32_t valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(valid) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// A thread index the compiler cannot hoist out of the task loop: every routine's thread-dependent
// values would otherwise be live at once in the one kernel they are inlined into.
__device__ __forceinline__ int thread_index() {
  int t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t;
}

// Predicated accesses: a branch costs a warp about 30 cycles, and with two warps per scheduler
// little hides it.
__device__ __forceinline__ double ldcg_if(const double* p, bool in) {
  double v;
  asm volatile("{\n .reg .pred a;\n setp.ne.s32 a, %2, 0;\n mov.f64 %0, 0d0000000000000000;\n @a ld.global.cg.f64 %0, [%1];\n}\n"
               : "=&d"(v)
               : "l"(p), "r"((int)in)
               : "memory");
  return v;
}
__device__ __forceinline__ void ldcg2_if(double& x, double& y, const double* p, bool in) {  // 16-byte aligned
  asm volatile("{\n .reg .pred a;\n setp.ne.s32 a, %3, 0;\n mov.f64 %0, 0d0000000000000000;\n mov.f64 %1, %0;\n"
               " @a ld.global.cg.v2.f64 {%0, %1}, [%2];\n}\n"
               : "=&d"(x), "=&d"(y)
               : "l"(p), "r"((int)in)
               : "memory");
}
__device__ __forceinline__ void st_if(double* p, double v, bool in) {
  asm volatile("{\n .reg .pred a;\n setp.ne.s32 a, %2, 0;\n @a st.global.f64 [%1], %0;\n}\n" ::"d"(v), "l"(p), "r"((int)in)
               : "memory");
}

__device__ __forceinline__ void sts_if(double* p, double v, bool in) {
  asm volatile("{\n .reg .pred a;\n setp.ne.s32 a, %2, 0;\n @a st.shared.f64 [%1], %0;\n}\n" ::"d"(v), "r"(smem_u32(p)),
               "r"((int)in)
               : "memory");
}

__host__ __device__ constexpr int log2_of(int v) { return v <= 1 ? 0 : 1 + log2_of(v / 2); }

// Four copies of one thread (16 bytes of `valid`, or 8), rows r, r + step, ... below `rows`, the
// source and the destination advancing by sstep and dstep bytes; predicated, without branches.
template <bool WIDE>
__device__ __forceinline__ void copy_rows4(uint32_t& dst, const char*& src, int& r, uint32_t dstep, uint64_t sstep,
                                           int step, int rows, uint32_t valid) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (WIDE)
      asm volatile("{\n .reg .pred p;\n setp.lt.s32 p, %2, %3;\n @p cp.async.cg.shared.global [%0], [%1], 16, %4;\n}\n" ::"r"(dst),
                   "l"(src), "r"(r), "r"(rows), "r"(valid)
                   : "memory");
    else
      asm volatile("{\n .reg .pred p;\n setp.lt.s32 p, %2, %3;\n @p cp.async.ca.shared.global [%0], [%1], 8;\n}\n" ::"r"(dst),
                   "l"(src), "r"(r), "r"(rows)
                   : "memory");
    r += step;
    src += sstep;
    dst += dstep;
  }
}

// ------------------------------------------------------------------------- GEMM
// C[m x n] = C (or 0, beta = 0) + alpha op(A) op(B); every element's k
// products in ascending order from beta c_ij (the reference's chain, see above), or with
// `free_order` a small output's k split over warps.
//
// One piece of code for every shape and transposition: a task's instructions have usually been
// evicted by the tasks before it, so much of what a small product costs is fetching its code
// (forms specialised by tile shape, ten times the code, ran small shapes at half the speed inside
// the VM and faster outside of it).  The output is walked in CTA tiles of TM x TN (128 x 16,
// 64 x 32, 128 x 32, 16 x 128, 64 x 64: the narrowest that covers it) of 16 x 16 warp tiles, one or
// two side by side per warp, k in chunks of GM_KC through a ring of GM_ST shared-memory stages over
// (tile, chunk) pairs, so that the loads of the next chunks are in flight during the products.
// Operands are staged as A[m][k] and B[k][n] whatever their storage, so that a fragment's address
// is a register and a constant; the strides (4 mod 16 doubles) keep fragment loads free of bank
// conflicts.
// What bounds it: the loads' latency and the staging's instructions for small products, the FP64
// tensor rate (2.1 M cycles for 512^3) and the staging that is not overlapped with it for large ones.
// Time per instruction on a B200, hop to the next task included (before: SIMT tiles by shape, whose
// operand loads were waited for before each chunk's products):
//   64 x 64 x 64     17 -> 7.3 us        64 x 16 x 64      16 -> 5.1 us
//   64 x 64 x 256    42 -> 17 us         16 x 16 x 512     25 -> 7.4 us (k over 8 warps)
//   512 x 512 x 512  2640 -> 1655 us     512 x 32 x 512    327 -> 105 us
#define GM_KC 64
#define GM_LD (GM_KC + 4)
#define GM_ST 2
#define GM_STAGE (VM_SMEM_BYTES / 8 / GM_ST)  /* doubles: A 128 x 68 and B 64 x 36, 64 x 68 and 64 x 68, 16 x 68 and 64 x 132 */

// v with its sign bit flipped where `mask` has it set (the factor alpha = -1, exactly: a
// multiplication would take as long on the FP64 pipe as a product of fragments)
__device__ __forceinline__ double flip(double v, int mask) {
  return __hiloint2double(__double2hiint(v) ^ mask, __double2loint(v));
}

// passes of 8 k each (two steps of 4) on a 16 x (8 NW) warp tile
template <int NW>
__device__ __forceinline__ void gemm_passes(double (&acc)[2][4][2], const double* pa, const double* pb, int b_ld,
                                            int first, int passes, int kw, int sgn) {
#pragma unroll 1
  for (int s = first; s < passes; s += kw) {
    double av[2][2], bv[2][NW];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int i = 0; i < 2; ++i) av[h][i] = pa[8 * i * GM_LD + 4 * h];
#pragma unroll
      for (int j = 0; j < NW; ++j) bv[h][j] = pb[4 * h * b_ld + 8 * j];
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const double a = flip(av[h][i], sgn);
#pragma unroll
        for (int j = 0; j < NW; ++j) dmma(acc[i][j][0], acc[i][j][1], a, bv[h][j]);
      }
    pa += 8 * kw;
    pb += 8 * kw * b_ld;
  }
}

__device__ __forceinline__ void dev_gemm(double* __restrict__ C, int ldc, const double* __restrict__ A, int lda, bool tA,
                                         const double* __restrict__ B, int ldb, bool tB, int m, int n, int k,
                                         double alpha, double beta, bool free_order) {
  extern __shared__ __align__(16) double vm_smem[];
  const int tid = thread_index(), warp = tid >> 5, lane = tid & 31, fa = lane >> 2, fb = lane & 3;
  // tile shape (log2 of TM and TN), this warp's 16 x 16 tile and whether it has the next one too,
  // and the warps that share a tile's k (free order, outputs of at most four warp tiles)
  int lm, ln, r1, c1, wide_n = 0, kw = 1, kp = 0;
  if (n <= 16) { lm = 7; ln = 4; r1 = 16 * warp; c1 = 0; }
  else if (n <= 32 && m <= 64) { lm = 6; ln = 5; r1 = 16 * (warp & 3); c1 = 16 * (warp >> 2); }
  else if (n <= 32) { lm = 7; ln = 5; r1 = 16 * warp; c1 = 0; wide_n = 1; }
  else if (m <= 16) { lm = 4; ln = 7; r1 = 0; c1 = 16 * warp; }
  else { lm = 6; ln = 6; r1 = 16 * (warp & 3); c1 = 32 * (warp >> 2); wide_n = 1; }
  if (free_order && m <= 32 && n <= 32 && k >= 64) {
    const int wt = (m > 16 ? 1 : 0) + (n > 16 ? 1 : 0);  // 2^wt warp tiles
    lm = 5; ln = 5; wide_n = 0;
    kw = 8 >> wt;
    kp = warp >> wt;
    const int t = warp & ((1 << wt) - 1);
    r1 = m > 16 ? 16 * (t & 1) : 0;
    c1 = n > 16 ? 16 * (t >> (wt - 1)) : 0;
  }
  const int TM = 1 << lm, TN = 1 << ln, b_ld = TN + 4, AE = TM * GM_LD, sgn = alpha == -1.0 ? (int)0x80000000 : 0;
  const bool scaled = alpha != 1.0 && alpha != -1.0;  // no generated program; A is scaled in its stage
  const int nch = (k + GM_KC - 1) / GM_KC, total = ((m + TM - 1) >> lm) * ((n + TN - 1) >> ln) * max(nch, 1);
  // Staging: warps 0-3 copy A, warps 4-7 copy B.  A thread keeps a column (or an aligned pair) of
  // its operand as stored and walks down the rows; `krows`: the stored rows run along k.
  const bool opB = warp >= 4, krows = opB ? !tB : tA;
  const double* src = opB ? B : A;
  const int sld = opB ? ldb : lda, osize = opB ? n : m, lo = opB ? ln : lm, lk = log2_of(GM_KC);
  const bool trans = opB ? tB : tA, wide = !trans && !((sld | (int)(reinterpret_cast<uintptr_t>(src) >> 3)) & 1);
  const int lp = (krows ? lo : lk) - (wide ? 1 : 0), sc = ((tid & 127) & ((1 << lp) - 1)) << (wide ? 1 : 0);
  const int sr = (tid & 127) >> lp, sstep = 128 >> lp, dld = opB ? b_ld : GM_LD;
  const uint32_t sdst = smem_u32(vm_smem) + 8u * (uint32_t)((opB ? AE : 0) + (trans ? sc * dld + sr : sr * dld + sc));
  const uint32_t ddst = 8u * (uint32_t)(trans ? sstep : sstep * dld);
  const uint64_t dsrc = 8ull * (uint64_t)((uint32_t)sstep * (uint32_t)sld);
  const double* sthr = src + (size_t)sr * sld + sc;
  int pi = 0, pj = 0, pc = 0, ps = 0;  // (tile, chunk) of the next stage to fill, and its slot
  int i0 = 0, j0 = 0, ch = 0, cs = 0;
  double acc[2][4][2];
#pragma unroll 1
  for (int q = 1 - GM_ST; q < total; ++q) {
    if (q >= 0) {
      if (ch == 0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int r = i0 + r1 + 8 * i + fa, c = j0 + c1 + 2 * fb;
          const double* p = C + (size_t)r * ldc + c;
          const bool in = beta != 0.0 && r < m && kp == 0;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            acc[i][j][0] = ldcg_if(p + 8 * j, in && (j < 2 || wide_n) && c + 8 * j < n);
            acc[i][j][1] = ldcg_if(p + 8 * j + 1, in && (j < 2 || wide_n) && c + 8 * j + 1 < n);
          }
        }
      }
      cp_async_wait<GM_ST - 2>();
      __syncthreads();  // stage q has landed for every thread, and stage q - 1 is free
    }
    if (q + GM_ST - 1 < total && nch > 0) {
      const int o0 = opB ? pj : pi, osz = min(1 << lo, osize - o0), kc = min(GM_KC, k - pc);
      const int rows = krows ? kc : osz, cols = krows ? osz : kc;
      const char* sp = reinterpret_cast<const char*>(sthr + (krows ? (size_t)pc * sld + o0 : (size_t)o0 * sld + pc));
      uint32_t dp = sdst + (uint32_t)ps * (8u * GM_STAGE);
      if (sc < cols) {
        int r = sr;
        if (wide) {
          const uint32_t v = cols - sc > 1 ? 16u : 8u;
#pragma unroll 1
          while (r < rows) copy_rows4<true>(dp, sp, r, ddst, dsrc, sstep, rows, v);
        } else {
#pragma unroll 1
          while (r < rows) copy_rows4<false>(dp, sp, r, ddst, dsrc, sstep, rows, 8u);
        }
      }
      if (kc & 7) {  // k past the end, up to the next multiple of 8, is zero
        double* st = vm_smem + ps * GM_STAGE;
        for (int e = tid; e < TM * 8; e += NT)
          if ((e & 7) >= (kc & 7)) st[(e >> 3) * GM_LD + (kc & ~7) + (e & 7)] = 0.0;
        for (int e = tid; e < TN * 8; e += NT)
          if ((e >> ln) >= (kc & 7)) st[AE + ((kc & ~7) + (e >> ln)) * b_ld + (e & (TN - 1))] = 0.0;
      }
      ps = ps + 1 == GM_ST ? 0 : ps + 1;
      pc += GM_KC;
      if (pc >= k) {
        pc = 0;
        pj += TN;
        if (pj >= n) { pj = 0; pi += TM; }
      }
    }
    cp_async_commit();
    if (q < 0) continue;
    if (scaled) {
      for (int e = tid; e < TM * GM_LD; e += NT) vm_smem[cs * GM_STAGE + e] *= alpha;
      __syncthreads();
    }
    if (nch > 0 && i0 + r1 < m && j0 + c1 < n) {
      const int passes = (min(GM_KC, k - ch * GM_KC) + 7) >> 3, first = (kp - ch * (GM_KC / 8)) & (kw - 1);
      const double* st = vm_smem + cs * GM_STAGE;
      const double *pa = st + (r1 + fa) * GM_LD + fb + 8 * first, *pb = st + AE + (fb + 8 * first) * b_ld + c1 + fa;
      if (wide_n && j0 + c1 + 16 < n) gemm_passes<4>(acc, pa, pb, b_ld, first, passes, kw, sgn);
      else gemm_passes<2>(acc, pa, pb, b_ld, first, passes, kw, sgn);
    }
    cs = cs + 1 == GM_ST ? 0 : cs + 1;
    if (++ch >= nch) {
      if (kw > 1) {  // the k parts of a tile, added in order (one CTA tile only)
        const int wt = kw == 8 ? 0 : kw == 4 ? 1 : 2;
        cp_async_wait<0>();
        __syncthreads();
        if (kp > 0) {
#pragma unroll
          for (int e = 0; e < 8; ++e) vm_smem[warp * 256 + e * 32 + lane] = acc[e >> 2][(e >> 1) & 1][e & 1];
        }
        __syncthreads();
        if (kp == 0) {
#pragma unroll 1
          for (int p = 1; p < kw; ++p)
#pragma unroll
            for (int e = 0; e < 8; ++e)
              acc[e >> 2][(e >> 1) & 1][e & 1] += vm_smem[(warp + (p << wt)) * 256 + e * 32 + lane];
        }
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = i0 + r1 + 8 * i + fa, c = j0 + c1 + 2 * fb;
        double* p = C + (size_t)r * ldc + c;
        const bool in = r < m && kp == 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          st_if(p + 8 * j, acc[i][j][0], in && (j < 2 || wide_n) && c + 8 * j < n);
          st_if(p + 8 * j + 1, acc[i][j][1], in && (j < 2 || wide_n) && c + 8 * j + 1 < n);
        }
      }
      ch = 0;
      j0 += TN;
      if (j0 >= n) { j0 = 0; i0 += TM; }
    }
  }
  cp_async_wait<0>();
  __syncthreads();
}

// ------------------------------------------------------------------------- tensor-core GEMM
// Mixed-precision contraction on the 5th-generation tensor cores:
//   C[m x n] (FP64) = beta C + alpha op(A) op(B),  op(A), op(B) rounded to TF32,
//   products summed in FP32 in tensor memory (TMEM), the sum added to C in FP64.
// Tile 128 x 64 (tcgen05.mma.cta_group::1.kind::tf32, M = 128, N = 64, K = 8 per
// instruction), k in chunks of 32.  Operands are staged in shared memory in the canonical
// K-major layout without swizzle: 8-row x 16-byte core matrices, core matrices 128 B apart
// along M/N (SBO) and one k16-column of core matrices apart along K (LBO).  One thread
// issues the MMAs and commits them to an mbarrier; the CTA waits on it (bounded) before
// reusing the staging buffers or reading the accumulators with tcgen05.ld.
#define TC_M 128
#define TC_N 64
#define TC_K 32
#define TC_A_BYTES (TC_M * TC_K * 4)
#define TC_B_BYTES (TC_N * TC_K * 4)
#define TC_LBO_A (TC_M / 8 * 128)  /* bytes between k16 columns of A's core matrices */
#define TC_LBO_B (TC_N / 8 * 128)
#define TC_TMEM_COLS 512  /* all of an SM's tensor memory: the VM runs one CTA per SM */

struct TcCtx {
  uint32_t tmem;      // accumulator base address in tensor memory
  uint32_t mbar;      // shared address of the MMA-completion mbarrier
  uint32_t phase;     // parity of the next completion
  long long limit;    // nanoseconds before a wait for the tensor core gives up
  int pending;        // a commit whose completion was not observed (after a timeout)
  int active;         // tensor memory and the mbarrier were set up for this CTA
  // BF16 pipeline (dev_gemm_bf16): shared address of its 10 mbarriers, the number of stage
  // fills and accumulator tiles used so far (every thread counts the same), an abort flag in
  // shared memory, and the last stage fill / tile commit whose completion nobody waited for
  uint32_t bars;
  uint32_t q;
  uint32_t u;
  int* abort;
};

__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version of sm_100; layout type 0 = no swizzle
  return d;
}

// instruction descriptor: D F32 (bits 4-5 = 1), A and B TF32 (bits 7-9, 10-12 = 2), both
// K-major, N >> 3 at bits 17-22, M >> 4 at bits 24-28
constexpr uint32_t kIdescTf32 = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(TC_N >> 3) << 17) |
                                ((uint32_t)(TC_M >> 4) << 24);

__device__ __forceinline__ uint32_t to_tf32(double v) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(__double2float_rn(v)));
  return r;
}

__device__ __forceinline__ unsigned long long gtimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// bounded wait for the completion of phase `phase` of an mbarrier: false after `limit_ns`
__device__ __forceinline__ bool mbar_wait(uint32_t addr, uint32_t phase, long long limit_ns) {
  const unsigned long long t0 = gtimer_ns();
  for (;;) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(addr), "r"(phase)
        : "memory");
    if (done) return true;
    if ((long long)(gtimer_ns() - t0) > limit_ns) return false;
  }
}

__device__ __noinline__ bool dev_gemm_tc(double* __restrict__ C, int ldc, const double* __restrict__ A, int lda,
                                         bool tA, const double* __restrict__ B, int ldb, bool tB, int m, int n, int k,
                                         double alpha, double beta, double* smem, TcCtx& tc) {
  uint8_t* sbase = reinterpret_cast<uint8_t*>(smem);
  const uint32_t s0 = smem_u32(sbase);
  const uint32_t pad = ((s0 + 1023u) & ~1023u) - s0;  // core matrices from a 1 KB boundary
  uint32_t* As = reinterpret_cast<uint32_t*>(sbase + pad);
  uint32_t* Bs = reinterpret_cast<uint32_t*>(sbase + pad + TC_A_BYTES);
  const uint32_t a_addr = s0 + pad, b_addr = s0 + pad + TC_A_BYTES;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nch = (k + TC_K - 1) / TC_K;
  bool ok = true;
  for (int i0 = 0; i0 < m; i0 += TC_M)
    for (int j0 = 0; j0 < n; j0 += TC_N) {
      for (int ch = 0; ch < nch && ok; ++ch) {
        const int k0 = ch * TC_K;
        for (int e = tid; e < TC_M * TC_K; e += NT) {
          int r, kk;
          if (!tA) { r = e / TC_K; kk = e % TC_K; }
          else { kk = e / TC_M; r = e % TC_M; }
          double v = 0.0;
          if (i0 + r < m && k0 + kk < k)
            v = tA ? ldcg(&A[(size_t)(k0 + kk) * lda + i0 + r]) : ldcg(&A[(size_t)(i0 + r) * lda + k0 + kk]);
          As[((kk >> 2) * TC_LBO_A + (r >> 3) * 128 + (r & 7) * 16 + (kk & 3) * 4) >> 2] = to_tf32(v);
        }
        for (int e = tid; e < TC_N * TC_K; e += NT) {
          int c, kk;
          if (!tB) { kk = e / TC_N; c = e % TC_N; }
          else { c = e / TC_K; kk = e % TC_K; }
          double v = 0.0;
          if (j0 + c < n && k0 + kk < k)
            v = tB ? ldcg(&B[(size_t)(j0 + c) * ldb + k0 + kk]) : ldcg(&B[(size_t)(k0 + kk) * ldb + j0 + c]);
          Bs[((kk >> 2) * TC_LBO_B + (c >> 3) * 128 + (c & 7) * 16 + (kk & 3) * 4) >> 2] = to_tf32(v);
        }
        // generic-proxy smem writes become visible to the tensor core's async proxy
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
          for (int ks = 0; ks < TC_K / 8; ++ks) {
            const uint64_t ad = umma_desc(a_addr + ks * 2 * TC_LBO_A, TC_LBO_A, 128);
            const uint64_t bd = umma_desc(b_addr + ks * 2 * TC_LBO_B, TC_LBO_B, 128);
            const uint32_t acc = (ch > 0 || ks > 0) ? 1u : 0u;
            asm volatile(
                "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                " tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}\n" ::"r"(tc.tmem),
                "l"(ad), "l"(bd), "r"(kIdescTf32), "r"(acc)
                : "memory");
          }
          asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tc.mbar)
                       : "memory");
        }
        // one verdict for the whole CTA, so that every thread takes the same path below
        ok = __syncthreads_and(mbar_wait(tc.mbar, tc.phase, tc.limit) ? 1 : 0) != 0;
        tc.phase ^= 1u;
        if (!ok) tc.pending = 1;
      }
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // accumulators: warp w reads TMEM lanes 32 (w % 4) .. + 31 (rows), columns 32 (w / 4) .. + 31
      const int q = warp & 3, h = warp >> 2;
      const int row = i0 + 32 * q + lane;
      uint32_t v[32];
      if (nch > 0) {
        const uint32_t taddr = tc.tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(32 * h);
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
            "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
              "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
              "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]),
              "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]),
              "=r"(v[30]), "=r"(v[31])
            : "r"(taddr)
            : "memory");
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      } else {
#pragma unroll
        for (int c = 0; c < 32; ++c) v[c] = 0u;
      }
      if (row < m) {
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          const int col = j0 + 32 * h + c;
          if (col < n) {
            double* p = &C[(size_t)row * ldc + col];
            const double s = alpha * (double)__uint_as_float(v[c]);
            *p = beta != 0.0 ? ldcg(p) + s : s;
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncthreads();
    }
  return ok;
}

// ------------------------------------------------------------------------- BF16 Schur GEMM
// Operands are BF16 shadows in the tiled layout of pp_task.h (PP_OP_SHADOW writes them), so
// every 128-row x 64-column chunk of an operand moves into shared memory with ONE bulk copy of
// 16 KB (the TMA engine's untiled mode: no tensor map, no per-element work) and lands in the
// canonical no-swizzle K-major layout tcgen05.mma reads.
//
// C[m x n] (FP64) = beta C + alpha A B, tile loop over 128 x 256 sub-tiles of C, k in chunks of
// 64 through a 3-stage ring of shared-memory stages (A chunk + two B chunks = 48 KB each).
// Roles inside the CTA (warp specialised):
//   warp 0, one lane   producer: waits for a free stage, posts the expected bytes on the
//                      stage's "full" mbarrier and issues the three bulk copies;
//   warp 1, one lane   MMA issuer: per stage four K=16 steps x two 128 x 128 MMAs
//                      (kind::f16, BF16 inputs, FP32 accumulators in tensor memory), then
//                      tcgen05.commit to the stage's "empty" mbarrier; after a sub-tile's last
//                      stage, a commit to the accumulator buffer's "full" mbarrier;
//   warps 4..7         epilogue: tcgen05.ld of the accumulator buffer (warp w reads TMEM lanes
//                      32 (w % 4) ..), C += alpha acc in FP64, then an arrive on the buffer's
//                      "empty" mbarrier.
// Two accumulator buffers of 256 TMEM columns: the epilogue of one sub-tile overlaps the MMAs
// of the next, and the producer runs up to three stages ahead of the MMAs.
#define BG_STAGES 3
#define BG_CHUNK PP_SHADOW_CHUNK_BYTES
#define BG_STAGE_BYTES (3 * BG_CHUNK)
#define BG_TILE_N 256
// instruction descriptor: D F32 (bits 4-5 = 1), A and B BF16 (bits 7-9, 10-12 = 1), both
// K-major, M = 128 (bits 24-28 = M >> 4); N (bits 17-22 = N >> 3) is added per task
constexpr uint32_t kIdescBf16Base = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(128 >> 4) << 24);

// byte offset of element (r, c) of an R x K operand in the tiled layout with chunks of cr rows
// (32, 64 or 128) and 64 columns
__device__ __forceinline__ size_t tiled_at(int r, int c, int K, int cr) {
  const size_t chunk = (size_t)(r / cr) * (K >> 6) + (c >> 6);
  const int rr = r % cr, cc = c & 63;
  return chunk * ((size_t)cr * 128) + (size_t)((((cc >> 3) * (cr >> 3)) + (rr >> 3)) << 7) + ((rr & 7) << 4) +
         ((cc & 7) << 1);
}

// S := the tiled BF16 shadow of X (m x k, padded with zeros beyond the source's mr rows and nc
// columns), X(r, c) = A[r lda + c] or A[c lda + r] (tA).  Each thread converts 8 consecutive columns
// of a row and stores them as one 16-byte word, lanes along the rows of a chunk (the words of 32
// consecutive rows fill 512 contiguous bytes), four words per thread at a time: 32 values in flight.
// With tA the loads are coalesced as they stand; otherwise a thread reads its 64 bytes as two whole
// sectors (one by one where they are not aligned).  A split shadow (split =
// PP_SPLIT_*, k = nseg segments of ks columns) writes each word once per segment: bf16(x), or the
// residual bf16(x - bf16(x)) in the segments of the low mask.
// Bound by the loads a CTA has in flight and by the conversions (15 per clock and SM).  512 x 512 on a
// B200: 104 -> 63 us, split 172 -> 90 us (before: 128 x 64 blocks staged through shared memory, and a
// rounding with a branch per element, which alone cost 25 us).

// two doubles to BF16, to nearest even through FP32, packed (x in the low half)
__device__ __forceinline__ uint32_t bf16_pair(double x, double y) {
  uint32_t v;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(v) : "f"(__double2float_rn(y)), "f"(__double2float_rn(x)));
  return v;
}
__device__ __forceinline__ uint4 bf16_word(const double (&x)[8], bool low) {
  uint32_t h[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    h[q] = bf16_pair(x[2 * q], x[2 * q + 1]);
    if (low)
      h[q] = bf16_pair(x[2 * q] - (double)__uint_as_float(h[q] << 16),
                       x[2 * q + 1] - (double)__uint_as_float(h[q] & 0xFFFF0000u));
  }
  return make_uint4(h[0], h[1], h[2], h[3]);
}
__device__ __forceinline__ void dev_shadow(uint8_t* S, const double* A, int lda, bool tA, int m, int k, int mr, int nc,
                                           int cr, int split) {
  constexpr int W = 4;
  const int tid = thread_index(), ks = split ? k / (split >> 8) : k;  // source columns (one segment)
  const int lc = 31 - __clz(cr), rr = tid & (cr - 1), cstep = 8 * (NT >> lc);
  const bool wide = !tA && nc >= 8 && ((lda & 3) == 0) && ((reinterpret_cast<uintptr_t>(A) & 31) == 0);
#pragma unroll 1
  for (int r0 = 0; r0 < m; r0 += cr) {
    const int r = r0 + rr;
#pragma unroll 1
    for (int cb = 8 * (tid >> lc); cb < ks; cb += W * cstep) {
      double x[W][8];
#pragma unroll
      for (int j = 0; j < W; ++j) {
        const int c = cb + j * cstep;
        const bool row = r < mr && c < ks;
        if (wide) {  // words past the source's edge are read anew below
          const double* p = A + (size_t)(row ? r : 0) * lda + (row && c + 8 <= nc ? c : 0);
#pragma unroll
          for (int h = 0; h < 2; ++h)
            asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                         : "=d"(x[j][4 * h]), "=d"(x[j][4 * h + 1]), "=d"(x[j][4 * h + 2]), "=d"(x[j][4 * h + 3])
                         : "l"(p + 4 * h)
                         : "memory");
        } else {
#pragma unroll
          for (int q = 0; q < 8; ++q)
            x[j][q] = ldcg_if(tA ? &A[(size_t)(c + q) * lda + r] : &A[(size_t)r * lda + c + q], row && c + q < nc);
        }
      }
#pragma unroll
      for (int j = 0; j < W; ++j) {
        const int c = cb + j * cstep;
        if (c >= ks) break;
        if (wide && !(r < mr && c + 8 <= nc)) {
#pragma unroll
          for (int q = 0; q < 8; ++q) x[j][q] = ldcg_if(&A[(size_t)r * lda + c + q], r < mr && c + q < nc);
        }
        const uint4 high = bf16_word(x[j], false);
        if (!split) {
          *reinterpret_cast<uint4*>(S + tiled_at(r, c, k, cr)) = high;
        } else {
          const uint4 low = bf16_word(x[j], true);
          const int nseg = split >> 8;
#pragma unroll 1
          for (int sg = 0; sg < nseg; ++sg)
            *reinterpret_cast<uint4*>(S + tiled_at(r, c + sg * ks, k, cr)) = ((split >> sg) & 1) ? low : high;
        }
      }
    }
  }
  // the shadow is read by bulk copies (the async proxy) of other CTAs
  asm volatile("fence.proxy.async.global;" ::: "memory");
  __syncthreads();
}

__device__ __forceinline__ void mbar_init(uint32_t addr, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(addr), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t addr) {
  asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.shared::cta.b64 st, [%0];\n}\n" ::"r"(addr) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t addr, uint32_t bytes) {
  asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}\n" ::"r"(addr),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
// bounded wait that also gives up when another role of the CTA has given up
__device__ __forceinline__ bool mbar_wait_or_abort(uint32_t addr, uint32_t phase, long long limit_ns,
                                                   volatile int* abort) {
  const unsigned long long t0 = gtimer_ns();
  for (;;) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(addr), "r"(phase)
        : "memory");
    if (done) return true;
    if (*abort) return false;
    if ((long long)(gtimer_ns() - t0) > limit_ns) {
      *abort = 1;
      return false;
    }
  }
}
__device__ __forceinline__ void tc_mma_bf16(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
      "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void red_add_f64(double* p, double v) {
  asm volatile("red.relaxed.gpu.global.add.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}

// C[r][lane] = beta C + alpha T[r][lane] for the warp's 32 rows (row stride ldc), T the 32 x 32
// FP32 transpose buffer (row stride 33).  With beta = 1 and alpha = +-1 (every Schur update) the
// sum goes to the L2 as a fire-and-forget FP64 reduction: one rounding of C + alpha T, the value
// fma(alpha, T, C) gives, with no load latency on the epilogue's path.  Otherwise 32 coalesced
// loads in flight per lane, then the stores.
__device__ __noinline__ void bg_rows_update(double* __restrict__ cp, int ldc, const float* tb, int lane, double alpha,
                                            double beta) {
  if (beta == 1.0 && (alpha == 1.0 || alpha == -1.0)) {
#pragma unroll
    for (int rr = 0; rr < 32; ++rr) red_add_f64(cp + (size_t)rr * ldc, alpha * (double)tb[rr * 33 + lane]);
    return;
  }
  double cv[32];
#pragma unroll
  for (int rr = 0; rr < 32; ++rr) cv[rr] = beta != 0.0 ? __ldcg(cp + (size_t)rr * ldc) : 0.0;
#pragma unroll
  for (int rr = 0; rr < 32; ++rr) cp[(size_t)rr * ldc] = fma(alpha, (double)tb[rr * 33 + lane], beta * cv[rr]);
}

// the same for two adjacent 32-column pieces (buffers T and T + 32 x 33): 64 loads in flight
__device__ __noinline__ void bg_rows_update2(double* __restrict__ cp, int ldc, const float* tb, int lane, double alpha,
                                             double beta) {
  if (beta == 1.0 && (alpha == 1.0 || alpha == -1.0)) {
#pragma unroll
    for (int rr = 0; rr < 32; ++rr) {
      red_add_f64(cp + (size_t)rr * ldc, alpha * (double)tb[rr * 33 + lane]);
      red_add_f64(cp + (size_t)rr * ldc + 32, alpha * (double)tb[32 * 33 + rr * 33 + lane]);
    }
    return;
  }
  double cv[64];
#pragma unroll
  for (int rr = 0; rr < 32; ++rr) {
    cv[rr] = beta != 0.0 ? __ldcg(cp + (size_t)rr * ldc) : 0.0;
    cv[32 + rr] = beta != 0.0 ? __ldcg(cp + (size_t)rr * ldc + 32) : 0.0;
  }
#pragma unroll
  for (int rr = 0; rr < 32; ++rr) {
    cp[(size_t)rr * ldc] = fma(alpha, (double)tb[rr * 33 + lane], beta * cv[rr]);
    cp[(size_t)rr * ldc + 32] = fma(alpha, (double)tb[32 * 33 + rr * 33 + lane], beta * cv[32 + rr]);
  }
}

// With a second pair (As2, Bs2, inner dimension k2 > 0) the k loop runs over the chunks of both
// pairs into the same accumulator: C := beta C + alpha (A B + A2 B2), one pass over C.
__device__ __noinline__ bool dev_gemm_bf16(double* __restrict__ C, int ldc, const uint8_t* __restrict__ As,
                                           const uint8_t* __restrict__ Bs, int m, int n, int k, double alpha,
                                           double beta, double* smem, TcCtx& tc, const uint8_t* __restrict__ As2,
                                           const uint8_t* __restrict__ Bs2, int k2) {
  uint8_t* sbase = reinterpret_cast<uint8_t*>(smem);
  const uint32_t s0 = smem_u32(sbase);
  const uint32_t stage0 = (s0 + 1023u) & ~1023u;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int kchunks = k >> 6, kchunks2 = k2 >> 6, nch = kchunks + kchunks2;
  // tile width: 256 (two 128-column MMAs) when n is a multiple of 256, else n itself (32, 64, 128:
  // one MMA of that width reading the first n rows of one B chunk)
  const int tw = (n % BG_TILE_N == 0) ? BG_TILE_N : n, nbc = tw > 128 ? 2 : 1;
  const int tiles_n = n / tw, tiles = (m >> 7) * tiles_n;
  // B chunks of cb_rows rows (the B shadow's chunk height: 128, or n itself below 128)
  const int cb_rows = tw > 128 ? 128 : tw;
  const uint32_t b_chunk = (uint32_t)cb_rows * 128u, b_lbo = (uint32_t)cb_rows * 16u;
  const uint32_t stage_bytes = BG_CHUNK + (uint32_t)nbc * b_chunk;
  const uint32_t idesc = kIdescBf16Base | ((uint32_t)((tw > 128 ? 128 : tw) >> 3) << 17);
  volatile int* abort = tc.abort;
  if (tid == 0) *abort = 0;
  // shared memory written by earlier tasks (generic proxy) is overwritten by bulk copies
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  auto full = [&](uint32_t s) { return tc.bars + 8u * s; };
  auto empty = [&](uint32_t s) { return tc.bars + 8u * (BG_STAGES + s); };
  auto tfull = [&](uint32_t b) { return tc.bars + 8u * (2 * BG_STAGES + b); };
  auto tempty = [&](uint32_t b) { return tc.bars + 8u * (2 * BG_STAGES + 2 + b); };
  if (warp == 0) {
    if (lane == 0) {  // producer
      // the shadows were written with ordinary stores by other CTAs (acquired through the
      // dependency counters); order them before this thread's bulk copies read them
      asm volatile("fence.proxy.async.global;" ::: "memory");
      uint32_t q = tc.q;
      for (int t = 0; t < tiles && !*abort; ++t) {
        const int rb = (t / tiles_n), cb = (t % tiles_n) * nbc;
        for (int kc = 0; kc < nch; ++kc, ++q) {
          const uint32_t s = q % BG_STAGES, ph = (q / BG_STAGES) & 1u;
          if (!mbar_wait_or_abort(empty(s), ph ^ 1u, tc.limit, abort)) break;
          const uint32_t dst = stage0 + s * BG_STAGE_BYTES;
          mbar_expect_tx(full(s), stage_bytes);
          const bool first = kc < kchunks;  // chunk of the first pair, else of the second
          const uint8_t* a = first ? As : As2;
          const uint8_t* b = first ? Bs : Bs2;
          const int kcp = first ? kc : kc - kchunks, kch = first ? kchunks : kchunks2;
          bulk_g2s(dst, a + ((size_t)rb * kch + kcp) * BG_CHUNK, BG_CHUNK, full(s));
          bulk_g2s(dst + BG_CHUNK, b + ((size_t)cb * kch + kcp) * b_chunk, b_chunk, full(s));
          if (nbc == 2)
            bulk_g2s(dst + BG_CHUNK + b_chunk, b + ((size_t)(cb + 1) * kch + kcp) * b_chunk, b_chunk, full(s));
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {  // MMA issuer
      uint32_t q = tc.q, u = tc.u;
      for (int t = 0; t < tiles && !*abort; ++t, ++u) {
        const uint32_t b = u & 1u;
        if (!mbar_wait_or_abort(tempty(b), ((u >> 1) & 1u) ^ 1u, tc.limit, abort)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc0 = tc.tmem + b * BG_TILE_N;
        bool ok = true;
        for (int kc = 0; kc < nch; ++kc, ++q) {
          const uint32_t s = q % BG_STAGES, ph = (q / BG_STAGES) & 1u;
          if (!mbar_wait_or_abort(full(s), ph, tc.limit, abort)) { ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a = stage0 + s * BG_STAGE_BYTES;
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
            const uint32_t acc = (kc > 0 || ks > 0) ? 1u : 0u;
            const uint64_t ad = umma_desc(a + ks * 4096u, 2048u, 128u);
            tc_mma_bf16(acc0, ad, umma_desc(a + BG_CHUNK + ks * 2u * b_lbo, b_lbo, 128u), idesc, acc);
            if (nbc == 2)
              tc_mma_bf16(acc0 + 128u, ad, umma_desc(a + BG_CHUNK + b_chunk + ks * 2u * b_lbo, b_lbo, 128u), idesc,
                          acc);
          }
          tc_commit(empty(s));  // the stage is free once these MMAs have read it
        }
        if (!ok) break;
        tc_commit(tfull(b));  // the accumulator tile is complete
      }
    }
  } else if (warp >= 4) {  // epilogue
    // per warp two 32 x 32 FP32 transpose buffers (row stride 33: conflict-free both ways): the
    // warp reads its 32 accumulator rows from TMEM (a thread per row), then updates C a row at a
    // time with the lanes along the columns, so every load and store of C is coalesced; two
    // 32-column pieces at a time, so each lane has 64 loads of C in flight
    const int qd = warp & 3;
    float* tb = reinterpret_cast<float*>(sbase + (stage0 - s0) + BG_STAGES * BG_STAGE_BYTES) + qd * (2 * 32 * 33);
    uint32_t u = tc.u;
    for (int t = 0; t < tiles; ++t, ++u) {
      const uint32_t b = u & 1u;
      const bool ok = mbar_wait_or_abort(tfull(b), (u >> 1) & 1u, tc.limit, abort);
      if (__any_sync(0xffffffffu, !ok)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int i0 = (t / tiles_n) << 7, j0 = (t % tiles_n) * tw;
      double* cblk = C + (size_t)(i0 + 32 * qd) * ldc + j0 + lane;
      const int pieces = tw / 32;
#pragma unroll 1
      for (int p = 0; p < pieces; p += 2) {
        const int np = pieces - p >= 2 ? 2 : 1;
        for (int h = 0; h < np; ++h) {
          uint32_t v[32];
          const uint32_t taddr = tc.tmem + ((uint32_t)(32 * qd) << 16) + b * BG_TILE_N + 32u * (p + h);
          asm volatile(
              "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
              "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
              : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]),
                "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]),
                "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
              : "r"(taddr)
              : "memory");
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          float* th = tb + h * (32 * 33);
#pragma unroll
          for (int c = 0; c < 32; ++c) th[lane * 33 + c] = __uint_as_float(v[c]);
        }
        __syncwarp();
        if (np == 2) bg_rows_update2(cblk + 32 * p, ldc, tb, lane, alpha, beta);
        else bg_rows_update(cblk + 32 * p, ldc, tb, lane, alpha, beta);
        __syncwarp();
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty(b));
    }
  }
  __syncthreads();
  const bool ok = !*abort;
  // every thread advances the pipeline counters alike (the next BF16 task continues the phases)
  tc.q += (uint32_t)(tiles * nch);
  tc.u += (uint32_t)tiles;
  if (!ok) tc.pending = 1;
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  return ok;
}

// Estimates from the special-function unit: PTX rsqrt.approx.ftz.f64 / rcp.approx.ftz.f64
// (computed from the upper word of the double, about single-precision accuracy, full double
// exponent range; zero gives infinity).
__device__ __forceinline__ double rsqrt_est(double v) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(v));
  return y;
}
__device__ __forceinline__ double rcp_est(double v) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(v));
  return y;
}
// ------------------------------------------------------------------------- quotients
// A division takes 128 cycles of dependent work on this chip, and the triangular routines have one
// per row on their critical path.  These are the same correctly rounded quotients from published
// iterations (P. Markstein, Computation of elementary functions on the IBM RISC System/6000, 1990):
// a reciprocal estimate (special-function unit, about 20 bits) is brought to RN(1 / t) by a
// third-order and a second-order step, and with y = RN(1 / t) two corrections q += (x - t q) y of
// q = RN(x y), the residual exact in an fma, leave RN(x / t), as long as nothing over- or underflows.
// quotient_unsafe: exponents for which that may not hold (a positive zero is fine); the routines fall
// back to divisions then.  Compared with `/` on 2^32 random pairs: no difference.
__device__ __forceinline__ double reciprocal(double t, double y) {  // y: rcp_est(t)
  const double e = fma(-t, y, 1.0);
  y = fma(y, fma(e, e, e), y);
  return fma(fma(-t, y, 1.0), y, y);
}
__device__ __forceinline__ double reciprocal(double t) { return reciprocal(t, rcp_est(t)); }
__device__ __forceinline__ double quotient(double x, double t, double y) {
  double q = x * y;
  q = fma(fma(-q, t, x), y, q);
  return fma(fma(-q, t, x), y, q);
}
__device__ __forceinline__ int quotient_unsafe(double x, double t) {  // without branches
  const int hx = __double2hiint(x), lx = __double2loint(x), ht = __double2hiint(t), lt = __double2loint(t);
  const int ex = (int)((unsigned)((hx >> 20) & 0x7FF) - 600u >= 846u), et = (int)((unsigned)((ht >> 20) & 0x7FF) - 600u >= 846u);
  // the all-ones mantissa is the one divisor whose reciprocal the last step may not round right
  const int ones = (int)(((ht | 0xFFF00000) & lt) == -1);
  return et | ones | (ex & (int)((hx | lx) != 0));
}

// ------------------------------------------------------------------------- GETRF
#define GETRF_LD (TL + 3)  /* odd: lanes along rows and fragments both nearly free of bank conflicts */
// the whole block with divisions, for values out of the quotients' range
__device__ __noinline__ void getrf_by_division(double* A, int lda, int m, int n) {
  extern __shared__ __align__(16) double vm_smem[];
  double* S = vm_smem;
  const int tid = threadIdx.x;
  for (int e = tid; e < m * n; e += NT) S[(e / n) * GETRF_LD + e % n] = ldcg(&A[(size_t)(e / n) * lda + e % n]);
  __syncthreads();
  for (int i = 0; i < min(m, n); ++i) {
    const double* u = S + i * GETRF_LD;
    for (int r = i + 1 + tid; r < m; r += NT) S[r * GETRF_LD + i] = S[r * GETRF_LD + i] / u[i];
    __syncthreads();
    for (int e = tid; e < (m - i - 1) * (n - i - 1); e += NT) {
      double* x = S + (i + 1 + e / (n - i - 1)) * GETRF_LD;
      const int c = i + 1 + e % (n - i - 1);
      x[c] = fma(u[c], -x[i], x[c]);
    }
    __syncthreads();
  }
  for (int e = tid; e < m * n; e += NT) A[(size_t)(e / n) * lda + e % n] = S[(e / n) * GETRF_LD + e % n];
}

// A[m x n] := L\U in place (m, n <= TL), like kernel.cu:104-147: step i divides the entries below the
// pivot by a_ii and applies a_rc = fma(a_ic, -l_r, a_rc) to the trailing block.
//
// The block stays in shared memory, eight columns per warp.  When a panel of eight is factored, the warp
// of the next one applies it to its columns and factors them, two rows per lane, while the warps
// further right solve their eight rows against it and update the rows below on the FP64 tensor cores (a
// chain of fma in ascending i, see dmma): one CTA barrier per eight steps.  A lane's row moves one place
// to the left in its registers with each step, so that the steps are one loop: beside SMs that load the
// memory system, what the instruction costs is its code's way here (the unrolled form before, with
// a barrier and a division per step: 20 us alone, 56 us beside the products of a mixed-precision
// factorization).  What bounds it is a step's chain: shuffle, reciprocal, quotient, update.
// 64 x 64 on a B200, hop included: 20.4 -> 18.2 us alone, 56 -> 21 us there.
__device__ __forceinline__ void dev_getrf(double* A, int lda, int m, int n) {
  extern __shared__ __align__(16) double vm_smem[];
  double* S = vm_smem;  // TL x GETRF_LD (and a panel's width of reads past its end)
  const int tid = thread_index(), warp = tid >> 5, lane = tid & 31, fa = lane >> 2, fb = lane & 3;
  const int mn = min(m, n), panels = (mn + 7) >> 3, cg = 8 * warp;
  int bad = 0;
  {
    const int c = tid & 63;
    if (c < n) {
#pragma unroll 4
      for (int r = tid >> 6; r < m; r += NT / 64) cp_async8(smem_u32(S + r * GETRF_LD + c), A + (size_t)r * lda + c, 8u);
    }
    cp_async_commit();
    cp_async_wait<0>();
  }
  __syncthreads();
#pragma unroll 1
  for (int J = -1; J < panels; ++J) {
    const int c0 = 8 * J;
    const bool next = warp == J + 1 && warp < panels;
    if (J >= 0 && cg < n && warp > J && !next) {
      // rows c0 .. c0 + 7 of these columns: solve against the panel's unit lower triangle
      double* u = S + (c0 + fa) * GETRF_LD;
      double x0 = u[cg + 2 * fb], x1 = u[cg + 2 * fb + 1], c = u[c0];
#pragma unroll 1
      for (int i = 0; i < 7; ++i) {
        const double v0 = __shfl_sync(0xffffffffu, x0, 4 * i + fb), v1 = __shfl_sync(0xffffffffu, x1, 4 * i + fb);
        const double y0 = fma(v0, -c, x0), y1 = fma(v1, -c, x1);
        c = u[c0 + i + 1];
        x0 = fa > i ? y0 : x0;
        x1 = fa > i ? y1 : x1;
      }
      u[cg + 2 * fb] = x0;
      u[cg + 2 * fb + 1] = x1;
      __syncwarp();
      const double b0 = S[(c0 + fb) * GETRF_LD + cg + fa], b1 = S[(c0 + 4 + fb) * GETRF_LD + cg + fa];
#pragma unroll 4
      for (int t = c0 + 8; t < m; t += 8) {  // tiles of eight rows; rows past m stay inside S
        double* p = S + (t + fa) * GETRF_LD;
        double y0 = p[cg + 2 * fb], y1 = p[cg + 2 * fb + 1];
        dmma(y0, y1, -p[c0 + fb], b0);
        dmma(y0, y1, -p[c0 + 4 + fb], b1);
        p[cg + 2 * fb] = y0;
        p[cg + 2 * fb + 1] = y1;
      }
      __syncwarp();
    }
    if (next) {  // the next panel, in rows: this panel's steps applied to it, then its own
      const int w = min(8, n - cg), steps = min(8, mn - cg), r0 = max(c0, 0), off = cg - r0;
      const int ra = min(r0 + lane, TL - 1), rb = min(r0 + lane + 32, TL - 1);
      double x[2][8];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        x[0][c] = S[ra * GETRF_LD + cg + c];
        x[1][c] = S[rb * GETRF_LD + cg + c];
      }
      double la = S[ra * GETRF_LD + r0], lb = S[rb * GETRF_LD + r0];
#pragma unroll 1
      for (int i = 0; i < off; ++i) {
        double* row = S + (r0 + i) * GETRF_LD + cg;  // becomes a row of U
#pragma unroll
        for (int c = 0; c < 8; ++c) sts_if(row + c, x[0][c], lane == i && c < w);
        __syncwarp();
        double u[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) u[c] = row[c];
        const double na = -la, nb = -lb;
        la = S[ra * GETRF_LD + r0 + i + 1];
        lb = S[rb * GETRF_LD + r0 + i + 1];
#pragma unroll
        for (int c = 0; c < 8; ++c) {  // lanes up to i have their row of U in place: of no consequence
          x[0][c] = fma(u[c], na, x[0][c]);
          x[1][c] = fma(u[c], nb, x[1][c]);
        }
      }
#pragma unroll 1
      for (int i = 0; i < steps; ++i) {
        double* row = S + (cg + i) * GETRF_LD + cg + i;
        const double p = __shfl_sync(0xffffffffu, x[0][0], off + i), seed = rcp_est(p);
#pragma unroll
        for (int c = 0; c < 8; ++c) sts_if(row + c, x[0][c], lane == off + i && c < w - i);
        __syncwarp();
        double u[8];
#pragma unroll
        for (int c = 1; c < 8; ++c) u[c] = row[c];  // past the panel: of no consequence
        const double y = reciprocal(p, seed);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = r0 + lane + 32 * h, below = (int)(lane + 32 * h > off + i) & (int)(r < m);
          const double l = quotient(x[h][0], p, y);
          bad |= below & quotient_unsafe(x[h][0], p);
          sts_if(S + (h ? rb : ra) * GETRF_LD + cg + i, l, below);
#pragma unroll
          for (int c = 1; c < 8; ++c) x[h][c - 1] = fma(u[c], -l, x[h][c]);
        }
      }
    }
    __syncthreads();
  }
  if (__syncthreads_or(bad)) {
    getrf_by_division(A, lda, m, n);
  } else {
    const int c = tid & 63;
    if (c < n)
#pragma unroll 4
      for (int r = tid >> 6; r < m; r += NT / 64) A[(size_t)r * lda + c] = S[r * GETRF_LD + c];
  }
  __syncthreads();
}

// A[m x n] := L\U of P A with partial pivoting inside the block (m, n <= TL), P written to Pout (m
// doubles of row indices).  Step i first swaps whole rows i and r, r >= i the row of largest |a_ri|
// (the first of equal ones), then eliminates as the unpivoted routine does, so a block that needs
// no swap gets the same bits.
//
// The block stays in shared memory, eight columns per warp.  The warp of a column group factors it
// (two rows per lane, which stay where they are: only their positions are swapped), then the warps
// of the groups to the right solve their eight rows against it and update the rows below on the
// FP64 tensor cores (a chain of fma in ascending i, see dmma); the next group's warp goes on to
// factor it while the others still update.  One CTA barrier per eight steps; the instructions of
// the one warp that factors bound it.  64 x 64, hop included: 80 -> 41 us (before: the whole block
// in shared memory with four CTA barriers per step).
// the pivot of step ci among the rows at positions >= ci (a lane's two rows: values v0, v1 at
// positions pos): lane pl, half ph; swaps the positions of the pivot row and of the row at ci
__device__ __forceinline__ void getrf_pivot(double v0, double v1, int (&pos)[2], int ci, int m, int& pl, int& ph) {
  double best = -1.0;
  int bp = ci;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const double v = fabs(h ? v1 : v0);
    if (pos[h] >= ci && pos[h] < m && (v > best || (v == best && pos[h] < bp))) {
      best = v;
      bp = pos[h];
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int op = __shfl_xor_sync(0xffffffffu, bp, o);
    if (ov > best || (ov == best && op < bp)) {
      best = ov;
      bp = op;
    }
  }
  const unsigned h0 = __ballot_sync(0xffffffffu, pos[0] == bp), h1 = __ballot_sync(0xffffffffu, pos[1] == bp);
  pl = __ffs((int)(h0 | h1)) - 1;
  ph = h1 != 0u;
#pragma unroll
  for (int h = 0; h < 2; ++h) pos[h] = pos[h] == bp ? ci : pos[h] == ci ? bp : pos[h];
}

// a panel with divisions, in shared memory, for values out of the quotients' range (rows stay where
// they are, pos gives their positions)
__device__ __noinline__ void getrf_panel_by_division(double* S, int cg, int m, int w, int steps, int (&pos)[2],
                                                     int lane) {
#pragma unroll
  for (int h = 0; h < 2; ++h) pos[h] = cg + lane + 32 * h;
  double* r0 = S + min(cg + lane, TL - 1) * GETRF_LD + cg;
  double* r1 = S + min(cg + lane + 32, TL - 1) * GETRF_LD + cg;
#pragma unroll 1
  for (int i = 0; i < steps; ++i) {
    const int ci = cg + i;
    int pl, ph;
    getrf_pivot(r0[i], r1[i], pos, ci, m, pl, ph);
    const double* pr = S + (cg + pl + 32 * ph) * GETRF_LD + cg;
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      double* r = h ? r1 : r0;
      if (cg + lane + 32 * h < m && (h ? pos[1] : pos[0]) > ci) {
        const double l = r[i] / pr[i];
        r[i] = l;
        for (int c = i + 1; c < w; ++c) r[c] = fma(pr[c], -l, r[c]);
      }
    }
    __syncwarp();
  }
}

__device__ __forceinline__ void dev_getrf_piv(double* A, int lda, int m, int n, double* Pout) {
  extern __shared__ __align__(16) double vm_smem[];
  double* S = vm_smem;                                         // TL x GETRF_LD
  int* from = reinterpret_cast<int*>(S + TL * GETRF_LD);       // [2][TL]: row now at p was at from[p] before the panel
  int* perm = from + 2 * TL;                                   // row at p came from row perm[p] of A
  const int tid = thread_index(), warp = tid >> 5, lane = tid & 31, fa = lane >> 2, fb = lane & 3;
  const int mn = min(m, n), panels = (mn + 7) >> 3;
  {
    const int c = tid & 63;
    if (c < n) {
#pragma unroll 4
      for (int r = tid >> 6; r < m; r += NT / 64) cp_async8(smem_u32(S + r * GETRF_LD + c), A + (size_t)r * lda + c, 8u);
    }
    cp_async_commit();
    cp_async_wait<0>();
    if (tid < TL) perm[tid] = tid;
  }
  __syncthreads();
#pragma unroll 1
  for (int J = -1; J < panels; ++J) {
    const int c0 = 8 * J, cg = 8 * warp;
    if (J >= 0 && cg < n && warp != J) {
      {  // the panel's row swaps, applied to this warp's columns
        const int* f = from + (J & 1) * TL;
        double x[8][2];
#pragma unroll
        for (int t = 0; t < 8; ++t) {
          const int r = min(8 * t + fa, m - 1), sr = r < c0 ? r : f[r];
          x[t][0] = S[sr * GETRF_LD + cg + 2 * fb];
          x[t][1] = S[sr * GETRF_LD + cg + 2 * fb + 1];
        }
        __syncwarp();
#pragma unroll
        for (int t = 0; t < 8; ++t) {
          const int r = 8 * t + fa;
          if (r < m) {
            S[r * GETRF_LD + cg + 2 * fb] = x[t][0];
            S[r * GETRF_LD + cg + 2 * fb + 1] = x[t][1];
          }
        }
        __syncwarp();
      }
      if (warp > J) {
        // rows c0 .. c0 + 7 of these columns: solve against the panel's unit lower triangle
        double* u = S + (c0 + fa) * GETRF_LD;
        double x0 = u[cg + 2 * fb], x1 = u[cg + 2 * fb + 1];
#pragma unroll
        for (int i = 0; i < 7; ++i) {
          const double v0 = __shfl_sync(0xffffffffu, x0, 4 * i + fb), v1 = __shfl_sync(0xffffffffu, x1, 4 * i + fb);
          const double c = u[c0 + i];
          const double y0 = fma(v0, -c, x0), y1 = fma(v1, -c, x1);
          x0 = fa > i ? y0 : x0;
          x1 = fa > i ? y1 : x1;
        }
        u[cg + 2 * fb] = x0;
        u[cg + 2 * fb + 1] = x1;
        __syncwarp();
        const double b0 = S[(c0 + fb) * GETRF_LD + cg + fa], b1 = S[(c0 + 4 + fb) * GETRF_LD + cg + fa];
#pragma unroll 2
        for (int r = c0 + 8 + fa; r < m + fa; r += 8) {  // tiles of eight rows; rows past m stay inside S
          double* p = S + r * GETRF_LD;
          double y0 = p[cg + 2 * fb], y1 = p[cg + 2 * fb + 1];
          dmma(y0, y1, -p[c0 + fb], b0);
          dmma(y0, y1, -p[c0 + 4 + fb], b1);
          p[cg + 2 * fb] = y0;
          p[cg + 2 * fb + 1] = y1;
        }
        __syncwarp();
      }
    }
    if (warp == J + 1 && warp < panels) {  // factor the next panel: columns cg .., rows cg ..
      const int w = min(8, n - cg), steps = min(8, mn - cg);
      double x[2][8];
      int pos[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        pos[h] = cg + lane + 32 * h;
#pragma unroll
        for (int c = 0; c < 8; ++c) x[h][c] = (pos[h] < m && c < w) ? S[pos[h] * GETRF_LD + cg + c] : 0.0;
      }
      int bad = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int ci = cg + i;
        int pl = i, ph = 0;
        if (i < steps) getrf_pivot(x[0][i], x[1][i], pos, ci, m, pl, ph);
        double u[8];
#pragma unroll
        for (int c = i; c < 8; ++c) u[c] = __shfl_sync(0xffffffffu, ph ? x[1][c] : x[0][c], pl);
        const double y = reciprocal(u[i]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int below = (int)(i < steps) & (int)(pos[h] > ci) & (int)(pos[h] < m);
          const double l = quotient(x[h][i], u[i], y);
          bad |= below & quotient_unsafe(x[h][i], u[i]);
          x[h][i] = below ? l : x[h][i];
#pragma unroll
          for (int c = i + 1; c < 8; ++c) {
            const double v = fma(u[c], -l, x[h][c]);
            x[h][c] = below ? v : x[h][c];
          }
        }
      }
      if (__any_sync(0xffffffffu, bad)) {
        getrf_panel_by_division(S, cg, m, w, steps, pos, lane);
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int c = 0; c < 8; ++c)
            if (cg + lane + 32 * h < m && c < w) x[h][c] = S[(cg + lane + 32 * h) * GETRF_LD + cg + c];
        __syncwarp();
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int row = cg + lane + 32 * h;
        if (row < m) {
#pragma unroll
          for (int c = 0; c < 8; ++c)
            if (c < w) S[pos[h] * GETRF_LD + cg + c] = x[h][c];
          from[((J + 1) & 1) * TL + pos[h]] = row;
        }
      }
      {
        __syncwarp();
        int v[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int p = lane + 32 * h;
          v[h] = p < m ? perm[p < cg ? p : from[((J + 1) & 1) * TL + p]] : 0;
        }
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 2; ++h)
          if (lane + 32 * h < m) perm[lane + 32 * h] = v[h];
      }
    }
    __syncthreads();
  }
  {
    const int c = tid & 63;
    if (c < n)
#pragma unroll 4
      for (int r = tid >> 6; r < m; r += NT / 64) A[(size_t)r * lda + c] = S[r * GETRF_LD + c];
    for (int i = tid; i < m; i += NT) Pout[i] = (double)perm[i];
  }
  __syncthreads();
}

// ------------------------------------------------------------------------- triangular solves
// TRSMR's eight positions of a block against each other with divisions, for values out of the
// quotients' range (a call: beside it in one loop the compiler's code for the usual case is three
// times slower).  w: the lane's row of coefficients within the block.
__device__ __noinline__ double2 tri_by_division(double x0, double x1, double tii, const double* w, int lane) {
  const int fa = lane >> 2, fb = lane & 3;
#pragma unroll 1
  for (int i = 0; i < 8; ++i) {
    const double v0 = __shfl_sync(0xffffffffu, x0 / tii, 4 * i + fb), v1 = __shfl_sync(0xffffffffu, x1 / tii, 4 * i + fb);
    const double c = w[i], y0 = fma(-c, v0, x0), y1 = fma(-c, v1, x1);
    x0 = fa > i ? y0 : fa == i ? v0 : x0;
    x1 = fa > i ? y1 : fa == i ? v1 : x1;
  }
  return make_double2(x0, x1);
}

// Triangular solve with one triangle of len <= TL rows, in place on `lines` independent lines of B:
// the columns of B for TRSML / TRSMRT / TRSMU, the rows for TRSMR.  Position i of a line is solved,
// then x_p = fma(-coef(i, p), x_i, x_p) for the later ones, i ascending (descending for TRSMU):
//   TRSML   coef T[p][i], unit diagonal            (kernel.cu:150-182; perm: B's rows permuted first)
//   TRSMRT  coef T[i][p], x_i = x_i * (1 / t_ii)   (kernel.cu:229-285)
//   TRSMR   coef T[i][p], x_i = x_i / t_ii         (kernel.cu:185-226)
//   TRSMU   coef T[p][i], x_i = x_i * (1 / t_ii), from the last position to the first
// The coefficients are staged as W[p][i] (for TRSMU with positions counted from the end, so that
// every kind runs forward), a warp takes eight lines and needs no other warp from there on.  Eight
// positions at a time: the sum over the earlier positions on the FP64 tensor cores (a chain of fma
// in ascending i, see dmma), then the eight against each other with shuffles (about 40 cycles a
// position, 140 with a quotient), which bounds it.  On a B200, hop to the next task included (before: a
// shuffled sweep over all 64 positions, unrolled, its coefficients fetched step by step):
//   64 x 64: TRSML 18 -> 10.5 us, TRSMR 22.5 -> 14 us;  TRSML 256 x 64: 148 -> 61 us
#define TRI_LDX 12  /* doubles between positions of a warp's lines: 4 mod 8, no bank conflicts */
__device__ __forceinline__ void dev_tri(int op, double* B, int ldb, const double* T, int ldt, int len, int lines,
                                        const double* perm) {
  extern __shared__ __align__(16) double vm_smem[];
  double* W = vm_smem;                // TL x GM_LD
  double* rd = W + TL * GM_LD;        // reciprocals of the diagonal
  const int tid = thread_index(), warp = tid >> 5, lane = tid & 31, fa = lane >> 2, fb = lane & 3;
  double* X = rd + TL + warp * (TL * TRI_LDX);
  const bool ct = op == PP_OP_TRSMR || op == PP_OP_TRSMRT, back = op == PP_OP_TRSMU, byrow = op == PP_OP_TRSMR;
  const size_t ps = byrow ? 1 : (size_t)ldb, ls = byrow ? (size_t)ldb : 1;
  {  // the triangle's half with i <= p, element (r, c) of T at (p, i)
    const int c = tid & 63;
#pragma unroll 4
    for (int r = tid >> 6; r < len; r += NT / 64) {
      int p = ct ? c : r, i = ct ? r : c;
      if (back) { p = len - 1 - p; i = len - 1 - i; }
      if (c < len && i <= p) cp_async8(smem_u32(W + p * GM_LD + i), T + (size_t)r * ldt + c, 8u);
    }
  }
  bool first = true;
  for (int q0 = 8 * warp;; q0 += NT / 4) {
    const int nq = min(8, lines - q0);
    if (nq > 0) {
      // lanes along what is contiguous in B: the positions of a row, or the lines
      const int qs = byrow ? 1 : 32, p_step = byrow ? 32 : 4;
#pragma unroll 1
      for (int q = byrow ? 0 : lane & 7; q < nq; q += qs)
#pragma unroll 4
        for (int p = byrow ? lane : lane >> 3; p < len; p += p_step) {
          int src = back ? len - 1 - p : p;
          if (perm) {
            const int v = (int)ldcg(&perm[p]);
            src = (v >= 0 && v < len) ? v : p;  // indices come from the block's GETRF; guard anyway
          }
          cp_async8(smem_u32(X + p * TRI_LDX + q), B + (size_t)(q0 + q) * ls + (size_t)src * ps, 8u);
        }
    }
    cp_async_commit();
    cp_async_wait<0>();
    if (first) {
      __syncthreads();
      if (tid < len) rd[tid] = 1.0 / W[tid * GM_LD + tid];
      __syncthreads();
      first = false;
    }
    __syncwarp();
    if (nq <= 0) break;
#pragma unroll 1
    for (int t = 0; t < len; t += 8) {
      double x0 = X[(t + fa) * TRI_LDX + 2 * fb], x1 = X[(t + fa) * TRI_LDX + 2 * fb + 1];
      const double* w = W + (t + fa) * GM_LD;
#pragma unroll 2
      for (int j = 0; j < t; j += 8) {
        const double a0 = -w[j + fb], a1 = -w[j + 4 + fb];
        const double b0 = X[(j + fb) * TRI_LDX + fa], b1 = X[(j + 4 + fb) * TRI_LDX + fa];
        dmma(x0, x1, a0, b0);
        dmma(x0, x1, a1, b1);
      }
      const double mine = rd[t + fa], tii = w[t + fa];
      if (op == PP_OP_TRSMR) {
        const double s0 = x0, s1 = x1;
        int bad = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          bad |= (int)(fa == i) & (quotient_unsafe(x0, tii) | quotient_unsafe(x1, tii));
          const double v0 = __shfl_sync(0xffffffffu, quotient(x0, tii, mine), 4 * i + fb);
          const double v1 = __shfl_sync(0xffffffffu, quotient(x1, tii, mine), 4 * i + fb);
          const double c = w[t + i], y0 = fma(-c, v0, x0), y1 = fma(-c, v1, x1);
          x0 = fa > i ? y0 : fa == i ? v0 : x0;
          x1 = fa > i ? y1 : fa == i ? v1 : x1;
        }
        if (__any_sync(0xffffffffu, bad & (int)(t + fa < len))) {
          const double2 r = tri_by_division(s0, s1, tii, w + t, lane);
          x0 = r.x;
          x1 = r.y;
        }
      } else {
        const double f = op == PP_OP_TRSML ? 1.0 : mine;  // a product with 1 changes nothing
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const double v0 = __shfl_sync(0xffffffffu, x0 * f, 4 * i + fb);
          const double v1 = __shfl_sync(0xffffffffu, x1 * f, 4 * i + fb);
          const double c = w[t + i], y0 = fma(-c, v0, x0), y1 = fma(-c, v1, x1);
          x0 = fa > i ? y0 : fa == i ? v0 : x0;
          x1 = fa > i ? y1 : fa == i ? v1 : x1;
        }
      }
      __syncwarp();
      X[(t + fa) * TRI_LDX + 2 * fb] = x0;
      X[(t + fa) * TRI_LDX + 2 * fb + 1] = x1;
      const int p = t + fa, dst = back ? len - 1 - p : p;
      double* o = B + (size_t)(q0 + 2 * fb) * ls + (size_t)dst * ps;
      st_if(o, x0, p < len && 2 * fb < nq);
      st_if(o + ls, x1, p < len && 2 * fb + 1 < nq);
      __syncwarp();
    }
  }
  __syncthreads();
}

// ------------------------------------------------------------------------- skinny products
// Rows of a matrix times a few right-hand sides: rows [0, rows) of M S into O, M's row r at M + r ldm
// (m columns), S m x n (n <= 16), O := beta O + alpha (M S).  tri 0: M lower triangular, tri 1: upper
// (diagonal included; row r of the call is row r0 + r of the triangle), tri 2: full.  O may be S.
// The explicit inverses of the leaves (TRMV) and the solves' products with a leaf or a low-rank
// factor: S is staged in shared memory, a warp takes eight rows of M at a time straight from global
// memory into FP64 tensor-core fragments, two columns per load (the k order is free: even columns in
// one chain, odd ones in another); nothing of a row depends on which other rows the call covers.  Bound
// by one CTA's loads and by the instructions around them: with the next 64 columns loading during the
// products it is no faster (10.4 k cycles either way at 64 x 8 x 512), and those registers cost every
// instruction of the VM 1% in spills.  On a B200, time of the task (before: warps along the columns, a
// shuffle reduction per row and right-hand side):
//   TRMV 128 x 4, 64 rows  11.5 -> 3.3 us   512 x 8, 64 rows  29 -> 7.5 us
//   products 64 x 8 x 512  42 -> 10.2 us   256 x 4 x 32  17 -> 4.9 us
// A fragment's zeros outside the triangle, or past the last column, would make NaN of an infinity or a
// NaN in S: with one there the product is summed entry by entry (rows_exact).
#define RW_U 8  /* steps of 8 columns whose loads go out together */
__device__ __noinline__ void rows_exact(double* O, int ldo, const double* M, int ldm, int ls, int m, int n, int rows,
                                        int tri, int r0, double alpha, double beta) {
  extern __shared__ __align__(16) double vm_smem[];
  for (int e = threadIdx.x; e < rows * n; e += NT) {
    const int r = e / n, q = e - r * n, end = tri == 0 ? r0 + r + 1 : m;
    double sum = 0.0;
    for (int c = tri == 1 ? r0 + r : 0; c < end; ++c) sum = fma(ldcg(&M[(size_t)r * ldm + c]), vm_smem[c * ls + q], sum);
    double* o = O + (size_t)r * ldo + q;
    *o = beta != 0.0 ? fma(alpha, sum, ldcg(o)) : alpha * sum;
  }
  __syncthreads();
}
__device__ __forceinline__ void dev_rows(double* O, int ldo, const double* M, int ldm, const double* S, int lds, int m,
                                         int n, int rows, int tri, int r0, double alpha, double beta) {
  extern __shared__ __align__(16) double vm_smem[];
  const int tid = thread_index(), warp = tid >> 5, lane = tid & 31, fa = lane >> 2, fb = lane & 3;
  const int ns = n <= 8 ? 8 : 16, ls = ns + 2, lm = (m + 7) & ~7;  // stride 2 mod 8: no bank conflicts
  int special = 0;
#pragma unroll 4
  for (int e = tid; e < lm * ns; e += NT) {
    const int r = n <= 8 ? e >> 3 : e >> 4, q = e & (ns - 1);
    const double v = ldcg_if(S + (size_t)r * lds + q, r < m && q < n);
    special |= (int)((__double2hiint(v) & 0x7FF00000) == 0x7FF00000);
    vm_smem[r * ls + q] = v;
  }
  const bool wide = !((ldm | (int)(reinterpret_cast<uintptr_t>(M) >> 3)) & 1);
  if (__syncthreads_or(special)) {
    rows_exact(O, ldo, M, ldm, ls, m, n, rows, tri, r0, alpha, beta);
    return;
  }
#pragma unroll 1
  for (int t = 8 * warp; t < rows; t += 64) {
    const int r = t + fa;
    const bool rin = r < rows;
    // columns the eight rows have entries in
    const int cb = tri == 1 ? (r0 + t) & ~7 : 0, ce = tri == 0 ? min(m, r0 + t + 8) : m;
    const double* row = M + (size_t)(rin ? r : 0) * ldm;
    double acc[2][2][2];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int j = 0; j < 2; ++j) acc[h][j][0] = acc[h][j][1] = 0.0;
    // a block of 64 columns in registers: even and odd columns of each step of 8
    auto load = [&](int c0, double (&v)[RW_U][2]) {
      const double* p = row + c0 + 2 * fb;
      if (wide && c0 + 8 * RW_U <= m) {
#pragma unroll
        for (int u = 0; u < RW_U; ++u) {
          const double2 x = __ldcg(reinterpret_cast<const double2*>(p + 8 * u));
          v[u][0] = x.x;
          v[u][1] = x.y;
        }
      } else {
#pragma unroll
        for (int u = 0; u < RW_U; ++u) {
          const int c = c0 + 8 * u + 2 * fb;
          v[u][0] = ldcg_if(p + 8 * u, c < m);
          v[u][1] = ldcg_if(p + 8 * u + 1, c + 1 < m);
        }
      }
    };
    double v[RW_U][2], old[2][2];
    load(cb, v);
    double* o = O + (size_t)r * ldo + 2 * fb;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) old[j][e] = ldcg_if(o + 8 * j + e, rin && 8 * j + 2 * fb + e < n && beta != 0.0);
#pragma unroll 1
    for (int c0 = cb; c0 < ce; c0 += 8 * RW_U) {
      if ((tri == 0 && c0 + 8 * RW_U > r0 + t) || (tri == 1 && c0 < r0 + t + 8)) {
        // what lies outside the triangle is not used as a value
#pragma unroll
        for (int u = 0; u < RW_U; ++u) {
          const int c = c0 + 8 * u + 2 * fb, d = r0 + r;
          v[u][0] = (tri == 0 ? c <= d : c >= d) ? v[u][0] : 0.0;
          v[u][1] = (tri == 0 ? c + 1 <= d : c + 1 >= d) ? v[u][1] : 0.0;
        }
      }
#pragma unroll
      for (int u = 0; u < RW_U; ++u) {
        const double* b = vm_smem + min(c0 + 8 * u + 2 * fb, lm - 2) * ls + fa;
        dmma(acc[0][0][0], acc[0][0][1], v[u][0], b[0]);
        dmma(acc[1][0][0], acc[1][0][1], v[u][1], b[ls]);
        if (n > 8) {
          dmma(acc[0][1][0], acc[0][1][1], v[u][0], b[8]);
          dmma(acc[1][1][0], acc[1][1][1], v[u][1], b[ls + 8]);
        }
      }
      if (c0 + 8 * RW_U < ce) load(c0 + 8 * RW_U, v);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        st_if(o + 8 * j + e, fma(alpha, acc[0][j][e] + acc[1][j][e], old[j][e]), rin && 8 * j + 2 * fb + e < n);
      }
  }
  __syncthreads();
}

// The same for one right-hand side, with FMAs: 4 columns per lane (adjacent, or a row's width apart where
// pairs are not aligned), 4 to 32 lanes along a row or along 128 columns of it, eight rows per lane at a
// time, from global memory; the eight sums are exchanged so that each lane ends with one (or two).  The
// tensor-core form above spends seven eighths of its work on columns that are not there, and its
// instructions are what such a product costs (about five cycles each, fetched for this task).  O may be
// S: it is read once, before a barrier, or kept in shared memory where it has more than 128 rows.  Cycles on a B200, the form above -> this one:
//   256 x 16  6100 -> 1650   111 x 24  3500 -> 1630   94 x 94 triangle  5600 -> 4400   111 x 111  6600 -> 4600
//   64 x 256  3200 -> 2500   256 x 256  18000 -> 15200
__device__ __forceinline__ void dev_column(double* O, int ldo, const double* M, int ldm, const double* S, int sr, int m,
                                           int rows, int tri, int r0, double alpha, double beta) {
  extern __shared__ __align__(16) double vm_smem[];
  const int tid = thread_index(), warp = tid >> 5, lane = tid & 31;
  const int lg = m <= 16 ? 2 : m <= 32 ? 3 : m <= 64 ? 4 : 5;  // log2 of the lanes per row
  const int cl = lane & ((1 << lg) - 1), rl = lane >> lg, step = 32 >> lg;
  const bool wide = !((ldm | m | (int)(reinterpret_cast<uintptr_t>(M) >> 3)) & 1), once = m <= 128, inplace = O == S;
  const int cs = wide ? 1 : 1 << lg;  // this lane's columns: c + e cs
  const int fin = 4 * (cl & 1) + (cl & 2) + (lg > 2 ? (cl >> 2) & 1 : 0);  // the first of the eight sums that stays here
  const bool staged = inplace && !once;
  if (staged) {
    for (int e = tid; e < m; e += NT) vm_smem[e] = ldcg(S + (size_t)e * sr);
    __syncthreads();
  }
  double s[4];
  bool first = true;
#pragma unroll 1
  for (int t = 8 * step * warp; t < rows || (first && inplace && once); t += 64 * step) {
    double v[8], old[2];
    const int r = t + rl + fin * step, end = once || tri != 0 ? m : min(m, r0 + t + 8);
    double* o = O + (size_t)r * ldo;
    old[0] = ldcg_if(o, beta != 0.0 && r < rows && cl < 8);
    old[1] = ldcg_if(o + (size_t)step * ldo, beta != 0.0 && lg == 2 && r + step < rows);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = 0.0;
#pragma unroll 1
    for (int c0 = once || tri != 1 ? 0 : (r0 + t) & ~127; c0 < end; c0 += 128) {
      const int c = c0 + (wide ? 4 * cl : cl);
      const double* p = M + (size_t)(t + rl) * ldm + c;
      double x[8][4];
      if (!once || first) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (staged) s[e] = c + e * cs < m ? vm_smem[c + e * cs] : 0.0;
          else s[e] = ldcg_if(S + (size_t)(c + e * cs) * sr, c + e * cs < m);
        }
      }
      if (wide) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const bool in = t + rl + i * step < rows;
          ldcg2_if(x[i][0], x[i][1], p, in && c < end);
          ldcg2_if(x[i][2], x[i][3], p + 2, in && c + 2 < end);
          p += (size_t)step * ldm;
        }
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const bool in = t + rl + i * step < rows;
#pragma unroll
          for (int e = 0; e < 4; ++e) x[i][e] = ldcg_if(p + e * cs, in && c + e * cs < end);
          p += (size_t)step * ldm;
        }
      }
      if (first && inplace && once) __syncthreads();  // every thread has its part of S
      first = false;
      const int k = c - (r0 + t + rl);
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int i = 0; i < 8; ++i) {  // what lies outside the triangle, or the matrix, is not used
          const double y = fma(x[i][e], s[e], v[i]);
          v[i] = (tri == 2 || (tri == 0 ? k + e * cs <= i * step : k + e * cs >= i * step)) ? y : v[i];
        }
    }
#pragma unroll
    for (int h = 4; h > 0; h >>= 1) {  // halves exchanged with the lane 4 / h away
      if (h > 1 || lg > 2) {
        const bool up = cl & (4 / h);
#pragma unroll
        for (int i = 0; i < h; ++i) {
          const double other = __shfl_xor_sync(0xffffffffu, up ? v[i] : v[i + h], 4 / h);
          v[i] = (up ? v[i + h] : v[i]) + other;
        }
      }
    }
    if (lg > 3) v[0] += __shfl_xor_sync(0xffffffffu, v[0], 8);
    if (lg > 4) v[0] += __shfl_xor_sync(0xffffffffu, v[0], 16);
    st_if(o, fma(alpha, v[0], old[0]), r < rows && cl < 8);
    st_if(o + (size_t)step * ldo, fma(alpha, v[1], old[1]), lg == 2 && r + step < rows);
  }
  __syncthreads();
}

// TRMV: the whole product in place (l == 0) or rows [o, o + l) of it out of place (l > 0)
__device__ __forceinline__ bool trmv_ok(const pp_task& T) {
  return T.m <= PP_VM_INV && T.n >= 1 && T.n <= 16 && (T.l <= 0 || (T.o >= 0 && T.o + T.l <= T.m && T.p[2]));
}

// ------------------------------------------------------------------------- composite instructions
// Instructions made of triangular solves on TL-blocks and of products: the VM has one copy of the
// product's code, so each of them is walked as a sequence of such steps.

// One product of the reference's association orders of GEMM3 / GEMM4 (kernel.cu:886-955): step 0,
// 1 (, 2) of the instruction, intermediates t1 (and t2) in task scratch.
struct Product {
  double* C;
  const double *A, *B;
  int ldc, lda, ldb, m, n, k;
  bool tA, tB;
  double alpha, beta;
};

__device__ __forceinline__ bool chain_step(const pp_task& T, int step, Product& P) {
  const int m = T.m, n = T.n, k = T.k, l = T.l, o = T.o;
  double *t1 = T.tmp, *t2 = T.tmp + T.aux;  // second intermediate (reference gemm_4x `offset`)
  auto operand = [&](int i, const double*& p, int& ld, bool& t) {
    p = T.p[i];
    ld = T.ld[i];
    t = (T.flags & PP_T(i)) != 0;
  };
  auto work = [&](const double* w, int wld, const double*& p, int& ld, bool& t) {
    p = w;
    ld = wld;
    t = false;
  };
  auto target = [&](double* c, int ldc, int mm, int nn, int kk, bool last) {
    P.C = c;
    P.ldc = ldc;
    P.m = mm;
    P.n = nn;
    P.k = kk;
    P.alpha = last ? T.alpha : 1.0;
    P.beta = last ? 1.0 : 0.0;
  };
  if (T.op == PP_OP_GEMM) {
    if (step > 0) return false;
    operand(1, P.A, P.lda, P.tA);
    operand(2, P.B, P.ldb, P.tB);
    target(T.p[0], T.ld[0], m, n, k, true);
    P.beta = T.beta;
    return true;
  }
  if (T.op == PP_OP_GEMM3) {
    if (step > 1) return false;
    if (T.ctrl) {  // (A B) C, t1: m x l
      if (step == 0) { operand(1, P.A, P.lda, P.tA); operand(2, P.B, P.ldb, P.tB); target(t1, l, m, l, k, false); }
      else { work(t1, l, P.A, P.lda, P.tA); operand(3, P.B, P.ldb, P.tB); target(T.p[0], T.ld[0], m, n, l, true); }
    } else {       // A (B C), t1: k x n
      if (step == 0) { operand(2, P.A, P.lda, P.tA); operand(3, P.B, P.ldb, P.tB); target(t1, n, k, n, l, false); }
      else { operand(1, P.A, P.lda, P.tA); work(t1, n, P.B, P.ldb, P.tB); target(T.p[0], T.ld[0], m, n, k, true); }
    }
    return true;
  }
  if (step > 2) return false;
  switch (T.ctrl) {
    case 0:  // ((A B) C) D; t1 m x l, t2 m x o
      if (step == 0) { operand(1, P.A, P.lda, P.tA); operand(2, P.B, P.ldb, P.tB); target(t1, l, m, l, k, false); }
      else if (step == 1) { work(t1, l, P.A, P.lda, P.tA); operand(3, P.B, P.ldb, P.tB); target(t2, o, m, o, l, false); }
      else { work(t2, o, P.A, P.lda, P.tA); operand(4, P.B, P.ldb, P.tB); target(T.p[0], T.ld[0], m, n, o, true); }
      break;
    case 1:  // (A (B C)) D; t1 k x o, t2 m x o
      if (step == 0) { operand(2, P.A, P.lda, P.tA); operand(3, P.B, P.ldb, P.tB); target(t1, o, k, o, l, false); }
      else if (step == 1) { operand(1, P.A, P.lda, P.tA); work(t1, o, P.B, P.ldb, P.tB); target(t2, o, m, o, k, false); }
      else { work(t2, o, P.A, P.lda, P.tA); operand(4, P.B, P.ldb, P.tB); target(T.p[0], T.ld[0], m, n, o, true); }
      break;
    case 2:  // A ((B C) D); t1 k x o, t2 k x n
      if (step == 0) { operand(2, P.A, P.lda, P.tA); operand(3, P.B, P.ldb, P.tB); target(t1, o, k, o, l, false); }
      else if (step == 1) { work(t1, o, P.A, P.lda, P.tA); operand(4, P.B, P.ldb, P.tB); target(t2, n, k, n, o, false); }
      else { operand(1, P.A, P.lda, P.tA); work(t2, n, P.B, P.ldb, P.tB); target(T.p[0], T.ld[0], m, n, k, true); }
      break;
    case 3:  // A (B (C D)); t1 l x n, t2 k x n
      if (step == 0) { operand(3, P.A, P.lda, P.tA); operand(4, P.B, P.ldb, P.tB); target(t1, n, l, n, o, false); }
      else if (step == 1) { operand(2, P.A, P.lda, P.tA); work(t1, n, P.B, P.ldb, P.tB); target(t2, n, k, n, l, false); }
      else { operand(1, P.A, P.lda, P.tA); work(t2, n, P.B, P.ldb, P.tB); target(T.p[0], T.ld[0], m, n, k, true); }
      break;
    default:  // 4: (A B) (C D); t1 m x l, t2 l x n
      if (step == 0) { operand(1, P.A, P.lda, P.tA); operand(2, P.B, P.ldb, P.tB); target(t1, l, m, l, k, false); }
      else if (step == 1) { operand(3, P.A, P.lda, P.tA); operand(4, P.B, P.ldb, P.tB); target(t2, n, l, n, o, false); }
      else { work(t1, l, P.A, P.lda, P.tA); work(t2, n, P.B, P.ldb, P.tB); target(T.p[0], T.ld[0], m, n, l, true); }
      break;
  }
  return true;
}

// One step of a triangular solve with a triangle of `size` rows, op one of the TRSM* kinds: even
// steps solve a diagonal TL-block (triangle *t at offset d in both), odd ones couple it to the rest.
// Every element gets the update sequence the tiled DAG would apply (i ascending), so results are
// identical.
__device__ __forceinline__ bool tri_step(int op, double* B, int ldb, const double* T, int ldt, int size, int lines,
                                         int step, int& d, int& len, Product& P) {
  const int nb = (size + TL - 1) / TL, at = step >> 1;
  if (at >= nb) return false;
  const int b = op == PP_OP_TRSMU ? nb - 1 - at : at;
  d = b * TL;
  len = min(TL, size - d);
  if (!(step & 1)) return true;
  const int e = d + len, rest = op == PP_OP_TRSMU ? d : size - e;
  if (rest <= 0) return false;
  P.alpha = -1.0;
  P.beta = 1.0;
  P.ldc = ldb;
  P.k = len;
  P.tA = P.tB = false;
  if (op == PP_OP_TRSMR) {  // B(:, right) -= B_d U(d, right)
    P.C = B + e;
    P.A = B + d;
    P.lda = ldb;
    P.B = T + (size_t)d * ldt + e;
    P.ldb = ldt;
    P.m = lines;
    P.n = rest;
    return true;
  }
  P.B = B + (size_t)d * ldb;
  P.ldb = ldb;
  P.lda = ldt;
  P.m = rest;
  P.n = lines;
  if (op == PP_OP_TRSML) {  // B_below -= L(below, d) B_d
    P.C = B + (size_t)e * ldb;
    P.A = T + (size_t)e * ldt + d;
  } else if (op == PP_OP_TRSMRT) {  // V_below -= U(d, below)^T V_d
    P.C = B + (size_t)e * ldb;
    P.A = T + (size_t)d * ldt + e;
    P.tA = true;
  } else {  // B_above -= U(above, d) B_d
    P.C = B;
    P.A = T + d;
  }
  return true;
}

// ------------------------------------------------------------------------- low-rank instructions
// ACCUM, ORTH and LRTRUNC, made of four pieces with one copy of code each (see dev_gemm for why):
//   tn    S = X^T [W1 W2], small outputs over many rows, on the FP64 tensor cores
//   rows  Y = A1 S1^T + alpha A2 S2^T row by row, on the FP64 tensor cores
//   chol  Cholesky G = C^T C of a Gram matrix: S1 = C^-T with Y C^-1 = Y S1^T
//   svd   pivoted factor C of a Gram matrix, one-sided Jacobi on C and the rank decision: the matrix S2 of
//         kept singular directions
// ACCUM: U1 V1^T := Q Q^T (U1 V1^T + alpha U2 V2^T), Q spanning (U1 V1^T + alpha U2 V2^T) R, the
// reference's randomized accumulation (kernel.cu:1255-1280) with Q from shifted CholeskyQR3 (three
// Gram passes) in place of the reference's Givens sweeps; m = ny, n = nx, k = k1 (target rank),
// l = k2; k1, k2 <= PP_VM_MAX_RANK:
//   [S1 S2] = R^T [V1 V2],  Y = U1 S1^T + alpha U2 S2^T            (the sketch, ny x k1)
//   3x: G = Y^T Y (+ shift), G = C^T C, Y := Y C^-1
//   [S1 S2] = Y^T [U1 U2],  V1 := V1 S1^T + alpha V2 S2^T,  U1 := Y
//   adaptive (PP_ADAPT_RANK): U1 V1^T = Y V1^T with Y orthonormal, so the singular values are those
//   of V1; both factors are turned into the eigenbasis of V1^T V1 and the directions whose singular
//   value exceeds beta times the largest are kept (zero columns beyond the new rank)
// ORTH: the three passes on Y = p[0] alone.  LRTRUNC: the adaptive part on U = p[0] (orthonormal
// columns) and V = p[1].  The sketch stays in shared memory when it fits, else in the task's scratch.
//
// Measured on a B200, hop included (before: reductions with one k step of loads in flight, a
// one-warp Cholesky, substitutions, a two-sided Jacobi on the Gram matrix):
//   ACCUM 128 x 128, k 32, adaptive   430 -> 134 us      ACCUM 94 x 94, k 16   54 -> 24 us
//   ORTH  512 x 32                    144 ->  78 us      LRTRUNC 512 x 512, k 32   420 -> 125 us
// 17 us of the first are products at the FP64 tensor rate, about 80 the chain of Jacobi steps.
template <int KB>
struct LrSmem {  // doubles; KB: largest rank, 16 or 32
  static constexpr int LD = KB + 4;                       // row stride: 4 mod 16, no bank conflicts
  static constexpr int S1 = 0, S2 = KB * LD, G = 2 * KB * LD, MISC = 3 * KB * LD, Y = MISC + 288;
  static constexpr int YCAP = VM_SMEM_BYTES / 8 - Y;
};

// whether ACCUM keeps its ny x k1 sketch in shared memory; otherwise it lives in the task's scratch
__host__ __device__ constexpr bool accum_y_on_chip(long long ny, int k1, int k2) {
  return ny * (k1 + 1) <= ((k1 <= 16 && k2 <= 16) ? LrSmem<16>::YCAP : LrSmem<32>::YCAP);
}

// a double anywhere (shared or global) under a predicate, else zero
__device__ __forceinline__ double ld_if(const double* p, bool in) {
  double v;
  asm volatile("{\n .reg .pred a;\n setp.ne.s32 a, %2, 0;\n mov.f64 %0, 0d0000000000000000;\n @a ld.f64 %0, [%1];\n}\n"
               : "=&d"(v)
               : "l"(p), "r"((int)in)
               : "memory");
  return v;
}

// a matrix of rows with strides (row, column); null: absent (zero)
struct LrMat {
  const double* p;
  int sr, sc, cols;
};

// NJ 8 x 8 tiles of X^T W over L rows: tile row mi of X's columns, tile columns j0 .. of W's
template <int NJ>
__device__ __forceinline__ void lr_tn_tiles(double (&acc)[4][2], const LrMat& X, const LrMat& W, int mi, int j0, int L,
                                            int fa, int fb) {
  constexpr int U = 4;  // k steps (of 4 rows) whose loads go out together
  const bool xin = 8 * mi + fa < X.cols;
  const double* xp = X.p + (size_t)fb * X.sr + (size_t)(8 * mi + fa) * X.sc;
  const double* wp = W.p + (size_t)fb * W.sr + (size_t)(8 * j0 + fa) * W.sc;
#pragma unroll 1
  for (int l = fb; l < L + fb; l += 4 * U) {
    double x[U], w[U][NJ];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool in = l + 4 * u < L;
      x[u] = ld_if(xp + (size_t)(4 * u) * X.sr, in && xin);
#pragma unroll
      for (int j = 0; j < NJ; ++j) w[u][j] = ld_if(wp + (size_t)(4 * u) * W.sr + (size_t)(8 * j) * W.sc, in && 8 * (j0 + j) + fa < W.cols);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int j = 0; j < NJ; ++j) dmma(acc[j][0], acc[j][1], x[u], w[u][j]);
    xp += (size_t)(4 * U) * X.sr;
    wp += (size_t)(4 * U) * W.sr;
  }
}

// out1 = X^T W1 and out2 = X^T W2 (when W2.p is set), zero-padded KB x KB blocks of stride KB + 4.
// Every warp owns output tiles and walks all rows: no partial sums to combine, ascending row order.
template <int KB>
__device__ __forceinline__ void lr_tn(const LrMat& X, const LrMat& W1, const LrMat& W2, int L, double* out1, double* out2) {
  constexpr int MT = KB / 8, LD = LrSmem<KB>::LD;
  const int tid = thread_index(), warp = tid >> 5, lane = tid & 31, fa = lane >> 2, fb = lane & 3;
  const int mi = warp % MT, part = warp / MT;  // 8 / MT warps share a tile row
  const bool both = W2.p != nullptr;
  double acc[4][2];
#pragma unroll
  for (int j = 0; j < 4; ++j) acc[j][0] = acc[j][1] = 0.0;
  int nj, j0;
  const bool second = both && part >= 4 / MT;
  if (KB == 32) {  // both: two warps of four tiles each; one: two of two
    nj = both ? 4 : 2;
    j0 = both ? 0 : 2 * part;
  } else {         // both: four warps of one tile each; one: the first two
    nj = both || part < 2 ? 1 : 0;
    j0 = part & 1;
  }
  const LrMat W = second ? W2 : W1;
  if (KB == 32 && both) lr_tn_tiles<4>(acc, X, W, mi, j0, L, fa, fb);
  else if (KB == 32) lr_tn_tiles<2>(acc, X, W, mi, j0, L, fa, fb);
  else if (nj) lr_tn_tiles<1>(acc, X, W, mi, j0, L, fa, fb);
  __syncthreads();  // the operands may lie where the results go
  double* o = (second ? out2 : out1) + (8 * mi + fa) * LD + 8 * j0 + 2 * fb;
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (j < nj) {
      o[8 * j] = acc[j][0];
      o[8 * j + 1] = acc[j][1];
    }
  __syncthreads();
}

// Y[l][0 .. k) = A1[l] S1^T + alpha A2[l] S2^T (A2 absent when null) for every row l, S1 and S2
// zero-padded KB x KB blocks of stride KB + 4.  A warp takes 16 rows and reads them before it
// writes, so Y may be A1.
template <int KB>
__device__ __forceinline__ void lr_rows(double* Y, int ly, const LrMat& A1, const LrMat& A2, double alpha,
                                        const double* S1, const double* S2, int k, int L) {
  constexpr int LD = LrSmem<KB>::LD, NJ = KB / 8, KS = KB / 4;
  const int tid = thread_index(), warp = tid >> 5, lane = tid & 31, fa = lane >> 2, fb = lane & 3;
#pragma unroll 1
  for (int r0 = 16 * warp; r0 < L; r0 += 128) {
    double acc[2][NJ][2];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int j = 0; j < NJ; ++j) acc[h][j][0] = acc[h][j][1] = 0.0;
#pragma unroll 1
    for (int o = 0; o < 2; ++o) {
      const LrMat A = o ? A2 : A1;
      if (!A.p) continue;
      const double* S = (o ? S2 : S1) + fa * LD + fb;
      const double f = o ? alpha : 1.0;
      const double* ap = A.p + (size_t)(r0 + fa) * A.sr + (size_t)fb * A.sc;
      double a[2][KS];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int t = 0; t < KS; ++t)
          a[h][t] = ld_if(ap + (size_t)(8 * h) * A.sr + (size_t)(4 * t) * A.sc, r0 + 8 * h + fa < L && 4 * t + fb < A.cols);
      if (f != 1.0) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int t = 0; t < KS; ++t) a[h][t] *= f;
      }
#pragma unroll
      for (int t = 0; t < KS; ++t)
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          const double b = S[8 * j * LD + 4 * t];
          dmma(acc[0][j][0], acc[0][j][1], a[0][t], b);
          dmma(acc[1][j][0], acc[1][j][1], a[1][t], b);
        }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      double* y = Y + (size_t)(r0 + 8 * h + fa) * ly + 2 * fb;
      const bool in = r0 + 8 * h + fa < L;
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        if (in && 8 * j + 2 * fb < k) y[8 * j] = acc[h][j][0];
        if (in && 8 * j + 2 * fb + 1 < k) y[8 * j + 1] = acc[h][j][1];
      }
    }
  }
  __syncthreads();
}

// The power of two, 2^-half, that brings a Gram matrix's trace near 1 (a subnormal one to 2^-52 at
// least) when it is applied twice: every live pivot is then within the range of `reciprocal`, whose
// estimate takes no subnormal number.  `mine`: the lane's diagonal entry; tr: the trace.
__device__ __forceinline__ double lr_scale(double mine, double& tr) {
  tr = mine;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) tr += __shfl_xor_sync(0xffffffffu, tr, o);
  const int ex = (__double2hiint(tr) >> 20) & 0x7FF;
  const int half = ex < 0x7FF ? (max(ex, 1) - 1023) >> 1 : 0;
  return __hiloint2double((1023 - half) << 20, 0);
}

// Cholesky of a Gram matrix G = Y^T Y (k x k, zero-padded) of a Y of m rows, G (+ shift) = C^T C:
// S1 := C^-T, so that Y C^-1 = Y S1^T (one Cholesky-QR pass); G is overwritten.  Elimination of
// [G | I] without pivoting, eight rows at a time: one warp eliminates them against each other (a
// column of G and one of the right half per lane, the eight rows in registers, multipliers by
// shuffles), then all warps update the rows below on the FP64 tensor cores.  A non-positive pivot
// marks a rank-deficient column, which becomes zero.  The chain of one pivot's reciprocal after the
// other bounds it (a form with every thread on its own entries and a barrier per row took three times
// as long).
template <int KB>
__device__ __forceinline__ void lr_chol(double* G, double* S1, int k, int m, bool shifted) {
  constexpr int LD = LrSmem<KB>::LD;
  const int tid = thread_index(), warp = tid >> 5, lane = tid & 31, fa = lane >> 2, fb = lane & 3, col = lane & (KB - 1);
  double tr;
  const double down = lr_scale(lane < k ? G[lane * LD + lane] : 0.0, tr), down2 = down * down;
  // shift of shifted CholeskyQR3: 11 (m k + k (k + 1)) u ||Y||_F^2, u = 2^-53
  const double sh = shifted ? 11.0 * ((double)m * k + (double)k * (k + 1)) * 1.1102230246251565e-16 * (tr * down2) : 0.0;
  const double tiny = 1e-28 * (tr * down2);
  __syncthreads();
  for (int e = tid; e < KB * LD; e += NT) {
    const int r = e / LD, c = e % LD;
    G[e] = fma(G[e], down2, (r == c && r < k) ? sh : 0.0);
    S1[e] = r == c ? 1.0 : 0.0;
  }
  __syncthreads();
  const int nb = (k + 7) >> 3;
#pragma unroll 1
  for (int J = 0; J < nb; ++J) {
    if (warp == 0) {
      double *g = G + 8 * J * LD + col, *s = S1 + 8 * J * LD + col;
      double x[8], z[8], d[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        x[i] = g[i * LD];
        z[i] = s[i * LD];
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        d[i] = __shfl_sync(0xffffffffu, x[i], 8 * J + i);
        const double ri = d[i] > tiny ? reciprocal(d[i]) : 0.0;
#pragma unroll
        for (int a = i + 1; a < 8; ++a) {
          const double f = __shfl_sync(0xffffffffu, x[i], 8 * J + a) * ri;
          x[a] = fma(-f, x[i], x[a]);
          z[a] = fma(-f, z[i], z[a]);
        }
      }
      double mine = d[0];
#pragma unroll
      for (int i = 1; i < 8; ++i) mine = (lane & 7) == i ? d[i] : mine;
      const double rs = mine > tiny ? rsqrt(mine) : 0.0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const double f = __shfl_sync(0xffffffffu, rs, i);
        if (lane < KB) {
          g[i * LD] = x[i] * f;
          s[i * LD] = z[i] * f;
        }
      }
    }
    __syncthreads();
    // rows of block t below: tiles u >= t of G, tiles u <= J of the right half
    const int items = (nb - 1 - J) * nb;
#pragma unroll 1
    for (int it = warp; it < items; it += NT / 32) {
      const int t = J + 1 + it / nb, u = it % nb;
      if (u > J && u < t) continue;
      double* M = u <= J ? S1 : G;
      const double *a = G + (8 * J + fb) * LD + 8 * t + fa, *b = M + (8 * J + fb) * LD + 8 * u + fa;
      double* c = M + (8 * t + fa) * LD + 8 * u + 2 * fb;
      double y0 = c[0], y1 = c[1];
      dmma(y0, y1, -a[0], b[0]);
      dmma(y0, y1, -a[4 * LD], b[4 * LD]);
      c[0] = y0;
      c[1] = y1;
    }
    __syncthreads();
  }
  for (int e = tid; e < KB * LD; e += NT) S1[e] *= down;
  __syncthreads();
}

// C^T C = G P times a power of two for the Gram matrix G of a factor to be truncated: rows of C, k of them
// at most (zero beyond; k x k, zero-padded), by elimination with the largest remaining diagonal entry as the
// pivot.  A column whose remaining entry is at most k u of what it was is noise and gets no row: dividing by
// its root would spread that noise over the others (an exactly rank-deficient G without pivoting: errors
// up to 2e-5 of G, and a rank beyond its own at tolerances of 1e-7 in a third of the cases), while all that
// is left then errs by k u sqrt(g_ii g_jj), as G's own rounding does.  The norms of the rows come out
// decreasing by and large, which also saves the Jacobi below one sweep or two.
// One warp, a column per lane: row s is pivot p's row of G minus the rows before it, times their
// entries in p; pivots by their upper 27 bits and lane in one integer reduction.  The chain of pivots
// bounds it: reduction, reciprocal root, update of the diagonal.
template <int KB>
__device__ __forceinline__ void lr_factor(const double* G, double* C, int k) {
  constexpr int LD = LrSmem<KB>::LD;
  const int tid = thread_index(), lane = tid & 31, col = lane & (KB - 1);
  for (int e = tid; e < KB * LD; e += NT) C[e] = 0.0;
  __syncthreads();
  if (tid < 32) {
    const double mine = lane < k ? G[lane * LD + lane] : 0.0;
    double tr;
    const double down = lr_scale(mine, tr), down2 = down * down;
    double left = mine * down2;  // of the lane's diagonal entry; 0 once it has been the pivot
    const double noise = (double)k * 1.1102230246251565e-16 * left;
    bool done = false;
#pragma unroll 1
    for (int s = 0; s < k; ++s) {
      const unsigned key = left > noise ? ((unsigned)__double2hiint(left) & ~31u) | (31u - lane) : 0u;
      const unsigned best = __reduce_max_sync(0xffffffffu, key);
      if (best < 32u) break;
      const int p = 31 - (int)(best & 31u);
      const double d = __shfl_sync(0xffffffffu, left, p), r = rsqrt(d);
      double x = G[p * LD + col] * down2, y = 0.0;
      const double *cp = C + p, *cc = C + col;
#pragma unroll 1
      for (int t = 0; t < s; t += 4) {  // rows past s are zero
#pragma unroll
        for (int u = 0; u < 4; u += 2) {
          x = fma(-cp[(t + u) * LD], cc[(t + u) * LD], x);
          y = fma(-cp[(t + u + 1) * LD], cc[(t + u + 1) * LD], y);
        }
      }
      const double c = done ? 0.0 : lane == p ? d * r : (x + y) * r;
      done |= lane == p;
      left = done ? 0.0 : fma(-c, c, left);
      if (lane < KB) C[s * LD + lane] = c;
      __syncwarp();
    }
  }
  __syncthreads();
}

// Singular directions of a matrix V from a factor C (k x k, k rows of B, stride LD, zero-padded) of its
// Gram matrix, V^T V ~ C^T C scaled to a trace near 1 (lr_factor): one-sided Jacobi makes the rows
// of C orthogonal, their norms are then V's singular values, scaled, and the rows themselves, normalized, its right singular
// vectors.  Then the rank decision: rows in decreasing order of norm, r = #{ norm_i > tol norm_0 }, at
// most rmax, and S[i] = the i-th direction for i < r (zero rows beyond), so that a row of V times S^T
// is its coordinates in the kept directions.  Returns r.
//
// The pivoted factor of a graded Gram matrix is close to row-orthogonal already: 5 or 6 sweeps where the
// two-sided Jacobi on the Gram matrix took 12 (its limit), a third of the shared-memory traffic, and
// the directions are orthogonal to rounding however small their singular value.  Round-robin order,
// k/2 disjoint pairs at once, eight lanes of the first four warps per pair, which all compute its
// rotation; one barrier of those warps per step.  A pair is rotated while |b_p . b_q| > 1e-15 |b_p| |b_q|
// (a few u: what is left bounds the directions' products) and the smaller norm counts for the rank
// (> 1e-2 tol of the largest); a sweep whose rotations were all below 1e-8 is the last (the next
// would find products of such angles), and at most 14 are made.  The rotation is the symmetric
// Schur decomposition of the pair's 2 x 2 Gram matrix (Golub & Van Loan, sym.schur2), t = tan(theta)
// written as 2 a sgn(d) / (|d| + h), d = |b_q|^2 - |b_p|^2, h = sqrt(d^2 + 4 a^2): cos = r / s,
// sin = 2 a sgn(d) / s with r = |d| + h, s = sqrt(r^2 + 4 a^2).  h only steers the angle and comes
// from an estimate of the reciprocal root; 1 / s, which makes the rotation orthogonal, is corrected
// to full precision (y (1 + e/2 + 3 e^2/8), e = 1 - s^2 y^2, binomial series).
__device__ __forceinline__ void round_robin(int kk, int r, int jp, int& p, int& q) {
  // positions of pair jp in step r: 1 + (pos - 1 + r) mod (kk - 1); position 0 stays
  int ua = jp - 1 + r, ub = kk - 2 - jp + r;
  ua -= ua >= kk - 1 ? kk - 1 : 0;
  ub -= ub >= kk - 1 ? kk - 1 : 0;
  const int a = jp == 0 ? 0 : 1 + ua, b = kk - 1 - jp == 0 ? 0 : 1 + ub;
  p = min(a, b);
  q = max(a, b);
}
__device__ __forceinline__ double sum8(double v) {
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// barrier of the CTA's first 128 threads; whether any of them has `flag` set
__device__ __forceinline__ int bar128_or(int flag) {
  int r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.s32 q, %1, 0;\n barrier.cta.red.or.pred p, 1, 128, q;\n selp.b32 %0, 1, 0, p;\n}\n"
      : "=r"(r)
      : "r"(flag)
      : "memory");
  return r;
}
template <int KB>
__device__ __forceinline__ void lr_norms(const double* B, double* n2, int tid) {
  constexpr int LD = LrSmem<KB>::LD;
#pragma unroll
  for (int h = 0; h < KB; h += 16) {
    const double* b = B + ((tid >> 3) + h) * LD + (tid & 7);
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < KB; i += 8) s = fma(b[i], b[i], s);
    s = sum8(s);
    if ((tid & 7) == 0) n2[(tid >> 3) + h] = s;
  }
}
template <int KB>
__device__ __forceinline__ int lr_svd(double* B, double* S, double* misc, int k, double tol, int rmax) {
  constexpr int LD = LrSmem<KB>::LD, NE = KB / 8;
  // an odd k gets a row k of zeros (B is zero-padded), which never rotates
  const int tid = thread_index(), lane = tid & 31, kk = (k + 1) & ~1, np = kk / 2, pair = tid >> 3, l = tid & 7;
  double* n2 = misc;  // squared norms
  int* perm = reinterpret_cast<int*>(misc + 32);
  if (tid < 128) {
#pragma unroll 1
    for (int sweep = 0; sweep < 14; ++sweep) {
      lr_norms<KB>(B, n2, tid);
      bar128_or(0);
      double top = n2[lane & (KB - 1)];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
      const double floor2 = 1e-4 * tol * tol * top;
      int seen = 0;
#pragma unroll 1
      for (int r = 0; r < kk - 1; ++r) {
        int p, q;
        round_robin(kk, r, min(pair, np - 1), p, q);
        double *bp = B + p * LD + l, *bq = B + q * LD + l;
        double x[NE], y[NE], dot = 0.0;
#pragma unroll
        for (int i = 0; i < NE; ++i) {
          x[i] = bp[8 * i];
          y[i] = bq[8 * i];
        }
#pragma unroll
        for (int i = 0; i < NE; ++i) dot = fma(x[i], y[i], dot);
        const double app = n2[p], aqq = n2[q], a = sum8(dot);
        const double d = aqq - app, g2 = d >= 0.0 ? 2.0 * a : -2.0 * a, gg = g2 * g2, v = fma(d, d, gg);
        const double rr = fma(v, rsqrt_est(v), fabs(d)), s2 = fma(rr, rr, gg), y0 = rsqrt_est(s2);
        const double e = fma(-s2 * y0, y0, 1.0), w = fma(y0 * e, fma(0.375, e, 0.5), y0);
        const double a2 = a * a, both = app * aqq;
        const int rot = (int)(a2 > 1e-30 * both) & (int)(fmin(app, aqq) > floor2) & (int)(v > 1e-280) &
                        (int)(s2 < 1e280) & (int)(pair < np);
        if (rot) {
          const double c = rr * w, sn = g2 * w;
#pragma unroll
          for (int i = 0; i < NE; ++i) {
            bp[8 * i] = fma(c, x[i], -sn * y[i]);
            bq[8 * i] = fma(sn, x[i], c * y[i]);
          }
          if (l == 0) {
            n2[p] = fma(c * c, app, fma(sn * sn, aqq, -2.0 * c * sn * a));
            n2[q] = fma(sn * sn, app, fma(c * c, aqq, 2.0 * c * sn * a));
          }
        }
        seen |= rot & (int)(a2 > 1e-16 * both);
        asm volatile("barrier.cta.sync 1, 128;" ::: "memory");
      }
      if (!bar128_or(seen)) break;
    }
    lr_norms<KB>(B, n2, tid);
  }
  __syncthreads();
  // the place of norm_i among the others (equal ones in index order)
  const double mine = lane < k ? n2[lane & (KB - 1)] : -1.0;
  double top = mine;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
  int place = 0;
  for (int j = 0; j < k; ++j) {
    const double v = n2[j];
    place += (v > mine || (v == mine && j < lane)) ? 1 : 0;
  }
  const unsigned kept = __ballot_sync(0xffffffffu, lane < k && top > 0.0 && mine > tol * tol * top);
  if (tid < k) {
    perm[place] = tid;
    misc[64 + place] = mine > 0.0 ? rsqrt(mine) : 0.0;
  }
  __syncthreads();
  const int rank = min(__popc(kept), rmax);
  for (int e = tid; e < KB * KB; e += NT) {
    const int i = e / KB, j = e % KB;
    S[i * LD + j] = (i < rank && j < k) ? B[perm[i] * LD + j] * misc[64 + i] : 0.0;
  }
  __syncthreads();
  return rank;
}

template <int KB>
__device__ __forceinline__ void lowrank_impl(const pp_task& T) {
  extern __shared__ __align__(16) double vm_smem[];
  using SM = LrSmem<KB>;
  double *S1 = vm_smem + SM::S1, *S2 = vm_smem + SM::S2, *G = vm_smem + SM::G, *misc = vm_smem + SM::MISC;
  const bool accum = T.op == PP_OP_ACCUM, orth = T.op == PP_OP_ORTH;
  const int m = T.m, n = T.n, k = orth ? T.n : T.k, k2 = accum ? T.l : 0;
  const bool on_chip = (accum || orth) && accum_y_on_chip(m, k, k2);
  const int pad = (long long)m * (k + 4) <= SM::YCAP ? 4 : (long long)m * (k + 2) <= SM::YCAP ? 2 : 1;
  double* U = T.p[0];
  double* Y = on_chip ? vm_smem + SM::Y : accum ? T.tmp : U;
  const int ly = on_chip ? k + pad : accum ? k : T.ld[0];
  const bool adapt = !orth && (!accum || ((T.flags & PP_ADAPT_RANK) && T.beta > 0.0));
  const LrMat none{nullptr, 0, 0, 0};
  const LrMat My{Y, ly, 1, k}, Mu{U, T.ld[0], 1, k}, Mv{T.p[1], T.ld[1], 1, k};
  LrMat Mu2 = none, Mv2 = none;
  if (accum && k2 > 0) {
    Mu2 = (T.flags & PP_T(2)) ? LrMat{T.p[2], 1, T.ld[2], k2} : LrMat{T.p[2], T.ld[2], 1, k2};
    Mv2 = (T.flags & PP_T(3)) ? LrMat{T.p[3], 1, T.ld[3], k2} : LrMat{T.p[3], T.ld[3], 1, k2};
  }
  if (orth && on_chip) {
    for (int e = threadIdx.x; e < m * k; e += NT) Y[(e / k) * ly + e % k] = ldcg(&U[e]);
    __syncthreads();
  }
  const int rmax = (!accum && T.o > 0) ? min(T.o, k) : k;
  int rank = k;
  // phases: 0 the sketch, 1-3 the Cholesky-QR passes, 4 the projection, 5 the truncation of V and
  // 6 of the orthonormal factor
#pragma unroll 1
  for (int ph = accum ? 0 : orth ? 1 : 5; ph <= (orth ? 3 : adapt ? 6 : 4); ++ph) {
    if (ph < 6) {
      const LrMat X = ph == 0 ? LrMat{T.p[4], T.ld[4], 1, k} : ph == 5 ? Mv : My;
      const LrMat W1 = ph == 0 || ph == 5 ? Mv : ph == 4 ? Mu : My;
      const LrMat W2 = ph == 0 ? Mv2 : ph == 4 ? Mu2 : none;
      const bool gram = ph != 0 && ph != 4;
      lr_tn<KB>(X, W1, W2, ph == 0 || ph == 5 ? n : m, gram ? G : S1, S2);
      if (ph >= 1 && ph <= 3) lr_chol<KB>(G, S1, k, m, ph == 1);
      if (ph == 5) lr_factor<KB>(G, S1, k);
      if (ph == 5) rank = lr_svd<KB>(S1, S2, misc, k, T.beta, rmax);
    }
    const bool first = ph == 0 || ph == 4;
    // the factor's last product writes it where it belongs
    double* out = ph == 4 || ph == 5 ? T.p[1] : ph == 6 || (orth && ph == 3) ? U : Y;
    const int lo = ph == 4 || ph == 5 ? T.ld[1] : ph == 6 || (orth && ph == 3) ? T.ld[0] : ly;
    const LrMat A1 = ph == 0 ? Mu : ph == 4 || ph == 5 ? Mv : (ph == 6 && !accum) ? Mu : My;
    lr_rows<KB>(out, lo, A1, first ? (ph == 0 ? Mu2 : Mv2) : none, T.alpha, ph >= 5 ? S2 : S1, S2, k,
                ph == 4 || ph == 5 ? n : m);
  }
  if (accum && !adapt) {  // U1 := Y
    for (int e = threadIdx.x; e < m * k; e += NT) U[(size_t)(e / k) * T.ld[0] + e % k] = Y[(size_t)(e / k) * ly + e % k];
  }
  if (adapt && threadIdx.x == 0 && T.p[5]) T.p[5][0] = (double)rank;
  __syncthreads();
}

__device__ __forceinline__ void dev_lowrank(const pp_task& T) {
  const int k = T.op == PP_OP_ORTH ? T.n : T.k;
  if (k <= 16 && (T.op != PP_OP_ACCUM || T.l <= 16)) lowrank_impl<16>(T);
  else lowrank_impl<32>(T);
}

__device__ __noinline__ void dev_kmul(const pp_task& T, double* smem);

// C[m x n] (m <= 16, n <= 32) = beta C + alpha A^T B in free order, A: k x m, B: k x n as stored (the
// solves' x^T V): every warp sums a slice of the rows, read straight into tensor-core fragments, and
// the slices are added in order.
__device__ __forceinline__ void dev_tn(double* C, int ldc, const double* A, int lda, const double* B, int ldb, int m, int n,
                                       int k, double alpha, double beta) {
  extern __shared__ __align__(16) double vm_smem[];
  const int tid = thread_index(), warp = tid >> 5, lane = tid & 31, fa = lane >> 2, fb = lane & 3;
  const int per = (((k + 7) >> 3) + 3) & ~3, l0 = min(k, warp * per), len = min(per, k - l0);
#pragma unroll 1
  for (int mi = 0; 8 * mi < m; ++mi) {
    double acc[4][2];
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[j][0] = acc[j][1] = 0.0;
    const LrMat X{A + (size_t)l0 * lda, lda, 1, m}, W{B + (size_t)l0 * ldb, ldb, 1, n};
    if (n > 16) lr_tn_tiles<4>(acc, X, W, mi, 0, len, fa, fb);
    else lr_tn_tiles<2>(acc, X, W, mi, 0, len, fa, fb);
    double* red = vm_smem + (mi * 8 + warp) * 256 + fa * 32 + 2 * fb;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      red[8 * j] = acc[j][0];
      red[8 * j + 1] = acc[j][1];
    }
  }
  __syncthreads();
  for (int e = tid; e < m * n; e += NT) {
    const int r = e / n, c = e - r * n;
    const double* red = vm_smem + (r >> 3) * 2048 + (r & 7) * 32 + c;
    double v = red[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) v += red[w * 256];
    double* p = C + (size_t)r * ldc + c;
    *p = beta != 0.0 ? fma(alpha, v, ldcg(p)) : alpha * v;
  }
  __syncthreads();
}

__device__ __forceinline__ void run_composite(const pp_task& T) {
  const bool product = T.op == PP_OP_GEMM || T.op == PP_OP_GEMM3 || T.op == PP_OP_GEMM4;
  const bool free_order = T.op == PP_OP_GEMM && (T.flags & PP_FREE_ORDER), tA = T.flags & PP_T(1), tB = T.flags & PP_T(2);
  // products of the solves, in free order: a leaf, its inverse or a low-rank factor times a few
  // right-hand sides (columns that stage in shared memory), and a few right-hand sides' transposes
  // times a low-rank factor (short k stays with the general product: 8 warps of 8 rows are not fewer
  // steps than its one chunk; so do several transposed columns: 94 x 16 x 16 took 3.05 us instead of 2.8)
  if (T.op == PP_OP_TRMV || (free_order && !tA && T.n <= (tB ? 1 : 16) && T.k <= 1024)) {
    const bool trmv = T.op == PP_OP_TRMV, part = trmv && T.l > 0;
    const int r0 = part ? T.o : 0;
    const double* S = trmv ? (part ? T.p[2] : T.p[0]) : T.p[2];
    const int lds = trmv ? (part ? T.ld[2] : T.ld[0]) : T.ld[2];
    const int m = trmv ? T.m : T.k, rows = part ? T.l : T.m, tri = !trmv ? 2 : T.ctrl == 1 ? 1 : T.ctrl == 0 ? 0 : 2;
    const double* M = T.p[1] + (size_t)r0 * T.ld[1];
    const double alpha = trmv ? 1.0 : T.alpha, beta = trmv ? 0.0 : T.beta;
    // one column: with FMAs; more of them: on the tensor cores
    if (T.n == 1 && m > 0)
      dev_column(T.p[0], T.ld[0], M, T.ld[1], S, !trmv && tB ? 1 : lds, m, rows, tri, r0, alpha, beta);
    else
      dev_rows(T.p[0], T.ld[0], M, T.ld[1], S, lds, m, T.n, rows, tri, r0, alpha, beta);
    return;
  }
  if (free_order && tA && !tB && T.m <= 16 && T.n <= 32 && T.k >= 64) {
    dev_tn(T.p[0], T.ld[0], T.p[1], T.ld[1], T.p[2], T.ld[2], T.m, T.n, T.k, T.alpha, T.beta);
    return;
  }
  int op = T.op, size = T.op == PP_OP_TRSMR ? T.n : T.m, lines = T.op == PP_OP_TRSMR ? T.m : T.n;
  double* B = T.p[0];
  const double* A = T.p[1];
  const int ldb = T.ld[0], lda = T.ld[1];
  if (T.op == PP_OP_TRINV) {
    // columns [o, o + n) of L^-1 (ctrl 0) or U^-1 (1): identity columns, then the solve on the
    // sub-triangle they need (rows o.. of L^-1 are the only nonzeros; rows ..o + n of U^-1)
    const int w = T.n, c0 = T.o;
    for (int e = threadIdx.x; e < T.m * w; e += NT) {
      const int r = e / w, j = e % w;
      B[(size_t)r * ldb + j] = r == c0 + j ? 1.0 : 0.0;
    }
    __syncthreads();
    op = T.ctrl ? PP_OP_TRSMU : PP_OP_TRSML;
    size = T.ctrl ? c0 + w : T.m - c0;
    lines = w;
    if (!T.ctrl) {
      B += (size_t)c0 * ldb;
      A += (size_t)c0 * lda + c0;
    }
  }
#pragma unroll 1
  for (int step = 0;; ++step) {
    Product P;
    if (product) {
      if (!chain_step(T, step, P)) break;
    } else {
      int d = 0, len = 0;
      if (!tri_step(op, B, ldb, A, lda, size, lines, step, d, len, P)) break;
      if (!(step & 1)) {
        double* Bd = B + (op == PP_OP_TRSMR ? (size_t)d : (size_t)d * ldb);
        dev_tri(op, Bd, ldb, A + (size_t)d * lda + d, lda, len, lines, (T.flags & PP_PIVOT) ? T.p[2] : nullptr);
        continue;
      }
    }
    dev_gemm(P.C, P.ldc, P.A, P.lda, P.tA, P.B, P.ldb, P.tB, P.m, P.n, P.k, P.alpha, P.beta, free_order);
  }
}

// C[m x n] := A[m x n], eight loads in flight per thread
__device__ __forceinline__ void dev_copy(double* C, int ldc, const double* A, int lda, int m, int n) {
  const int tid = thread_index();
#pragma unroll 1
  for (int e0 = tid; e0 < m * n; e0 += 8 * NT) {
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int e = e0 + u * NT, r = e / n;
      v[u] = ldcg_if(A + (size_t)r * lda + (e - r * n), e < m * n);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int e = e0 + u * NT, r = e / n;
      st_if(C + (size_t)r * ldc + (e - r * n), v[u], e < m * n);
    }
  }
  __syncthreads();
}

// C[m x n] := beta C + sum_p T_p (p ascending), T_p the p-th m x n block of T
__device__ __noinline__ void dev_sum(double* C, int ldc, const double* T, int ldt, int m, int n, int parts,
                                     double beta) {
  for (int e = threadIdx.x; e < m * n; e += NT) {
    const int r = e / n, c = e % n;
    double s = 0.0;
    for (int p = 0; p < parts; ++p) s += ldcg(&T[(size_t)(p * m + r) * ldt + c]);
    double* q = &C[(size_t)r * ldc + c];
    *q = beta != 0.0 ? ldcg(q) + s : s;
  }
  __syncthreads();
}

__device__ bool run_task(const pp_task& T, double* smem, TcCtx& tc, int& err) {
  switch (T.op) {
    case PP_OP_NOP: return true;
    case PP_OP_GETRF:
      if (T.m > TL || T.n > TL) return false;
      if (T.flags & PP_PIVOT) {
        if (!T.p[1]) return false;
        dev_getrf_piv(T.p[0], T.ld[0], T.m, T.n, T.p[1]);
      } else {
        dev_getrf(T.p[0], T.ld[0], T.m, T.n);
      }
      return true;
    case PP_OP_TRSML:
      if (T.flags & PP_PIVOT) {  // one pivoted block per instruction
        if (T.m > TL || !T.p[2]) return false;
        break;
      }
      if (T.m > PP_VM_TRI) return false;
      break;
    case PP_OP_TRSMR:
      if (T.n > PP_VM_TRI) return false;
      break;
    case PP_OP_TRSMRT:
    case PP_OP_TRSMU:
      if (T.m > PP_VM_TRI) return false;
      break;
    case PP_OP_GEMM:
      if (T.prec == PP_PREC_BF16) {
        if (!tc.active || T.m < 128 || T.m % 128 || T.k < 64 || T.k % 64 || T.l < 0 || T.l % 64 ||
            (T.l > 0 && (!T.p[3] || !T.p[4])) ||
            !(T.n == 32 || T.n == 64 || T.n == 128 || (T.n >= BG_TILE_N && T.n % BG_TILE_N == 0)))
          return false;
        if (!dev_gemm_bf16(T.p[0], T.ld[0], reinterpret_cast<const uint8_t*>(T.p[1]),
                           reinterpret_cast<const uint8_t*>(T.p[2]), T.m, T.n, T.k, T.alpha, T.beta, smem, tc,
                           reinterpret_cast<const uint8_t*>(T.p[3]), reinterpret_cast<const uint8_t*>(T.p[4]), T.l))
          err = PP_VM_MMA_TIMEOUT;
        return true;
      }
      if (T.prec == PP_PREC_TF32) {
        if (!tc.active) return false;  // launched without tensor memory
        if (!dev_gemm_tc(T.p[0], T.ld[0], T.p[1], T.ld[1], T.flags & PP_T(1), T.p[2], T.ld[2], T.flags & PP_T(2),
                         T.m, T.n, T.k, T.alpha, T.beta, smem, tc))
          err = PP_VM_MMA_TIMEOUT;
        return true;
      }
      break;
    case PP_OP_GEMM3:
    case PP_OP_GEMM4: break;
    case PP_OP_ACCUM:
      if (T.k > PP_VM_MAX_RANK || T.k < 1 || T.l > PP_VM_MAX_RANK || T.l < 0) return false;
      break;
    case PP_OP_SUM:
      dev_sum(T.p[0], T.ld[0], T.p[1], T.ld[1], T.m, T.n, T.k, T.beta);
      return true;
    case PP_OP_TRINV:
      if (T.m > PP_VM_INV || T.n < 1 || T.o < 0 || T.o + T.n > T.m) return false;
      break;
    case PP_OP_TRMV:
      if (!trmv_ok(T)) return false;
      break;
    case PP_OP_ORTH:
      if (T.n < 1 || T.n > PP_VM_MAX_RANK || T.ld[0] != T.n) return false;
      break;
    case PP_OP_COPY:
      dev_copy(T.p[0], T.ld[0], T.p[1], T.ld[1], T.m, T.n);
      return true;
    case PP_OP_KMUL:
      if (T.k < 1 || T.k > PP_VM_MAX_RANK || T.l < 1 || T.l > 3 || T.ctrl < 0 || T.ctrl > 3 || T.m < 0 || T.n < 0)
        return false;
      dev_kmul(T, smem);
      return true;
    case PP_OP_LRTRUNC:
      if (T.k < 1 || T.k > PP_VM_MAX_RANK || T.m < T.k || T.n < T.k) return false;
      break;
    case PP_OP_SHADOW:
      if (T.m < 32 || T.k < 64 || T.k % 64) return false;
      if (T.l < 0 || T.l > T.m || T.n < 0 || T.n > T.k) return false;
      if (!(T.ctrl == 0 || T.ctrl == 32 || T.ctrl == 64 || T.ctrl == 128) || T.m % (T.ctrl ? T.ctrl : 128)) return false;
      if (T.o != 0 && (T.o >> 8 != 3 || (T.o & ~0x7FF) || T.k % (64 * 3) || T.n > T.k / 3)) return false;
      dev_shadow(reinterpret_cast<uint8_t*>(T.p[0]), T.p[1], T.ld[1], T.flags & PP_T(1), T.m, T.k,
                 T.l > 0 ? T.l : T.m, T.n > 0 ? T.n : (T.o ? T.k / 3 : T.k), T.ctrl ? T.ctrl : 128, T.o);
      return true;
    default: return false;
  }
  if (T.op == PP_OP_ACCUM || T.op == PP_OP_ORTH || T.op == PP_OP_LRTRUNC) dev_lowrank(T);
  else run_composite(T);
  return true;
}

// Counters of the priority classes' queues, behind the slots: tasks available, taken and pushed
#define VM_AVAIL 0
#define VM_HEAD PP_VM_CLASSES
#define VM_TAIL (2 * PP_VM_CLASSES)

__global__ void vm_init(const int32_t* __restrict__ indeg, const int32_t* __restrict__ ready, int n_ready, int n,
                        int32_t* counters, int32_t* slots, pp_vm_state* st, int by_class,
                        const __grid_constant__ pp_vm_classes cls) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    counters[i] = indeg[i];
    int at = i, count = n_ready;
    if (by_class) {
      int q = 0;
      while (q < PP_VM_CLASSES - 1 && i >= cls.base[q + 1]) ++q;
      at = cls.first[q] + (i - cls.base[q]);
      count = cls.first[q + 1];
    }
    slots[i] = at < count ? ready[at] : -1;
  }
  if (by_class && i < PP_VM_CLASSES) {
    const int first = cls.first[i + 1] - cls.first[i];
    slots[n + VM_AVAIL + i] = first;
    slots[n + VM_HEAD + i] = 0;
    slots[n + VM_TAIL + i] = first;
  }
  if (i == 0) {
    st->head = 0;
    st->tail = n_ready;
    st->done = 0;
    st->error = 0;
    st->err_info = -1;
  }
}

__device__ __forceinline__ unsigned long long globaltimer_ns() { return gtimer_ns(); }
__device__ __forceinline__ unsigned smid() {
  unsigned s;
  asm volatile("mov.u32 %0, %%smid;" : "=r"(s));
  return s;
}

// Ready tasks by priority class (warp-wide).  A program with much work beside its critical path keeps
// many tasks ready, and in one queue a task of that path waits for all of them: 37 of the 116 ms of a
// mixed-precision factorization (N = 32768).  A push takes its slot with the class's tail, stores the
// task and then counts it as available; a take first secures one of the most urgent class that shows
// any (the count would go below zero otherwise: given back), then its slot.  A secured slot is filled,
// or about to be: its push holds an earlier count or a slot already taken.
__device__ __forceinline__ void push_by_class(int32_t* slots, int n, const pp_vm_classes& cls, int entry, int lane) {
  const int q = entry >= 0 ? entry >> PP_VM_ID_BITS : -1;
  const unsigned same = __match_any_sync(0xffffffffu, q);
  const int leader = __ffs((int)same) - 1, rank = __popc(same & ((1u << lane) - 1));
  int pos = 0;
  if (q >= 0 && lane == leader) pos = atom_add_relaxed(&slots[n + VM_TAIL + q], __popc(same));
  pos = __shfl_sync(0xffffffffu, pos, leader);
  if (q >= 0) st_release(&slots[cls.base[q] + pos + rank], entry & ((1 << PP_VM_ID_BITS) - 1));
  __syncwarp();
  if (q >= 0 && lane == leader)
    asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(&slots[n + VM_AVAIL + q]), "r"(__popc(same)) : "memory");
}
// -1: every task is done, or the run has failed
__device__ __forceinline__ int take_by_class(int32_t* slots, int n, const pp_vm_classes& cls, pp_vm_state* st,
                                             long long wait_ns, int lane) {
  const unsigned long long t0 = gtimer_ns();
  int slot = -1;  // of the secured task
  for (;;) {
    if (slot < 0) {
      const int avail = lane < PP_VM_CLASSES ? ld_relaxed(&slots[n + VM_AVAIL + lane]) : 0;
      const bool over = __any_sync(0xffffffffu, ld_relaxed(&st->error) != 0 || ld_relaxed(&st->done) >= n);
      const unsigned some = __ballot_sync(0xffffffffu, avail > 0);
      if (some) {
        const int q = __ffs((int)some) - 1;
        if (lane == 0) {
          if (atom_add_relaxed(&slots[n + VM_AVAIL + q], -1) > 0)
            slot = cls.base[q] + atom_add_relaxed(&slots[n + VM_HEAD + q], 1);
          else
            atom_add_relaxed(&slots[n + VM_AVAIL + q], 1);
        }
        slot = __shfl_sync(0xffffffffu, slot, 0);
      } else if (over) {
        return -1;
      } else {
        __nanosleep(32);
      }
    }
    if (slot >= 0) {
      const int id = __shfl_sync(0xffffffffu, ld_acquire(&slots[slot]), 0);
      if (id >= 0) return id;
    }
    // bounded in time, as a wait on the one queue is
    if (__any_sync(0xffffffffu, (long long)(gtimer_ns() - t0) > wait_ns)) {
      if (lane == 0 && atomicCAS(&st->error, 0, slot >= 0 ? PP_VM_TIMEOUT : PP_VM_IDLE) == 0)
        st->err_info = slot >= 0 ? slot : ld_relaxed(&st->done);
      return -1;
    }
  }
}

__global__ void __launch_bounds__(NT, 1)
    vm_kernel(const pp_task* __restrict__ tasks, int n_tasks, const int32_t* __restrict__ succ, int32_t* counters,
              int32_t* slots, pp_vm_state* st, long long wait_ns, unsigned long long* trace, int use_tc, int by_class,
              const __grid_constant__ pp_vm_classes cls) {
  extern __shared__ __align__(16) double smem[];
  __shared__ __align__(16) pp_task s_rec[2][4];  // this task's record, and those of its first successors
  __shared__ int s_succ[2][32];                  // its first successors, and the previous task's
  __shared__ int s_pub[32], s_npub;              // successors ready but not run here
  __shared__ int s_id;
  __shared__ int s_keep;  // position (in the successor list) of the successor run next, or -1
  __shared__ unsigned long long s_t0;
  __shared__ uint32_t s_tmem;
  __shared__ __align__(8) unsigned long long s_mbar;
  __shared__ __align__(8) unsigned long long s_bg[2 * BG_STAGES + 4];  // BF16 pipeline mbarriers
  __shared__ int s_abort;
  TcCtx tc{0u, 0u, 0u, wait_ns, 0, 0, 0u, 0u, 0u, &s_abort};
  if (use_tc) {
    // TF32 and BF16 tasks: all 512 TMEM columns (TF32 uses 64, BF16 two accumulators of 256) and mbarriers
    if ((threadIdx.x >> 5) == 0) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                   "r"(TC_TMEM_COLS)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x == 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&s_mbar)) : "memory");
      // BF16 pipeline: stage full / empty (one arrival each: the producer's expect_tx, the MMA
      // issuer's commit), accumulator full (a commit) / empty (one arrival per epilogue warp)
      for (int i = 0; i < 2 * BG_STAGES + 2; ++i) mbar_init(smem_u32(&s_bg[i]), 1);
      for (int i = 2 * BG_STAGES + 2; i < 2 * BG_STAGES + 4; ++i) mbar_init(smem_u32(&s_bg[i]), 4);
      s_abort = 0;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    tc.tmem = s_tmem;
    tc.mbar = smem_u32(&s_mbar);
    tc.bars = smem_u32(&s_bg[0]);
    tc.active = 1;
  }
  // Continuation: of the successors this CTA's task makes ready, the first in the
  // successor list (sorted by the host, longest remaining path first) is run next by the
  // same CTA without a round trip through the queue; the others are pushed.  Queue slots
  // therefore number fewer than tasks, so a CTA waiting on a slot also leaves once every
  // task is done.
  //
  // What a hop from a task to its successor costs is latency: a device-wide fence about 400 cycles
  // behind stores, an atomic 690 (1570 with acquire and release folded in, which fences twice), a
  // load 300 to 600.  So the successor list comes in while the task runs; after the task one CTA
  // barrier collects its stores, warp 0 fences once, decrements the counters with relaxed atomics
  // and fences again, while warps 1 to 4 fetch the records of the first four successors; and the
  // ready successors that are not run here are pushed by the last warp beside the next task's loads.
  // Between tasks of the critical path of the dense N = 1024 factor: 2.0 us before, 1.2 us so.
  const int id_mask = by_class ? (1 << PP_VM_ID_BITS) - 1 : 0x7FFFFFFF;
  int next = -1, par = 0, slot = 0;
  bool next_unfetched = false;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) s_npub = 0;
  for (;;) {
    int id = next;
    if (id < 0) {
      if (by_class) {
        if (warp == 0) {
          id = take_by_class(slots, n_tasks, cls, st, wait_ns, lane);
          if (lane == 0) s_id = id;
        }
      } else if (threadIdx.x == 0) {
        const int idx = atomicAdd(&st->head, 1);
        if (idx < n_tasks) {
          const unsigned long long t_wait = gtimer_ns();
          for (;;) {
            id = ld_acquire(&slots[idx]);
            if (id >= 0) break;
            if (ld_relaxed(&st->error) || ld_relaxed(&st->done) >= n_tasks) { id = -1; break; }
            // the wait is bounded in time (globaltimer), not in polls: a poll's cost varies
            // with the load on L2 and with other grids sharing the SMs
            if ((long long)(gtimer_ns() - t_wait) > wait_ns) {
              if (atomicCAS(&st->error, 0, PP_VM_TIMEOUT) == 0) st->err_info = idx;
              id = -1;
              break;
            }
            __nanosleep(32);
          }
        }
        s_id = id;
      }
      __syncthreads();
      id = s_id;
      if (id < 0) break;
      slot = 0;
    }
    pp_task& T = s_rec[par][slot];
    if (next < 0 || next_unfetched) {
      if (threadIdx.x < (int)(sizeof(pp_task) / 8))
        reinterpret_cast<unsigned long long*>(&T)[threadIdx.x] =
            __ldg(reinterpret_cast<const unsigned long long*>(&tasks[id]) + threadIdx.x);
      __syncthreads();
    }
    if (trace && threadIdx.x == 0) s_t0 = globaltimer_ns();
    const int nsucc = T.n_succ, sbeg = T.succ_begin;
    if (warp == 7) {
      // push what the previous task left ready, and fetch this task's successor list
      const int count = s_npub;
      if (count > 0 && by_class) {
        push_by_class(slots, n_tasks, cls, lane < count ? s_pub[lane] : -1, lane);
      } else if (count > 0) {
        int base = 0;
        if (lane == 0) base = atomicAdd(&st->tail, count);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (lane < count) st_release(&slots[base + lane], s_pub[lane]);
      }
      if (lane < nsucc)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(&s_succ[par][lane])), "l"(&succ[sbeg + lane])
                     : "memory");
      cp_async_commit();
    }
    int err = PP_VM_OK;
    const bool ok = run_task(T, smem, tc, err);
    if (warp == 7) cp_async_wait<0>();
    __syncthreads();  // the task's stores, and the successor list
    if (warp == 0) {
      __threadfence();
      if (lane == 0) {
        if (!ok && atomicCAS(&st->error, 0, PP_VM_BAD_TASK) == 0) st->err_info = id;
        if (err != PP_VM_OK && atomicCAS(&st->error, 0, err) == 0) st->err_info = id;
        if (trace) {
          trace[3 * (size_t)id] = s_t0;
          trace[3 * (size_t)id + 1] = globaltimer_ns();
          trace[3 * (size_t)id + 2] = smid() | ((unsigned long long)blockIdx.x << 32);
        }
      }
      const int mine = lane < nsucc ? s_succ[par][lane] : -1;
      const bool ready = mine >= 0 && atom_add_relaxed(&counters[mine & id_mask], -1) == 1;
      for (int q = 32; q < nsucc; q += 32) {
        const int sq = q + lane < nsucc ? succ[sbeg + q + lane] : -1;
        const bool now = sq >= 0 && atom_add_relaxed(&counters[sq & id_mask], -1) == 1;
        if (now) __threadfence();
        if (by_class) push_by_class(slots, n_tasks, cls, now ? sq : -1, lane);
        else if (now) st_release(&slots[atomicAdd(&st->tail, 1)], sq);
      }
      __threadfence();  // the other predecessors' stores are visible from here on
      const unsigned all = __ballot_sync(0xffffffffu, ready);
      const int keep = __ffs((int)all) - 1;
      const unsigned rest = all & (all - 1);
      if (ready && lane != keep) s_pub[__popc(rest & ((1u << lane) - 1))] = mine;
      if (lane == 0) {
        s_npub = __popc(rest);
        s_keep = keep;
        atomicAdd(&st->done, 1);
      }
    } else if (warp <= 4 && warp - 1 < nsucc) {
      const pp_task* rec = &tasks[s_succ[par][warp - 1] & id_mask];
      if (lane < (int)(sizeof(pp_task) / 8))
        reinterpret_cast<unsigned long long*>(&s_rec[par ^ 1][warp - 1])[lane] =
            __ldg(reinterpret_cast<const unsigned long long*>(rec) + lane);
    }
    __syncthreads();
    const int keep = s_keep;
    next = keep >= 0 ? s_succ[par][keep] & id_mask : -1;  // while the last warp fetches the next list
    par ^= 1;
    next_unfetched = keep >= 4;
    slot = keep >= 0 && keep < 4 ? keep : 0;
  }
  if (use_tc) {
    // an MMA group whose completion was never observed still owns the accumulators:
    // give it one more bounded wait before the columns are returned
    if (tc.pending) {
      mbar_wait(tc.mbar, tc.phase ^ 1u, tc.limit);
      // a BF16 task that gave up may still have bulk copies and MMAs in flight: they finish
      // within microseconds; give them a bounded 2 ms before the columns are returned
      const unsigned long long t0 = gtimer_ns();
      while (gtimer_ns() - t0 < 2000000ull) __nanosleep(1000);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if ((threadIdx.x >> 5) == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tc.tmem), "r"(TC_TMEM_COLS)
                   : "memory");
    }
  }
}

// ------------------------------------------------------------------------- residuals
// r = b - A x, one warp per row; columns of A read once per RHS block
__global__ void dense_residual_kernel(const double* __restrict__ A, int lda, int n, const double* __restrict__ x,
                                      const double* __restrict__ b, double* __restrict__ r, int nrhs) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= n) return;
  const double* a = A + (size_t)warp * lda;
  for (int q = 0; q < nrhs; ++q) {
    double s = 0.0;
    for (int j = lane; j < n; j += 32) s = fma(a[j], x[(size_t)j * nrhs + q], s);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0) r[(size_t)warp * nrhs + q] = b[(size_t)warp * nrhs + q] - s;
  }
}

// One third-order correction of an estimate y0 of 1/a: with e = 1 - a y0,
// 1/a = y0 (1 - e)^-1 = y0 (1 + e + e^2 + O(e^3)) (geometric series).  For |e| < 2^-19 the
// truncated terms are below 2^-57 relative: the result is within a few ulps of double, the
// accuracy of two Newton steps at 3 instead of 4 operations.
__device__ __forceinline__ double rcp_refine(double a, double y0) {
  const double e = fma(-a, y0, 1.0);
  return fma(y0, fma(e, e, e), y0);
}
// The distance of a squared one: y0 estimates 1 / sqrt(max(d2, 1e-300)), s0 = d2 y0 and
// e = 1 - s0 y0 = 1 - d2 y0^2; then sqrt(d2) = s0 (1 - e)^(-1/2) = s0 (1 + e/2 + 3e^2/8 + O(e^3))
// (binomial series, truncated terms below 2^-58 relative for |e| < 2^-19).  Exact zero on the
// diagonal and for coincident points, an absolute error below 1e-150 for 0 < d2 < 1e-300, a few ulps
// elsewhere; no number stays none.
__device__ __forceinline__ double distance_from(double d2, double y0) {
  const double s0 = d2 * y0;
  const double e = fma(-s0, y0, 1.0);
  return fma(s0 * e, fma(0.375, e, 0.5), s0);
}
// An overflowed d2 counts as 2^1023.  Both bounds are put on the upper word, by which the estimate goes: the
// FP64 pipe is the full one in the residual kernels (one column, 32 jobs of 8192: 4% of a refined
// batch; with a comparison in FP64 the product of 8 columns takes 8% longer).
__device__ __forceinline__ double distance_of(double d2) {
  const int up = __double2hiint(d2), hi = up == 0x7ff00000 ? 0x7fe00000 : up, lo = __double2loint(d2);
  // 0x01a56e1f: upper word of 1e-300
  return distance_from(__hiloint2double(hi, lo), rsqrt_est(__hiloint2double(max(hi, 0x01a56e1f), lo)));
}
// Entry of the kernel matrix at distance d.
template <int KIND>
__device__ __forceinline__ double kernel_at(double d, double p0, double inv_p0) {
  constexpr double c = KIND == 1 ? 4.0 * 3.14159265358979323846 : 1.0;
  if (KIND <= 1) {
    const double x = c * (d + p0);
    return rcp_refine(x, rcp_est(x));
  }
  if (KIND == 2) return exp(-d * inv_p0);
  const double s = 1.7320508075688772 * d * inv_p0;
  return (1.0 + s) * exp(-s);
}

// The same entry evaluated in FP32 with the hardware's approximate reciprocal square root,
// exponential and division: relative error of a few 1e-7 (the exponential's argument is
// rounded to FP32, so for the exp / Matern kernels the error grows like |argument| * 6e-8).
// Used only by the low-precision products of the Krylov steps, never by a residual that
// certifies a result.
template <int KIND>
__device__ __forceinline__ float kernel_eval_f32(float d2, float p0, float inv_p0) {
  const float d = d2 * rsqrtf(fmaxf(d2, 1e-30f));
  if (KIND <= 1) {
    constexpr float c = KIND == 1 ? 12.566370614359172f : 1.0f;
    return __fdividef(1.0f, c * (d + p0));
  }
  if (KIND == 2) return __expf(-d * inv_p0);
  const float sv = 1.7320508f * d * inv_p0;
  return (1.0f + sv) * __expf(-sv);
}

// C[m x k] = K(P_I, P_J) B (PP_OP_KMUL): a thread per row of C, the columns j of the kernel
// matrix in chunks of KM_JC whose points and B rows are staged in shared memory (read by all
// threads as broadcasts); points padded to three coordinates with zeros.  The distance is bounded below in
// FP64 and not above: distance_of here, a few instructions longer or shorter, shifts the VM's code and made
// every other instruction 2 to 5% slower.
#define KM_JC 128
template <int KIND>
__device__ __noinline__ void kmul_impl(const pp_task& T, double* smem) {
  const int m = T.m, n = T.n, k = T.k, dim = T.l;
  const double p0 = T.alpha, inv_p0 = KIND >= 2 ? 1.0 / p0 : 0.0;
  double* C = T.p[0];
  const double *PI = T.p[1], *PJ = T.p[2], *B = T.p[3];
  const int ldc = T.ld[0], ldi = T.ld[1], ldj = T.ld[2], ldb = T.ld[3];
  double* sp = smem;               // KM_JC x 3
  double* sb = smem + KM_JC * 3;   // KM_JC x PP_VM_MAX_RANK
  for (int r0 = 0; r0 < m; r0 += NT) {
    const int r = r0 + threadIdx.x;
    double pr[3] = {0.0, 0.0, 0.0};
    if (r < m)
      for (int d = 0; d < dim; ++d) pr[d] = ldcg(&PI[(size_t)r * ldi + d]);
    double acc[PP_VM_MAX_RANK];
#pragma unroll
    for (int c = 0; c < PP_VM_MAX_RANK; ++c) acc[c] = 0.0;
    for (int j0 = 0; j0 < n; j0 += KM_JC) {
      const int jc = min(KM_JC, n - j0);
      __syncthreads();
      for (int e = threadIdx.x; e < KM_JC * 3; e += NT) {
        const int j = e / 3, d = e % 3;
        sp[e] = (j < jc && d < dim) ? ldcg(&PJ[(size_t)(j0 + j) * ldj + d]) : 0.0;
      }
      for (int e = threadIdx.x; e < jc * PP_VM_MAX_RANK; e += NT) {
        const int j = e / PP_VM_MAX_RANK, c = e % PP_VM_MAX_RANK;
        sb[e] = c < k ? ldcg(&B[(size_t)(j0 + j) * ldb + c]) : 0.0;
      }
      __syncthreads();
      for (int j = 0; j < jc; ++j) {
        const double u0 = pr[0] - sp[3 * j], u1 = pr[1] - sp[3 * j + 1], u2 = pr[2] - sp[3 * j + 2];
        const double d2 = fma(u2, u2, fma(u1, u1, u0 * u0));
        const double a = kernel_at<KIND>(distance_from(d2, rsqrt_est(fmax(d2, 1e-300))), p0, inv_p0);
#pragma unroll
        for (int c = 0; c < PP_VM_MAX_RANK; ++c) acc[c] = fma(a, sb[j * PP_VM_MAX_RANK + c], acc[c]);
      }
    }
    if (r < m)
      for (int c = 0; c < k; ++c) C[(size_t)r * ldc + c] = acc[c];
  }
  __syncthreads();
}

__device__ __noinline__ void dev_kmul(const pp_task& T, double* smem) {
  switch (T.ctrl) {
    case 0: kmul_impl<0>(T, smem); break;
    case 1: kmul_impl<1>(T, smem); break;
    case 2: kmul_impl<2>(T, smem); break;
    default: kmul_impl<3>(T, smem); break;
  }
}

#define KR_SEG 128   /* columns per partial sum of the one-column products */
#define KW_SEG 256   /* and of the wider ones (kernel_residual_wide) */
// Jobs of one batched residual launch, passed by value (kernel parameter space): job j owns
// the launch's work items [first, next job's first) — tile pairs of the residual kernel,
// elements of the update and reduction kernels.
#define KR_LAUNCH_JOBS 64
struct ResidLaunch {
  struct Job {
    const double* pts;
    double* x;
    const double* dx;
    const double* b;
    double* r;
    double* part;
    double p0, shift;
    long long first;
    int n, nrhs, T, pad;
  } job[KR_LAUNCH_JOBS];
  int njobs;
};

// the job that owns work item `key` (the last job whose first <= key)
__device__ __forceinline__ int resid_job_of(const ResidLaunch& L, long long key) {
  int lo = 0, hi = L.njobs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (L.job[mid].first <= key) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// KR_SEG steps of one warp over a tile pair: lane l takes column (l + s) mod KR_SEG at step s.
// COL: also accumulate a_ij x_i into the warp's column sums (off-diagonal tiles); EDGE: skip
// columns at or past jn (the caller skips rows past n).  DUP: the tile's points, x and column
// sums are stored twice over (2 KR_SEG entries), so the column is addressed as l + s without
// the wrap-around; column c's sums are then split between entries c and c + KR_SEG.
template <int KIND, int DIM, int NR, bool COL, bool EDGE, bool DUP>
__device__ __forceinline__ void residual_steps(const double* sp, const double* sx, double* colw, const double (&pi)[DIM],
                                               const double (&xi)[NR], double (&acc)[NR], int lane, int jn, double p0,
                                               double inv_p0) {
#pragma unroll 4
  for (int st = 0; st < KR_SEG; ++st) {
    const int jj = DUP ? lane + st : (lane + st) & (KR_SEG - 1);
    // past the ragged edge the entry is masked, not skipped: a lane that skipped steps could
    // run ahead of the others into a column another lane is still updating.  For the same
    // reason each step's column-sum updates end with a warp barrier: seen from one thread the
    // next step's column is another address, so without it the compiler may load it before
    // the neighbouring lane has stored its update there
    const bool live = !EDGE || ((lane + st) & (KR_SEG - 1)) < jn;
    double d2 = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      const double u = pi[d] - sp[jj * DIM + d];
      d2 = fma(u, u, d2);
    }
    const double ak = kernel_at<KIND>(distance_of(d2), p0, inv_p0);
    const double a = live ? ak : 0.0;
#pragma unroll
    for (int q = 0; q < NR; ++q) acc[q] = fma(a, sx[jj * NR + q], acc[q]);
    if (COL) {
#pragma unroll
      for (int q = 0; q < NR; ++q) colw[jj * NR + q] = fma(a, xi[q], colw[jj * NR + q]);
      __syncwarp();
    }
  }
}

// residual_steps with the entries evaluated in FP32 from FP32 copies of the points (spf, pif);
// the products are still accumulated in FP64.  The skewed walk keeps the lanes of a warp on
// distinct columns only while they take their steps together: columns past the ragged edge are
// masked (entry 0) instead of skipped, and the column sums' read-modify-writes of one step end
// with a warp barrier, so no lane can run a step ahead of another into the same column.
template <int KIND, int DIM, int NR, bool COL, bool EDGE, bool DUP>
__device__ __forceinline__ void residual_steps_lowp(const float* spf, const double* sx, double* colw,
                                                    const float (&pif)[DIM], const double (&xi)[NR], double (&acc)[NR],
                                                    int lane, int jn, float p0, float inv_p0) {
#pragma unroll 4
  for (int st = 0; st < KR_SEG; ++st) {
    const int jj = DUP ? lane + st : (lane + st) & (KR_SEG - 1);
    const bool live = !EDGE || ((lane + st) & (KR_SEG - 1)) < jn;
    float d2 = 0.0f;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      const float u = pif[d] - spf[jj * DIM + d];
      d2 = fmaf(u, u, d2);
    }
    const float a32 = kernel_eval_f32<KIND>(d2, p0, inv_p0);
    const double a = live ? (double)a32 : 0.0;
#pragma unroll
    for (int q = 0; q < NR; ++q) acc[q] = fma(a, sx[jj * NR + q], acc[q]);
    if (COL) {
#pragma unroll
      for (int q = 0; q < NR; ++q) colw[jj * NR + q] = fma(a, xi[q], colw[jj * NR + q]);
      __syncwarp();
    }
  }
}

// Symmetric form of the partial products (kernel matrices are symmetric): a CTA takes the
// tile pair (I, J), I <= J, of KR_SEG x KR_SEG tiles of one job and evaluates each entry once.
// Thread t owns row I*KR_SEG + t: a_ij x_j goes to its register sums (part[J][i]); for I < J,
// a_ij x_i goes to the column sums of row j (part[I][j]) through per-warp accumulators in
// shared memory, walked on a skewed diagonal (lane l visits column (l + s) mod KR_SEG at step
// s, so the lanes of a warp never touch the same column) and added in warp order at the end.
// Every (segment, row) partial is written once, by one CTA: deterministic, no atomics, and the
// same bits whatever the other jobs of the launch.
// LOWP: entries evaluated in FP32 (residual_steps_lowp), for the Krylov steps' products.
template <int KIND, int DIM, int NR, bool LOWP>
__global__ void __launch_bounds__(KR_SEG) kernel_residual_sym(const __grid_constant__ ResidLaunch L) {
  constexpr int W = KR_SEG / 32;
  constexpr bool DUP = NR == 1;             // one RHS: tile stored twice over (residual_steps)
  constexpr int SW = DUP ? 2 * KR_SEG : KR_SEG;
  __shared__ double sp[SW * DIM];
  __shared__ float spf[LOWP ? SW * DIM : 1];
  __shared__ double sx[SW * NR];
  __shared__ double col[W][SW * NR];
  const ResidLaunch::Job& jb = L.job[resid_job_of(L, (long long)blockIdx.x)];
  const double* __restrict__ pts = jb.pts;
  const double* __restrict__ x = jb.x;
  double* __restrict__ part = jb.part;
  const int n = jb.n, nrhs = jb.nrhs, T = jb.T;
  const double p0 = jb.p0, shift = jb.shift;
  // (I, J) of the job's pair index b over the upper triangle, row by row:
  // b = I T - I (I - 1) / 2 + (J - I)
  const long long b = (long long)blockIdx.x - jb.first;
  const double tt = 2.0 * T + 1.0;
  int I = (int)floor((tt - sqrt(tt * tt - 8.0 * (double)b)) * 0.5);
  auto row_start = [&](int r) { return (long long)r * T - (long long)r * (r - 1) / 2; };
  while (I > 0 && row_start(I) > b) --I;
  while (row_start(I + 1) <= b) ++I;
  const int J = I + (int)(b - row_start(I));
  const int t = threadIdx.x, w = t >> 5, lane = t & 31;
  const int i = I * KR_SEG + t, j0 = J * KR_SEG;
  const double inv_p0 = 1.0 / p0;
  for (int e = t; e < SW * DIM; e += KR_SEG) {
    const int e0 = e % (KR_SEG * DIM), jj = e0 / DIM;
    sp[e] = j0 + jj < n ? pts[(size_t)j0 * DIM + e0] : 0.0;
    if (LOWP) spf[e] = (float)sp[e];
  }
  for (int e = t; e < SW * NR; e += KR_SEG) {
    const int e0 = e % (KR_SEG * NR), jj = e0 / NR, q = e0 % NR;
    sx[e] = (j0 + jj < n && q < nrhs) ? x[(size_t)(j0 + jj) * nrhs + q] : 0.0;
  }
  for (int e = t; e < W * SW * NR; e += KR_SEG) (&col[0][0])[e] = 0.0;
  const int ir = min(i, n - 1);
  double pi[DIM], xi[NR], acc[NR];
#pragma unroll
  for (int d = 0; d < DIM; ++d) pi[d] = pts[(size_t)ir * DIM + d];
#pragma unroll
  for (int q = 0; q < NR; ++q) {
    xi[q] = (i < n && q < nrhs) ? x[(size_t)ir * nrhs + q] : 0.0;
    acc[q] = 0.0;
  }
  __syncthreads();
  const bool offdiag = I != J;
  const int jn = min(KR_SEG, n - j0);
  const bool full = jn == KR_SEG && I * KR_SEG + KR_SEG <= n;  // full tiles: no per-entry predicates
  if constexpr (LOWP) {
    float pif[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) pif[d] = (float)pi[d];
    const float p0f = (float)p0, ip0f = (float)inv_p0;
    if (full) {
      if (offdiag) residual_steps_lowp<KIND, DIM, NR, true, false, DUP>(spf, sx, col[w], pif, xi, acc, lane, jn, p0f, ip0f);
      else residual_steps_lowp<KIND, DIM, NR, false, false, DUP>(spf, sx, col[w], pif, xi, acc, lane, jn, p0f, ip0f);
    } else if (i < n) {
      if (offdiag) residual_steps_lowp<KIND, DIM, NR, true, true, DUP>(spf, sx, col[w], pif, xi, acc, lane, jn, p0f, ip0f);
      else residual_steps_lowp<KIND, DIM, NR, false, true, DUP>(spf, sx, col[w], pif, xi, acc, lane, jn, p0f, ip0f);
    }
  } else if (full) {
    if (offdiag) residual_steps<KIND, DIM, NR, true, false, DUP>(sp, sx, col[w], pi, xi, acc, lane, jn, p0, inv_p0);
    else residual_steps<KIND, DIM, NR, false, false, DUP>(sp, sx, col[w], pi, xi, acc, lane, jn, p0, inv_p0);
  } else if (i < n) {  // ragged edge of the matrix
    if (offdiag) residual_steps<KIND, DIM, NR, true, true, DUP>(sp, sx, col[w], pi, xi, acc, lane, jn, p0, inv_p0);
    else residual_steps<KIND, DIM, NR, false, true, DUP>(sp, sx, col[w], pi, xi, acc, lane, jn, p0, inv_p0);
  }
  if (!offdiag && i < n) {  // the diagonal entry's shift
#pragma unroll
    for (int q = 0; q < NR; ++q) acc[q] = fma(shift, xi[q], acc[q]);
  }
  if (i < n)
    for (int q = 0; q < nrhs; ++q) part[((size_t)J * n + i) * nrhs + q] = acc[q];
  if (offdiag) {
    __syncthreads();
    const int jrow = j0 + t;
    if (jrow < n)
      for (int q = 0; q < nrhs; ++q) {
        double v = col[0][t * NR + q];
        if (DUP) v += col[0][(t + KR_SEG) * NR + q];
#pragma unroll
        for (int ww = 1; ww < W; ++ww) {
          v += col[ww][t * NR + q];
          if (DUP) v += col[ww][(t + KR_SEG) * NR + q];
        }
        part[((size_t)I * n + jrow) * nrhs + q] = v;
      }
  }
}

// The symmetric form for two and more right-hand sides, eight at a time (blockIdx.y: the group of
// eight): a CTA takes the tile pair (I, J), I <= J, of KW_SEG x KW_SEG tiles and evaluates each entry
// once; both products run on the FP64 tensor cores.  In an 8 x 8 block lane (a, b) = (l / 4, l % 4)
// evaluates entries (a, b) and (a, b + 4): as they are, they are the A fragments of E X_J, whose sums
// stay in the warp's registers; turned by four shuffles they are those of E^T X_I.  A warp owns 32
// rows, whose points, right-hand sides and sums it keeps in registers, and walks the columns in
// blocks of 32; in each of 8 phases the warps are on different blocks, so that the column sums are
// added in shared memory by one warp at a time and in a fixed order.  Every (segment, row) partial is
// written once, by one CTA: deterministic, no atomics.
// Bound by the FP64 pipe: 15 operations per entry and, with eight columns, 4 tensor instructions per
// 64 entries, as much again.  On a B200, 3-D Laplace: N = 65536,
// 8 columns 9.7 -> 5.8 ms (before: a row-block form that evaluated every entry twice), 3 columns 20.8 ->
// 5.6 ms (before: column sums of every entry read and written in shared memory).
#define KW_LDX 10  /* doubles between the rows of a staged right-hand side block: 2 mod 8 */
// kernel_at(distance_of(d2)) with c (d + p0) as c d + c p0: a few ulps apart, one operation less
template <int KIND>
__device__ __forceinline__ double kernel_eval_wide(double d2, double p0, double cp0, double inv_p0) {
  const double d = distance_of(d2);
  if (KIND <= 1) {
    constexpr double c = KIND == 1 ? 4.0 * 3.14159265358979323846 : 1.0;
    const double x = fma(c, d, cp0);
    return rcp_refine(x, rcp_est(x));
  }
  if (KIND == 2) return exp(-d * inv_p0);
  const double s = 1.7320508075688772 * d * inv_p0;
  return (1.0 + s) * exp(-s);
}
template <int KIND, int DIM>
__global__ void __launch_bounds__(KW_SEG) kernel_residual_wide(const __grid_constant__ ResidLaunch L) {
  extern __shared__ __align__(16) double kw_smem[];
  double* xj = kw_smem;                    // KW_SEG x KW_LDX: right-hand sides of the columns
  double* col = xj + KW_SEG * KW_LDX;      // KW_SEG x KW_LDX: column sums
  double* pj = col + KW_SEG * KW_LDX;      // KW_SEG x DIM: points of the columns
  const ResidLaunch::Job& jb = L.job[resid_job_of(L, (long long)blockIdx.x)];
  const double* __restrict__ pts = jb.pts;
  const double* __restrict__ x = jb.x;
  double* __restrict__ part = jb.part;
  const int n = jb.n, nrhs = jb.nrhs, T = jb.T, q0 = 8 * blockIdx.y;
  if (q0 >= nrhs) return;
  const double p0 = jb.p0, cp0 = (KIND == 1 ? 4.0 * 3.14159265358979323846 : 1.0) * p0, inv_p0 = 1.0 / p0;
  // (I, J) of the job's pair index over the upper triangle, row by row (as kernel_residual_sym)
  const long long b = (long long)blockIdx.x - jb.first;
  const double tt = 2.0 * T + 1.0;
  int I = (int)floor((tt - sqrt(tt * tt - 8.0 * (double)b)) * 0.5);
  auto row_start = [&](int r) { return (long long)r * T - (long long)r * (r - 1) / 2; };
  while (I > 0 && row_start(I) > b) --I;
  while (row_start(I + 1) <= b) ++I;
  const int J = I + (int)(b - row_start(I));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, fa = lane >> 2, fb = lane & 3;
  const int i0 = I * KW_SEG + 32 * warp, j0 = J * KW_SEG;
  // places past the last point take that point: an entry there is one of the matrix, so its product with a
  // zero of x or of xi is zero wherever the sums it goes to are numbers
  for (int e = tid; e < KW_SEG * DIM; e += KW_SEG) pj[e] = pts[(size_t)min(j0 + e / DIM, n - 1) * DIM + e % DIM];
  for (int e = tid; e < KW_SEG * 8; e += KW_SEG) {
    const int r = e >> 3, q = e & 7;
    xj[r * KW_LDX + q] = (j0 + r < n && q0 + q < nrhs) ? x[(size_t)(j0 + r) * nrhs + q0 + q] : 0.0;
    col[r * KW_LDX + q] = 0.0;
  }
  double pi[4][DIM], xi[4][2], acc[4][2];
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int i = min(i0 + 8 * t + fa, n - 1);
#pragma unroll
    for (int d = 0; d < DIM; ++d) pi[t][d] = pts[(size_t)i * DIM + d];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = i0 + 8 * t + 4 * h + fb;
      xi[t][h] = (r < n && q0 + fa < nrhs) ? x[(size_t)r * nrhs + q0 + fa] : 0.0;
      acc[t][h] = 0.0;
    }
  }
  const bool offdiag = I != J;
#pragma unroll 1
  for (int ph = 0; ph < 8; ++ph) {
    __syncthreads();
    const int cb = 32 * ((warp + ph) & 7);
#pragma unroll 1
    for (int c0 = cb; c0 < cb + 32; c0 += 8) {
      if (j0 + c0 >= n) break;
      double p[2][DIM];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int d = 0; d < DIM; ++d) p[h][d] = pj[(c0 + 4 * h + fb) * DIM + d];
      const double x0 = xj[(c0 + fb) * KW_LDX + fa], x1 = xj[(c0 + 4 + fb) * KW_LDX + fa];
      double s0 = 0.0, s1 = 0.0;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        double e[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          double d2 = 0.0;
#pragma unroll
          for (int d = 0; d < DIM; ++d) {
            const double u = pi[t][d] - p[h][d];
            d2 = fma(u, u, d2);
          }
          e[h] = kernel_eval_wide<KIND>(d2, p0, cp0, inv_p0);
        }
        dmma(acc[t][0], acc[t][1], e[0], x0);
        dmma(acc[t][0], acc[t][1], e[1], x1);
        if (offdiag) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            // entry (4 h + fb, fa) of the block: lane (4 h + fb, fa % 4), its first or second entry
            const int src = (4 * h + fb) * 4 + (fa & 3);
            const double v0 = __shfl_sync(0xffffffffu, e[0], src), v1 = __shfl_sync(0xffffffffu, e[1], src);
            dmma(s0, s1, fa < 4 ? v0 : v1, xi[t][h]);
          }
        }
      }
      if (offdiag) {
        double* c = col + (c0 + fa) * KW_LDX + 2 * fb;
        c[0] += s0;
        c[1] += s1;
      }
    }
  }
  // the diagonal entries' shift, and the row sums
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int i = i0 + 8 * t + fa;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int q = q0 + 2 * fb + h;
      if (i < n && q < nrhs) {
        const double v = offdiag ? acc[t][h] : fma(jb.shift, x[(size_t)i * nrhs + q], acc[t][h]);
        part[((size_t)J * n + i) * nrhs + q] = v;
      }
    }
  }
  if (offdiag) {
    __syncthreads();
    for (int e = tid; e < KW_SEG * 8; e += KW_SEG) {
      const int r = e >> 3, q = e & 7;
      if (j0 + r < n && q0 + q < nrhs) part[((size_t)I * n + j0 + r) * nrhs + q0 + q] = col[r * KW_LDX + q];
    }
  }
}
template <int DIM>
constexpr size_t kw_smem_bytes() { return sizeof(double) * (2 * KW_SEG * KW_LDX + KW_SEG * DIM); }

// r = b - (sum of the job's segments in order), one thread per (row, rhs) element
__global__ void residual_reduce(const __grid_constant__ ResidLaunch L) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const ResidLaunch::Job& jb = L.job[resid_job_of(L, e)];
  const long long k = e - jb.first, count = (long long)jb.n * jb.nrhs;
  if (k < 0 || k >= count) return;
  double s = 0.0;
  for (int g = 0; g < jb.T; ++g) s += jb.part[g * count + k];
  jb.r[k] = jb.b[k] - s;
}

// x += dx of every job, one thread per element
__global__ void residual_update(const __grid_constant__ ResidLaunch L) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const ResidLaunch::Job& jb = L.job[resid_job_of(L, e)];
  const long long k = e - jb.first, count = (long long)jb.n * jb.nrhs;
  if (k < 0 || k >= count) return;
  jb.x[k] += jb.dx[k];
}

template <int KIND, int DIM>
cudaError_t launch_residual_sym(const ResidLaunch& L, unsigned pairs, int nr, bool lowp, cudaStream_t s) {
  if (!lowp) kernel_residual_sym<KIND, DIM, 1, false><<<pairs, KR_SEG, 0, s>>>(L);
  else if (nr == 1) kernel_residual_sym<KIND, DIM, 1, true><<<pairs, KR_SEG, 0, s>>>(L);
  else kernel_residual_sym<KIND, DIM, 4, true><<<pairs, KR_SEG, 0, s>>>(L);
  return cudaGetLastError();
}

template <int KIND>
cudaError_t launch_residual_sym_dim(int dim, const ResidLaunch& L, unsigned pairs, int nr, bool lowp,
                                    cudaStream_t s) {
  if (dim == 1) return launch_residual_sym<KIND, 1>(L, pairs, nr, lowp, s);
  if (dim == 2) return launch_residual_sym<KIND, 2>(L, pairs, nr, lowp, s);
  return launch_residual_sym<KIND, 3>(L, pairs, nr, lowp, s);
}

template <int KIND, int DIM>
cudaError_t launch_residual_wide(const ResidLaunch& L, unsigned pairs, int nrhs, cudaStream_t s) {
  kernel_residual_wide<KIND, DIM><<<dim3(pairs, (nrhs + 7) / 8), KW_SEG, kw_smem_bytes<DIM>(), s>>>(L);
  return cudaGetLastError();
}

template <int KIND>
cudaError_t launch_residual_wide_dim(int dim, const ResidLaunch& L, unsigned pairs, int nrhs, cudaStream_t s) {
  if (dim == 1) return launch_residual_wide<KIND, 1>(L, pairs, nrhs, s);
  if (dim == 2) return launch_residual_wide<KIND, 2>(L, pairs, nrhs, s);
  return launch_residual_wide<KIND, 3>(L, pairs, nrhs, s);
}

// whether a job's product takes kernel_residual_wide: two and more right-hand sides in FP64
bool resid_wide(const pp_resid_job& j, bool lowp) { return j.nrhs > 4 || (j.nrhs > 1 && !lowp); }

ResidLaunch::Job resid_job(const pp_resid_job& j, bool lowp) {
  ResidLaunch::Job o{};
  o.pts = j.pts;
  o.x = j.x;
  o.dx = j.dx;
  o.b = j.b;
  o.r = j.r;
  o.part = j.part;
  o.p0 = j.p0;
  o.shift = j.shift;
  o.n = j.n;
  o.nrhs = j.nrhs;
  o.T = resid_wide(j, lowp) ? (j.n + KW_SEG - 1) / KW_SEG : (j.n + KR_SEG - 1) / KR_SEG;
  return o;
}

// element-wise launch (update or reduction) over jobs[sel] in chunks of KR_LAUNCH_JOBS
template <typename F>
cudaError_t launch_elementwise(const pp_resid_job* jobs, const std::vector<int>& sel, F kernel, bool lowp, cudaStream_t s) {
  for (size_t c = 0; c < sel.size(); c += KR_LAUNCH_JOBS) {
    ResidLaunch L;
    L.njobs = (int)std::min<size_t>(KR_LAUNCH_JOBS, sel.size() - c);
    long long total = 0;
    for (int q = 0; q < L.njobs; ++q) {
      L.job[q] = resid_job(jobs[sel[c + q]], lowp);
      L.job[q].first = total;
      total += (long long)L.job[q].n * L.job[q].nrhs;
    }
    kernel<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(L);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// Dense blocks of an H-matrix assembled in place from its points (the first step of building it
// on the device): entry (i, j) of the block at rows [r0, r0 + m), columns [c0, c0 + n) is
// K(|p_{r0+i} - p_{c0+j}|), plus the shift on the matrix diagonal, with the residual kernel's
// distance and entry evaluation (the bits of the matrix that the one-column product applies, a few ulps
// from those of the wider one).  One CTA per AS_ROWS rows of a block; blocks passed by value, up to
// AS_LAUNCH_JOBS per launch.
#define AS_LAUNCH_JOBS 64
#define AS_ROWS 16
struct AssembleLaunch {
  struct Job {
    double* a;
    long long first;  // first CTA of the block in the launch
    int ld, r0, c0, m, n, pad;
  } job[AS_LAUNCH_JOBS];
  const double* pts;
  double p0, shift;
  int njobs;
};

template <int KIND, int DIM>
__global__ void __launch_bounds__(256) assemble_dense_kernel(const __grid_constant__ AssembleLaunch L) {
  int lo = 0, hi = L.njobs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (L.job[mid].first <= (long long)blockIdx.x) lo = mid; else hi = mid - 1;
  }
  const AssembleLaunch::Job& jb = L.job[lo];
  const int rb = (int)((long long)blockIdx.x - jb.first) * AS_ROWS;
  const double inv_p0 = 1.0 / L.p0;
  for (int e = threadIdx.x; e < AS_ROWS * jb.n; e += blockDim.x) {
    const int i = rb + e / jb.n, j = e % jb.n;
    if (i >= jb.m) break;  // e only grows: every later element is past the block too
    const int gi = jb.r0 + i, gj = jb.c0 + j;
    double d2 = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      const double u = L.pts[(size_t)gi * DIM + d] - L.pts[(size_t)gj * DIM + d];
      d2 = fma(u, u, d2);
    }
    double a = kernel_at<KIND>(distance_of(d2), L.p0, inv_p0);
    if (gi == gj) a += L.shift;
    jb.a[(size_t)i * jb.ld + j] = a;
  }
}

template <int KIND>
cudaError_t launch_assemble_dim(int dim, const AssembleLaunch& L, unsigned ctas, cudaStream_t s) {
  if (dim == 1) assemble_dense_kernel<KIND, 1><<<ctas, 256, 0, s>>>(L);
  else if (dim == 2) assemble_dense_kernel<KIND, 2><<<ctas, 256, 0, s>>>(L);
  else assemble_dense_kernel<KIND, 3><<<ctas, 256, 0, s>>>(L);
  return cudaGetLastError();
}

// x += dx over `count` elements (the refinement update of a served request)
__global__ void axpy_kernel(double* __restrict__ x, const double* __restrict__ dx, size_t count) {
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < count; e += (size_t)gridDim.x * blockDim.x)
    x[e] += dx[e];
}

// out[0] = max |x|, out[1] = max |r| as the bit patterns of non-negative doubles (their
// integer order is their numeric order, so an integer atomicMax reduces them); out zeroed
// by the caller
__global__ void absmax2_kernel(const double* __restrict__ x, const double* __restrict__ r, size_t count,
                               unsigned long long* out) {
  double mx = 0.0, mr = 0.0;
  for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < count; e += (size_t)gridDim.x * blockDim.x) {
    mx = fmax(mx, fabs(x[e]));
    mr = fmax(mr, fabs(r[e]));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    mr = fmax(mr, __shfl_xor_sync(0xffffffffu, mr, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&out[0], (unsigned long long)__double_as_longlong(mx));
    atomicMax(&out[1], (unsigned long long)__double_as_longlong(mr));
  }
}

// One ACCUM on caller buffers; its scratch (T.tmp) is the static array below.
__global__ void __launch_bounds__(NT) accum_noalloc_kernel(pp_task T) {
  extern __shared__ __align__(16) double smem[];
  dev_lowrank(T);
}

}  // namespace

// Scratch of pp_lowrank_accum_noalloc: a file-scope device array, so the entry point never
// allocates.  Every device that loads the library holds it (8 MiB) until the process exits.
// Host code may not use its name as an address: the device address is looked up once per
// device with cudaGetSymbolAddress (below) and passed to the kernel.
#define PP_NOALLOC_SCRATCH_DOUBLES (1 << 20)
static __device__ __align__(256) double g_accum_noalloc_scratch[PP_NOALLOC_SCRATCH_DOUBLES];

long long pp_accum_noalloc_capacity() { return PP_NOALLOC_SCRATCH_DOUBLES; }

long long pp_accum_scratch_doubles(long long ny, int k1, int k2) {
  // dev_lowrank keeps the ny x k1 sketch Y in shared memory while it fits beside the rest of the
  // 180 KB; only a larger Y goes to the task's scratch, and nothing else does
  return accum_y_on_chip(ny, k1, k2) ? 0 : ny * k1;
}

namespace {
// device address of the static scratch array, looked up once per device (std::call_once, so
// two host threads making their first calls at once do not race on the cache)
constexpr int kNoallocMaxDevices = 64;
std::once_flag g_noalloc_once[kNoallocMaxDevices];
double* g_noalloc_addr[kNoallocMaxDevices] = {nullptr};
cudaError_t g_noalloc_err[kNoallocMaxDevices] = {cudaSuccess};
}  // namespace

cudaError_t pp_accum_noalloc_launch(const pp_task& T, long long scratch_doubles, cudaStream_t s) {
  if (scratch_doubles < 0 || scratch_doubles > PP_NOALLOC_SCRATCH_DOUBLES) return cudaErrorInvalidValue;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kNoallocMaxDevices) return cudaErrorInvalidDevice;
  std::call_once(g_noalloc_once[dev], [dev] {  // set-up, once per device, with that device current
    double* p = nullptr;
    g_noalloc_err[dev] = cudaGetSymbolAddress((void**)&p, g_accum_noalloc_scratch);
    g_noalloc_addr[dev] = p;
  });
  if (g_noalloc_err[dev] != cudaSuccess) return g_noalloc_err[dev];
  pp_task t = T;
  t.tmp = g_noalloc_addr[dev];
  // 180 KB of dynamic shared memory, as the VM's ACCUM has; pp_vm_prepare (run at context
  // creation on this device) raised the kernel's limit to that
  accum_noalloc_kernel<<<1, NT, VM_SMEM_BYTES, s>>>(t);
  return cudaGetLastError();
}

size_t pp_vm_smem_bytes() { return VM_SMEM_BYTES; }

int pp_vm_blocks_per_sm() {
  int nb = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, vm_kernel, NT, pp_vm_smem_bytes());
  return nb;
}

namespace {
// Loads one kernel's code now (lazy module loading would otherwise do it at its first launch,
// in the middle of a served request).
template <typename F>
cudaError_t preload(F f) {
  cudaFuncAttributes a;
  return cudaFuncGetAttributes(&a, f);
}
template <int KIND, int DIM>
cudaError_t preload_residual() {
  cudaError_t e = preload(kernel_residual_sym<KIND, DIM, 1, false>);
  if (e == cudaSuccess) e = preload(kernel_residual_sym<KIND, DIM, 1, true>);
  if (e == cudaSuccess) e = preload(kernel_residual_sym<KIND, DIM, 4, true>);
  if (e == cudaSuccess) e = preload(kernel_residual_wide<KIND, DIM>);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(kernel_residual_wide<KIND, DIM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kw_smem_bytes<DIM>());
  return e;
}
template <int KIND>
cudaError_t preload_residual_dims() {
  cudaError_t e = preload_residual<KIND, 1>();
  if (e == cudaSuccess) e = preload_residual<KIND, 2>();
  if (e == cudaSuccess) e = preload_residual<KIND, 3>();
  if (e == cudaSuccess) e = preload(assemble_dense_kernel<KIND, 1>);
  if (e == cudaSuccess) e = preload(assemble_dense_kernel<KIND, 2>);
  if (e == cudaSuccess) e = preload(assemble_dense_kernel<KIND, 3>);
  return e;
}
}  // namespace

cudaError_t pp_vm_prepare() {
  cudaError_t e = cudaFuncSetAttribute(vm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pp_vm_smem_bytes());
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(accum_noalloc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pp_vm_smem_bytes());
  // every kernel of the refinement and serving paths, loaded at context creation
  for (cudaError_t r : {preload(vm_init), preload(residual_reduce), preload(residual_update), preload(axpy_kernel),
                        preload(absmax2_kernel), preload(dense_residual_kernel), preload_residual_dims<0>(),
                        preload_residual_dims<1>(), preload_residual_dims<2>(), preload_residual_dims<3>()})
    if (e == cudaSuccess) e = r;
  return e;
}

cudaError_t pp_vm_run(const pp_vm_launch& L, cudaStream_t s) {
  if (L.n_tasks <= 0) return cudaSuccess;
  const int ib = 256;
  const pp_vm_classes cls = L.classes ? *L.classes : pp_vm_classes{};
  const int by_class = L.classes != nullptr;
  vm_init<<<(L.n_tasks + ib - 1) / ib, ib, 0, s>>>(L.indeg, L.ready, L.n_ready, L.n_tasks, L.counters, L.slots,
                                                  L.state, by_class, cls);
  vm_kernel<<<L.grid, NT, pp_vm_smem_bytes(), s>>>(L.tasks, L.n_tasks, L.succ, L.counters, L.slots, L.state,
                                                   L.wait_ns, L.trace, L.use_tc, by_class, cls);
  return cudaGetLastError();
}

cudaError_t pp_dense_residual(const double* A, int lda, int n, const double* x, const double* b, double* r, int nrhs,
                              cudaStream_t s) {
  const int threads = 256, warps = threads / 32;
  dense_residual_kernel<<<(n + warps - 1) / warps, threads, 0, s>>>(A, lda, n, x, b, r, nrhs);
  return cudaGetLastError();
}

cudaError_t pp_kernel_residual_batch(const pp_resid_job* jobs, int njobs, cudaStream_t s, bool lowp) {
  if (njobs <= 0) return cudaSuccess;
  if (!jobs) return cudaErrorInvalidValue;
  std::vector<int> all, upd;
  for (int q = 0; q < njobs; ++q) {
    const pp_resid_job& j = jobs[q];
    if (j.dim < 1 || j.dim > 3 || j.nrhs < 1 || j.nrhs > 16 || j.n <= 0 || j.kernel < 0 || j.kernel > 3 || !j.pts ||
        !j.x || !j.b || !j.r || !j.part)
      return cudaErrorInvalidValue;
    if (j.kernel <= 1 && !(j.p0 >= 0.0 && std::isfinite(j.p0))) return cudaErrorInvalidValue;
    all.push_back(q);
    if (j.dx) upd.push_back(q);
  }
  cudaError_t e = launch_elementwise(jobs, upd, residual_update, lowp, s);
  if (e != cudaSuccess) return e;
  // tile-pair launches, one per (kernel, dimension, right-hand-side width) group
  for (int kern = 0; kern < 4; ++kern)
    for (int dim = 1; dim <= 3; ++dim)
      for (int nr : {1, 4}) {
        std::vector<int> sel;
        for (int q = 0; q < njobs; ++q)
          if (jobs[q].kernel == kern && jobs[q].dim == dim && (nr == 1 ? jobs[q].nrhs == 1 : (jobs[q].nrhs > 1 && jobs[q].nrhs <= 4)))
            sel.push_back(q);
        for (size_t c = 0; c < sel.size(); c += KR_LAUNCH_JOBS) {
          ResidLaunch L;
          L.njobs = (int)std::min<size_t>(KR_LAUNCH_JOBS, sel.size() - c);
          long long pairs = 0;
          for (int q = 0; q < L.njobs; ++q) {
            L.job[q] = resid_job(jobs[sel[c + q]], lowp);
            L.job[q].first = pairs;
            pairs += (long long)L.job[q].T * (L.job[q].T + 1) / 2;
          }
          if (pairs >= (1LL << 31)) return cudaErrorInvalidValue;
          const bool wide = nr > 1 && !lowp;
          switch (kern) {
            case 0: e = wide ? launch_residual_wide_dim<0>(dim, L, (unsigned)pairs, nr, s) : launch_residual_sym_dim<0>(dim, L, (unsigned)pairs, nr, lowp, s); break;
            case 1: e = wide ? launch_residual_wide_dim<1>(dim, L, (unsigned)pairs, nr, s) : launch_residual_sym_dim<1>(dim, L, (unsigned)pairs, nr, lowp, s); break;
            case 2: e = wide ? launch_residual_wide_dim<2>(dim, L, (unsigned)pairs, nr, s) : launch_residual_sym_dim<2>(dim, L, (unsigned)pairs, nr, lowp, s); break;
            default: e = wide ? launch_residual_wide_dim<3>(dim, L, (unsigned)pairs, nr, s) : launch_residual_sym_dim<3>(dim, L, (unsigned)pairs, nr, lowp, s); break;
          }
          if (e != cudaSuccess) return e;
        }
      }
  // wider right-hand-side blocks: a launch per job
  for (int q = 0; q < njobs; ++q) {
    if (jobs[q].nrhs <= 4) continue;
    ResidLaunch L;
    L.njobs = 1;
    L.job[0] = resid_job(jobs[q], lowp);
    L.job[0].first = 0;
    const long long pairs = (long long)L.job[0].T * (L.job[0].T + 1) / 2;
    if (pairs >= (1LL << 31)) return cudaErrorInvalidValue;
    switch (jobs[q].kernel) {
      case 0: e = launch_residual_wide_dim<0>(jobs[q].dim, L, (unsigned)pairs, jobs[q].nrhs, s); break;
      case 1: e = launch_residual_wide_dim<1>(jobs[q].dim, L, (unsigned)pairs, jobs[q].nrhs, s); break;
      case 2: e = launch_residual_wide_dim<2>(jobs[q].dim, L, (unsigned)pairs, jobs[q].nrhs, s); break;
      default: e = launch_residual_wide_dim<3>(jobs[q].dim, L, (unsigned)pairs, jobs[q].nrhs, s); break;
    }
    if (e != cudaSuccess) return e;
  }
  return launch_elementwise(jobs, all, residual_reduce, lowp, s);
}

cudaError_t pp_kernel_residual(int kernel, double p0, double p1, double diag_shift, const double* pts, int dim, int n,
                               const double* x, const double* b, double* r, int nrhs, double* part,
                               cudaStream_t s) {
  (void)p1;
  pp_resid_job j{};
  j.kernel = kernel;
  j.dim = dim;
  j.n = n;
  j.nrhs = nrhs;
  j.p0 = p0;
  j.shift = diag_shift;
  j.pts = pts;
  j.x = const_cast<double*>(x);  // read only: no update without dx
  j.b = b;
  j.r = r;
  j.part = part;
  return pp_kernel_residual_batch(&j, 1, s);
}

cudaError_t pp_assemble_dense(const pp_assemble_block* blocks, int nblocks, int kernel, int dim, double p0,
                              double shift, const double* pts, cudaStream_t s) {
  if (nblocks <= 0) return cudaSuccess;
  if (!blocks || !pts || dim < 1 || dim > 3 || kernel < 0 || kernel > 3) return cudaErrorInvalidValue;
  if (kernel <= 1 && !(p0 >= 0.0 && std::isfinite(p0))) return cudaErrorInvalidValue;
  for (int c = 0; c < nblocks; c += AS_LAUNCH_JOBS) {
    AssembleLaunch L;
    L.pts = pts;
    L.p0 = p0;
    L.shift = shift;
    L.njobs = std::min(AS_LAUNCH_JOBS, nblocks - c);
    long long ctas = 0;
    for (int q = 0; q < L.njobs; ++q) {
      const pp_assemble_block& b = blocks[c + q];
      if (!b.a || b.m <= 0 || b.n <= 0 || b.ld < b.n || b.r0 < 0 || b.c0 < 0) return cudaErrorInvalidValue;
      L.job[q] = AssembleLaunch::Job{b.a, ctas, b.ld, b.r0, b.c0, b.m, b.n, 0};
      ctas += (b.m + AS_ROWS - 1) / AS_ROWS;
    }
    if (ctas >= (1LL << 31)) return cudaErrorInvalidValue;
    cudaError_t e;
    switch (kernel) {
      case 0: e = launch_assemble_dim<0>(dim, L, (unsigned)ctas, s); break;
      case 1: e = launch_assemble_dim<1>(dim, L, (unsigned)ctas, s); break;
      case 2: e = launch_assemble_dim<2>(dim, L, (unsigned)ctas, s); break;
      default: e = launch_assemble_dim<3>(dim, L, (unsigned)ctas, s); break;
    }
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t pp_axpy(double* x, const double* dx, size_t count, cudaStream_t s) {
  const unsigned blocks = (unsigned)std::min<size_t>((count + 255) / 256, 1184);
  axpy_kernel<<<blocks ? blocks : 1, 256, 0, s>>>(x, dx, count);
  return cudaGetLastError();
}

cudaError_t pp_absmax2(const double* x, const double* r, size_t count, unsigned long long* out, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(out, 0, 2 * sizeof(unsigned long long), s);
  if (e != cudaSuccess) return e;
  const unsigned blocks = (unsigned)std::min<size_t>((count + 255) / 256, 592);
  absmax2_kernel<<<blocks ? blocks : 1, 256, 0, s>>>(x, r, count, out);
  return cudaGetLastError();
}

size_t pp_kernel_residual_part_elems(int n, int nrhs) {
  return (size_t)((n + KR_SEG - 1) / KR_SEG) * n * nrhs;
}
