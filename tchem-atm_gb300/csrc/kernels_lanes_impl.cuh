// Batched TR-BDF2 kernel over a static-order sparse LU.
//
// A CTA advances S samples in step, one Newton iteration of each per round; every shared-memory
// array has the sample as its fastest index. A warp's 32 lanes are S samples x 32 / S slots, and the
// slots share the work of a round by the mechanism's instruction streams (lane_program.hpp): rates
// and species are dealt to the slots and live in registers, the matrix, the factorization and the
// triangular solves are streams of 16-byte packets read ahead from global memory (L1 / L2), the same
// for every sample, with a CTA barrier at the end of each level of the elimination schedule; the
// nearly dense trailing block is inverted in registers, a 2-D grid of slots each holding a tile.
//
// Each sample is at its own step, stage and iteration; what differs is decided once per round by one
// warp from the reduced norms and handed to the slots as a code per sample. A sample that ends
// hands its lane to the next one of the work queue. The right-hand side at a converged stage is the
// one the next round evaluates anyway (the next stage or step starts there), so a Newton iteration
// costs one right-hand side: f(y_n), f(y_gamma) and f(y_{n+1}) need no evaluations of their own.
//
// Why: the dense kernels spend 44 k (LU) to 140 k (Gauss-Jordan) products on a 51-species matrix whose
// sparse factors need 7.8 k, and every index of a sparse factorization costs as much as its product when
// one warp works on one sample. What bounds this one: chains of dependent shared-memory loads and FP64
// instructions (2 lanes per cycle and SM) between barriers, 34 k cycles per round with one sample on the SM,
// 104 k with 16. FP32 with 16 samples: solves 21 k, tail 24 k, sparse factorization 12 k, matrix 11 k,
// right-hand side 9 k, residual product 10 k, error test and norms 16 k. Measured against the dense kernels
// (one GB300): 51 species, one sample over 60 s 93 ms to 54 ms, 4,096 samples over 3,600 s 1.20 s to 1.03 s (FP32), 300 samples
// over 0.1 s 1.02 s to 178 ms (FP64); 120 species, 257 samples over 1 s 451 ms to 213 ms; 300 species, 24 samples over
// 1e-4 s 443 ms to 75 ms (the blocked LU on tensor cores with the matrix in L2); E3SM, 2,000 columns over 1,800 s
// 118 ms to 8.5 ms (FP64). Where a register kernel is the faster one: lanes_pay_for_box in lane_tables.cu.
//
// T = float: the full-Newton FP32 form (FP32 matrix, factors and solves, FP64 residual, one
// refinement sweep with an FP64 Jacobian-vector product per solve). T = double: the plain form.
// A sample whose factorization meets a zero, non-finite or small pivot (a multiplier above
// kLaneMaxGrowth), or that asks for something outside this kernel, is left untouched with status
// kStatusRedo and advanced by the general kernel, which pivots.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "aero_rhs.cuh"
#include "engine.cuh"
#include "kernels_lanes.hpp"
#include "lane_program.hpp"

namespace tchem_gb {
namespace lanes {

// Largest multiplier |l_ik| accepted without pivoting. The diagonal of I - c J is 1 + c x (loss
// rate), and a column's off-diagonal entries are c x (loss rate) x yield, so multipliers stay near
// the yields (about 1); partial pivoting would bound them by 1. Columns whose pivot row has no further entries are
// not asked (lane_program.cpp).
constexpr float kLaneMaxGrowth = 64.f;
constexpr int kLaneMaxGrowthHi = 0x40500000;  // the high word of 64.0

// Control block: doubles then ints, each [S].
enum CtlD { D_T, D_DT, D_TEND, D_DTMIN, D_DTMAX, D_COEF, D_COUNT };
enum CtlI { I_SMP, I_CODE, I_LAST, I_ITER, I_MAXITER, I_NEWT, I_MAXNEWT, I_TRY, I_STAGE, I_BAD, I_STEPS, I_REJ, I_NFAIL,
            I_NITS, I_NOK0, I_NATT, I_STATUS, I_ACC, I_COUNT,
            I_SLOT = I_LAST };  // the mechanism slot is needed only until the first step begins
enum Code {
  C_ITER = 0,     // next Newton iteration of the same stage
  C_STAGE = 1,    // stage 1 converged: stage 2 starts at y_gamma
  C_STEP = 2,     // stage 2 converged: error test
  C_RETRY = 3,    // Newton failed: the step starts again with half the step size
  C_IDLE = 4,     // no sample
  C_FRESH = 5,    // new sample
  C_ACCEPT = 6,   // step accepted, the next one starts
  C_REJECT = 7,   // step rejected
  C_DONE = 8      // finished: write the outputs
};

static_assert(D_COUNT == kLaneControlDoubles && I_COUNT == kLaneControlInts, "control block size");

template <typename T>
struct Num;
template <>
struct Num<float> {
  // hardware reciprocal (1 ulp): the factors are refined against an FP64 residual
  static __device__ __forceinline__ float recip(float v) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
  }
  static __device__ __forceinline__ float mul_sub(float a, float b, float c) { return fmaf(-a, b, c); }
};
template <>
struct Num<double> {
  // Newton-Raphson on the hardware's approximate reciprocal: each pass squares its relative error
  // (2^-20 at worst), the last one in residual form. A short dependent chain; zero, infinite and NaN
  // pivots give NaN or 0, which the caller rejects.
  static __device__ __forceinline__ double recip(double v) {
    double r;
    asm volatile("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(v));
    r = fma(fma(-v, r, 1.0), r, r);
    r = fma(fma(-v, r, 1.0), r, r);
    return r;
  }
  static __device__ __forceinline__ double mul_sub(double a, double b, double c) { return fma(-a, b, c); }
};

// Shared memory by 32-bit address: the sections' places are run-time values, and an address in the
// generic window would cost 64-bit arithmetic for each of a packet's eight operands.
template <typename T>
struct Shared {
  uint32_t at;
  __device__ __forceinline__ T load(uint32_t index) const;
  __device__ __forceinline__ void store(uint32_t index, T v) const;
};
template <>
__device__ __forceinline__ float Shared<float>::load(uint32_t index) const {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at + 4u * index));
  return v;
}
template <>
__device__ __forceinline__ void Shared<float>::store(uint32_t index, float v) const {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + 4u * index), "f"(v) : "memory");
}
template <>
__device__ __forceinline__ double Shared<double>::load(uint32_t index) const {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(at + 8u * index));
  return v;
}
template <>
__device__ __forceinline__ void Shared<double>::store(uint32_t index, double v) const {
  asm volatile("st.shared.f64 [%0], %1;" ::"r"(at + 8u * index), "d"(v) : "memory");
}
__device__ __forceinline__ uint4 load_packet(uint32_t at) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at));
  return v;
}
__device__ __forceinline__ uint32_t load_byte(uint32_t at) {
  uint32_t v;
  asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(at));
  return v;
}

// AERO: the gas-aerosol problem (T = double): rows of q and slots of d beyond the reactions'.
template <typename T, int S, int W, bool AERO>
struct Kernel {
  static constexpr int NT = 32 * W;
  static constexpr int SPW = 32 / S;  // slots per warp
  static constexpr int P = NT / S;    // slots
  static constexpr bool kRefine = sizeof(T) == 4;
  static constexpr int kPair = sizeof(T) == 4 ? 2 : 1;  // rounds of the factor stream worked on at a time
  static constexpr int NPS = lane_species(P), NRS = lane_reactions(P);

  const LaneParams& K;
  unsigned char* sm;
  int s, sl, slot, warp;  // sample, slot in the warp, slot, warp
  int bad;

  __device__ __forceinline__ uint32_t base() const { return static_cast<uint32_t>(__cvta_generic_to_shared(sm)); }
  __device__ __forceinline__ Shared<T> lus() const { return Shared<T>{base() + K.s.lu + s * static_cast<uint32_t>(sizeof(T))}; }
  __device__ __forceinline__ T* lu() const { return reinterpret_cast<T*>(sm + K.s.lu) + s; }
  __device__ __forceinline__ double* xs() const { return reinterpret_cast<double*>(sm + K.s.x) + s; }
  __device__ __forceinline__ double* vs() const { return reinterpret_cast<double*>(sm + K.s.v) + s; }
  // the iterate in T precision: in v's place until v is written (T = double: x itself)
  __device__ __forceinline__ T* xt() const { return reinterpret_cast<T*>(sm + (kRefine ? K.s.v : K.s.x)) + s; }
  __device__ __forceinline__ double* qs() const { return reinterpret_cast<double*>(sm + K.s.q) + s; }
  __device__ __forceinline__ T* ds() const { return reinterpret_cast<T*>(sm + K.s.q) + s; }  // while q is not needed
  __device__ __forceinline__ Shared<double> xsh() const { return Shared<double>{base() + K.s.x + s * 8u}; }
  __device__ __forceinline__ Shared<double> qsh() const { return Shared<double>{base() + K.s.q + s * 8u}; }
  __device__ __forceinline__ double& cd(int k, int smp) const {
    return reinterpret_cast<double*>(sm + K.s.ctl)[k * S + smp];
  }
  __device__ __forceinline__ int& ci(int k, int smp) const {
    return reinterpret_cast<int*>(sm + K.s.ctl + D_COUNT * S * sizeof(double))[k * S + smp];
  }
  __device__ __forceinline__ int& flag(int k) const {
    return reinterpret_cast<int*>(sm + K.s.ctl + S * (D_COUNT * sizeof(double) + I_COUNT * sizeof(int)))[k];
  }

  // This slot's packets of a stream, a warp's rounds SPW apart: in shared memory where it is resident.
  __device__ __forceinline__ const uint4* packets(int id, int& rounds) const {
    const int2 w = reinterpret_cast<const int2*>(sm + K.s.prog)[id * W + warp];
    rounds = w.y;
    return (K.s.stream[id] ? reinterpret_cast<const uint4*>(sm + K.s.stream[id]) : K.p.packets[id]) + w.x + sl;
  }

  // The rounds of one stream in order, two at a time, each pair read while the one before it is
  // worked on. A stream that is not resident goes through shared memory in chunks: every warp copies
  // its own packets (cp.async) into its part of [buf, buf + bytes), one half while it reads the other,
  // so that the warp waits once per chunk for L2 and not once per pair.
  struct Reader {
    const uint4* src;       // staged: the next packets to copy; read from global memory: the next packet
    uint32_t p, buf;        // shared addresses: the next packet, the warp's chunks
    int cap, left, in_chunk, half;
    bool global;
    uint4 a, b;
  };
  __device__ __forceinline__ void fetch(Reader& r) const {
    const int n = min(r.cap, r.left) * SPW, lane = threadIdx.x & 31;
    const uint32_t dst = r.buf + r.half * r.cap * SPW * 16;
    for (int i = lane; i < n; i += 32)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * i), "l"(r.src + i) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
    r.src += r.cap * SPW;
    r.left -= r.cap;
    r.half ^= 1;
  }
  __device__ __forceinline__ void next_chunk(Reader& r) const {
    __syncwarp();  // every lane has read the half that is filled now
    if (r.left > 0) {
      fetch(r);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      r.half ^= 1;
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncwarp();
    r.p = r.buf + (r.half * r.cap * SPW + sl) * 16;
    r.in_chunk = r.cap;
  }
  template <int N>
  __device__ __forceinline__ void read(Reader& r) const {
    if (r.global) {
      r.a = __ldg(r.src);
      if (N == 2) r.b = __ldg(r.src + SPW);
    } else {
      r.a = load_packet(r.p);
      if (N == 2) r.b = load_packet(r.p + SPW * 16);
    }
  }
  template <int N>
  __device__ __forceinline__ Reader open(int id, uint2 chunk, int& rounds) const {
    Reader r;
    const int2 w = reinterpret_cast<const int2*>(sm + K.s.prog)[id * W + warp];
    rounds = w.y;
    r.cap = static_cast<int>(chunk.y / (2 * W * SPW * 16)) & ~1;
    r.in_chunk = 1 << 30;
    r.global = false;
    r.src = K.p.packets[id] + w.x;
    if (K.s.stream[id]) {
      r.p = base() + K.s.stream[id] + (w.x + sl) * 16;
    } else if (r.cap >= 2) {
      r.buf = base() + chunk.x + warp * 2 * r.cap * SPW * 16;
      r.left = rounds;
      r.half = 0;
      fetch(r);
      next_chunk(r);
    } else {
      r.global = true;
      r.src += sl;
    }
    read<N>(r);
    return r;
  }
  // The next N rounds (beyond the last, what is read is not used; the streams end with a spare pair).
  template <int N>
  __device__ __forceinline__ void advance(Reader& r) const {
    r.p += N * SPW * 16;
    if (r.global) r.src += N * SPW;
    r.in_chunk -= N;
    if (r.in_chunk <= 0) next_chunk(r);
    read<N>(r);
  }
  // Shared memory that a stream's chunks may use: what the streams' placement left, or sections whose
  // contents are not needed at that time.
  __device__ __forceinline__ uint2 chunk_space(uint32_t off, uint32_t end) const {
    return K.s.stage_bytes >= end - off ? make_uint2(K.s.stage, K.s.stage_bytes) : make_uint2(off, end - off);
  }

  // Factor and substitution packets: the entry minus three products, times a pivot's reciprocal (the one
  // entry where nothing scales it), or the reciprocal of a pivot.
  template <int PAIR>
  __device__ __forceinline__ void run_lu(int id, uint2 chunk) {
    const Shared<T> A = lus();
    uint32_t rounds = base() + K.s.prog + K.p.level_at[id] + warp;
    const int levels = K.p.levels[id];
    if (levels == 0) return;
    int total, n = static_cast<int>(load_byte(rounds));
    Reader r = open<PAIR>(id, chunk, total);
#pragma unroll 1
    for (int lv = 0; lv < levels; ++lv) {
      rounds += lv + 1 < levels ? W : 0;
      const int next = static_cast<int>(load_byte(rounds));
#pragma unroll 1
      for (; n > 0; n -= PAIR) {
        if constexpr (PAIR == 2)
          packet_pair(A, r);
        else
          packet(A, r);
      }
      n = next;
      __syncthreads();
    }
  }
  // FP32 factor: two packets with all their operands read first, so that a level costs one chain of
  // dependent loads; no branches, unused places multiply zeros.
  __device__ __forceinline__ void packet_pair(Shared<T> A, Reader& r) {
    const uint4 w0 = r.a, w1 = r.b;
    const uint32_t d0 = (w0.x & 0x7fffu) * S, d1 = (w1.x & 0x7fffu) * S;
    const T e0 = A.load(d0), e1 = A.load(d1);
    const T a0 = A.load((w0.y & 0xffffu) * S), b0 = A.load((w0.y >> 16) * S);
    const T a1 = A.load((w0.z & 0xffffu) * S), b1 = A.load((w0.z >> 16) * S);
    const T a2 = A.load((w0.w & 0xffffu) * S), b2 = A.load((w0.w >> 16) * S);
    const T s0 = A.load(((w0.x >> LP_SCALE_SHIFT) & 511u) * S);
    const T f0 = A.load((w1.y & 0xffffu) * S), g0 = A.load((w1.y >> 16) * S);
    const T f1 = A.load((w1.z & 0xffffu) * S), g1 = A.load((w1.z >> 16) * S);
    const T f2 = A.load((w1.w & 0xffffu) * S), g2 = A.load((w1.w >> 16) * S);
    const T s1 = A.load(((w1.x >> LP_SCALE_SHIFT) & 511u) * S);
    advance<2>(r);
    T u = Num<T>::mul_sub(a2, b2, Num<T>::mul_sub(a1, b1, Num<T>::mul_sub(a0, b0, e0)));
    T v = Num<T>::mul_sub(f0, g0, (w1.x & LP_CONT) ? u : e1);
    v = Num<T>::mul_sub(f2, g2, Num<T>::mul_sub(f1, g1, v));
    A.store(d0, finish(w0.x, u * s0, u, Num<T>::recip(u)));
    A.store(d1, finish(w1.x, v * s1, v, Num<T>::recip(v)));
  }
  __device__ __forceinline__ T finish(uint32_t h, T scaled, T acc, T inverse) {
    const T v = (h & LP_PIVOT) ? inverse : scaled;
    if ((h & LP_PIVOT) && (!(fabs(acc) > T(0)) || !(fabs(v) > T(0)))) bad = 1;  // zero, infinite or NaN
    if ((h & LP_LCOL) && !(fabs(v) <= T(kLaneMaxGrowth))) bad = 1;
    return v;
  }
  // One packet. FP64: an instruction takes 16 cycles of the SM's pipe whatever its lanes do with it, so
  // a warp leaves out what none of its slots needs (volatile: the compiler must not compute both sides
  // and select). FP32 (substitutions): no branches; unused places multiply zeros.
  __device__ __forceinline__ void packet(Shared<T> A, Reader& r) {
    const uint4 w = r.a;
    const uint32_t dst = (w.x & 0x7fffu) * S;
    T acc = A.load(dst);
    const T a0 = A.load((w.y & 0xffffu) * S), b0 = A.load((w.y >> 16) * S);
    const T a1 = A.load((w.z & 0xffffu) * S), b1 = A.load((w.z >> 16) * S);
    const T a2 = A.load((w.w & 0xffffu) * S), b2 = A.load((w.w >> 16) * S);
    const T scale = A.load(((w.x >> LP_SCALE_SHIFT) & 511u) * S);
    advance<1>(r);
    if constexpr (sizeof(T) == 4) {
      A.store(dst, scale * Num<T>::mul_sub(a2, b2, Num<T>::mul_sub(a1, b1, Num<T>::mul_sub(a0, b0, acc))));
    } else {
      const uint32_t any = __shfl_sync(kFullMask, w.x, 0);  // the warp's flags, as a uniform value
      if (any & LP_ONE) acc_product(acc, a0, b0);
      if (any & LP_TWO) acc_product(acc, a1, b1);
      if (any & LP_THREE) acc_product(acc, a2, b2);
      T v = acc;
      if (any & LP_SCALED) asm volatile("mul.rn.f64 %0, %0, %1;" : "+d"(v) : "d"(scale));
      if (any & LP_PIVOTS) {
        const T p = Num<T>::recip(acc);
        if (w.x & LP_PIVOT) {
          v = p;
          if (!(fabs(acc) > T(0)) || !(fabs(v) > T(0))) bad = 1;
        }
      }
      // the size as the high word of |v| (monotonic): below 64, and neither infinite nor NaN
      if ((w.x & LP_LCOL) && (__double2hiint(static_cast<double>(v)) & 0x7fffffff) > kLaneMaxGrowthHi) bad = 1;
      A.store(dst, v);
    }
  }
  static __device__ __forceinline__ void acc_product(double& acc, double a, double b) {
    asm volatile("{\n .reg .f64 t;\n neg.f64 t, %1;\n fma.rn.f64 %0, t, %2, %0;\n}" : "+d"(acc) : "d"(a), "d"(b));
  }

  // In-place Gauss-Jordan inverse of the tail block, no pivot search, two pivots per step: slot (pr, pc) of
  // the grid holds rows pr TR .. and columns pc TC .. in registers. Per step the owners of the two pivot
  // rows and columns publish them (double-buffered, one barrier); every slot solves the 2 x 2 pivot
  // block for its columns and updates its tile with both rows. A step is bound by the instructions around
  // the products and by its chain of barrier, loads and reciprocals: two pivots share them, a slot's
  // stretch of a published row or column is one or two wide loads, and products go two to an instruction
  // (fma.rn.f32x2). One pivot per step took 27.8 k cycles for 16 samples' 32 x 32 blocks, two pivots with
  // cyclic tiles and single loads 24.0 k (one sample: 6.4 k; 160 x 160: 113 k), this 23.8 k (5.7 k; 113 k).
  template <int TR>
  __device__ __forceinline__ void invert_tail() {
    constexpr int GR = lane_grid_rows(P), GC = lane_grid_cols(P), F = GR / GC, N = TR * GR, TC = N / GC;
    constexpr int ST = lane_tail_stride(P, N), NS = N + 4;  // lane_publish_stride
    constexpr uint32_t kRow = NS * S * 4;                   // bytes of one published row of all samples
    static_assert(TC % 2 == 0, "pivots go in pairs");
    const Shared<T> A{lus().at + K.p.tail * S * static_cast<uint32_t>(sizeof(T))};
    const uint32_t pub = base() + K.s.q + s * NS * 4;  // [2]: two rows, two columns, each [S][NS]
    const int pr = slot / GC, pc = slot % GC;
    uint64_t t[TR][TC / 2];  // pairs of columns
#pragma unroll
    for (int a = 0; a < TR; ++a)
#pragma unroll
      for (int c = 0; c < TC / 2; ++c) {
        const int at = (pr * TR + a) * ST + pc * TC + 2 * c;
        t[a][c] = pack(A.load(at * S), A.load((at + 1) * S));
      }
    const uint32_t my_row = pub + pc * TC * 4, my_col = pub + 2 * kRow + pr * TR * 4;
    publish_step<TR, TC>(t, my_row, my_col, pr, pc, 0, 0);
    __syncthreads();
#pragma unroll 1
    for (int blk = 0; blk < GC; ++blk) {
#pragma unroll
      for (int c0 = 0; c0 < TC; c0 += 2) {
        // pivots k, k + 1: tile columns c0, c0 + 1 of grid column blk; tile rows and grid rows
        constexpr int kLast = TC - 2;
        const int k = blk * TC + c0;
        const int buf = (k >> 1) & 1;
        const int ra = c0 % TR, rb = (c0 + 1) % TR, ga = blk * F + c0 / TR, gb = blk * F + (c0 + 1) / TR;
        const uint32_t x0 = my_row + buf * 4 * kRow, y0 = my_col + buf * 4 * kRow;
        const uint32_t piv = pub + buf * 4 * kRow + k * 4;
        // [a b; c d] = [1 0; l 1] [a b; 0 e]
        float pa, pb, pcc, pd;
        load_pair(piv, pa, pb);
        load_pair(piv + kRow, pcc, pd);
        uint64_t u[TC / 2], v[TC / 2];
        float l0[TR], l1[TR];
        load_row<TC>(x0, u);
        load_row<TC>(x0 + kRow, v);
        load_col<TR>(y0, l0);
        load_col<TR>(y0 + kRow, l1);
        const float p0 = Num<float>::recip(pa), l = pcc * p0, w = pb * p0, e = fmaf(-l, pb, pd), p1 = Num<float>::recip(e);
        float big0 = 0.f, big1 = 0.f;
#pragma unroll
        for (int a = 0; a < TR; ++a) {
          big0 = fmaxf(big0, fabsf(l0[a]));
          big1 = fmaxf(big1, fabsf(fmaf(-l0[a], w, l1[a])));  // after the first elimination
        }
        // a multiplier beyond the bound, or a zero or non-finite pivot (its own row's multiplier is 1)
        if (!(big0 * fabsf(p0) <= kLaneMaxGrowth) || !(big1 * fabsf(p1) <= kLaneMaxGrowth)) bad = 1;
        if (!(fabsf(pa) > 0.f) || !(fabsf(e) > 0.f)) bad = 1;
        // rows of the inverse of the pivot block times the pivot rows
        const uint64_t ml = pack(-l, -l), mw = pack(-w, -w), pp0 = pack(p0, p0), pp1 = pack(p1, p1);
#pragma unroll
        for (int c = 0; c < TC / 2; ++c) {
          v[c] = mul2(pp1, fma2(ml, u[c], v[c]));
          u[c] = fma2(mw, v[c], mul2(pp0, u[c]));
        }
        if (pc == blk) {  // the pivot columns become the inverse's
          const float n1 = -l * p1;
          v[c0 / 2] = pack(n1, p1);
          u[c0 / 2] = pack(fmaf(-w, n1, p0), -w * p1);
#pragma unroll
          for (int a = 0; a < TR; ++a) t[a][c0 / 2] = 0ull;
        }
#pragma unroll
        for (int a = 0; a < TR; ++a) {
          const uint64_t m0 = pack(-l0[a], -l0[a]), m1 = pack(-l1[a], -l1[a]);
#pragma unroll
          for (int c = 0; c < TC / 2; ++c) t[a][c] = fma2(m1, v[c], fma2(m0, u[c], t[a][c]));
        }
        if (pr == ga) {
#pragma unroll
          for (int c = 0; c < TC / 2; ++c) t[ra][c] = u[c];
        }
        if (pr == gb) {
#pragma unroll
          for (int c = 0; c < TC / 2; ++c) t[rb][c] = v[c];
        }
        const uint32_t nrow = my_row + (buf ^ 1) * 4 * kRow, ncol = my_col + (buf ^ 1) * 4 * kRow;
        if (c0 < kLast) {
          publish_step<TR, TC>(t, nrow, ncol, pr, pc, blk, c0 + 2);
          __syncthreads();
        } else if (blk + 1 < GC) {
          publish_step<TR, TC>(t, nrow, ncol, pr, pc, blk + 1, 0);
          __syncthreads();
        }
      }
    }
#pragma unroll
    for (int a = 0; a < TR; ++a)
#pragma unroll
      for (int c = 0; c < TC / 2; ++c) {
        const int at = (pr * TR + a) * ST + pc * TC + 2 * c;
        float lo, hi;
        unpack(t[a][c], lo, hi);
        A.store(at * S, lo);
        A.store((at + 1) * S, hi);
      }
    __syncthreads();
  }
  // Publishes the pivot rows and columns of tile column c (and c + 1) of grid column blk.
  template <int TR, int TC>
  __device__ __forceinline__ void publish_step(const uint64_t (&t)[TR][TC / 2], uint32_t row, uint32_t col, int pr, int pc,
                                               int blk, int c) const {
    constexpr int F = lane_grid_rows(P) / lane_grid_cols(P);
    constexpr uint32_t kRow = (TR * lane_grid_rows(P) + 4) * S * 4;
    if (pr == blk * F + c / TR) store_row<TC>(row, t[c % TR]);
    if (pr == blk * F + (c + 1) / TR) store_row<TC>(row + kRow, t[(c + 1) % TR]);
    if (pc == blk) {
      float lo[TR], hi[TR];
#pragma unroll
      for (int a = 0; a < TR; ++a) unpack(t[a][c / 2], lo[a], hi[a]);
      store_col<TR>(col, lo);
      store_col<TR>(col + kRow, hi);
    }
  }
  static __device__ __forceinline__ uint64_t pack(float lo, float hi) {
    uint64_t v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
  }
  static __device__ __forceinline__ void unpack(uint64_t v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
  }
  static __device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t v;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
    return v;
  }
  static __device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t v;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
  }
  static __device__ __forceinline__ void load_pair(uint32_t at, float& a, float& b) {
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(a), "=f"(b) : "r"(at));
  }
  template <int N>
  static __device__ __forceinline__ void load_row(uint32_t at, uint64_t (&v)[N / 2]) {
    if constexpr (N % 4 == 0) {
#pragma unroll
      for (int i = 0; i < N / 2; i += 2)
        asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v[i]), "=l"(v[i + 1]) : "r"(at + 8 * i));
    } else {
#pragma unroll
      for (int i = 0; i < N / 2; ++i) asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v[i]) : "r"(at + 8 * i));
    }
  }
  template <int N>
  static __device__ __forceinline__ void store_row(uint32_t at, const uint64_t (&v)[N / 2]) {
    if constexpr (N % 4 == 0) {
#pragma unroll
      for (int i = 0; i < N / 2; i += 2)
        asm volatile("st.shared.v2.u64 [%0], {%1, %2};" ::"r"(at + 8 * i), "l"(v[i]), "l"(v[i + 1]) : "memory");
    } else {
#pragma unroll
      for (int i = 0; i < N / 2; ++i) asm volatile("st.shared.u64 [%0], %1;" ::"r"(at + 8 * i), "l"(v[i]) : "memory");
    }
  }
  template <int N>
  static __device__ __forceinline__ void load_col(uint32_t at, float (&v)[N]) {
    if constexpr (N % 4 == 0) {
#pragma unroll
      for (int i = 0; i < N; i += 4)
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(v[i]), "=f"(v[i + 1]), "=f"(v[i + 2]), "=f"(v[i + 3])
                     : "r"(at + 4 * i));
    } else if constexpr (N % 2 == 0) {
#pragma unroll
      for (int i = 0; i < N; i += 2) load_pair(at + 4 * i, v[i], v[i + 1]);
    } else {
#pragma unroll
      for (int i = 0; i < N; ++i) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v[i]) : "r"(at + 4 * i));
    }
  }
  template <int N>
  static __device__ __forceinline__ void store_col(uint32_t at, const float (&v)[N]) {
    if constexpr (N % 4 == 0) {
#pragma unroll
      for (int i = 0; i < N; i += 4)
        asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(at + 4 * i), "f"(v[i]), "f"(v[i + 1]),
                     "f"(v[i + 2]), "f"(v[i + 3])
                     : "memory");
    } else if constexpr (N % 2 == 0) {
#pragma unroll
      for (int i = 0; i < N; i += 2)
        asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(at + 4 * i), "f"(v[i]), "f"(v[i + 1]) : "memory");
    } else {
#pragma unroll
      for (int i = 0; i < N; ++i) asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + 4 * i), "f"(v[i]) : "memory");
    }
  }

  // The tail of the factorization, where there is one.
  __device__ __forceinline__ void tail() {
    if constexpr (kRefine) {
      switch (K.p.n_t / lane_grid_rows(P)) {
        case 0: break;
        case lane_tile(P, W, 0): invert_tail<lane_tile(P, W, 0)>(); break;
        case lane_tile(P, W, 1): invert_tail<lane_tile(P, W, 1)>(); break;
        case lane_tile(P, W, 2): invert_tail<lane_tile(P, W, 2)>(); break;
        default: invert_tail<lane_tile(P, W, 3)>(); break;
      }
    }
  }

  // The tail rows of the vector section times the tail's inverse. Rows beyond the species (a tail larger than
  // the matrix) are inputs of zero for the whole launch and are not written: a non-finite sample would leave NaNs
  // there for every later sample of the lane.
  __device__ __forceinline__ void apply_tail() {
    if constexpr (kRefine) {
      const int n = K.p.n_t, rows = K.p.m - K.p.ms;
      if (n == 0) return;
      const Shared<T> z{lus().at + (K.p.vec + K.p.ms) * S * static_cast<uint32_t>(sizeof(T))};
      constexpr int NR = (lane_tile(P, W, 3) * lane_grid_rows(P) + P - 1) / P;
      T out[NR];
#pragma unroll
      for (int a = 0; a < NR; ++a) {
        const int i = slot + P * a;
        T s0 = T(0), s1 = T(0);
        if (i < rows) {
          const Shared<T> row{lus().at + (K.p.tail + i * lane_tail_stride(P, n)) * S * static_cast<uint32_t>(sizeof(T))};
#pragma unroll 4
          for (int j = 0; j < n; j += 2) {
            const T a0 = row.load(j * S), z0 = z.load(j * S), a1 = row.load((j + 1) * S), z1 = z.load((j + 1) * S);
            s0 = Num<T>::mul_sub(a0, -z0, s0);
            s1 = Num<T>::mul_sub(a1, -z1, s1);
          }
        }
        out[a] = s0 + s1;
      }
      __syncthreads();
#pragma unroll
      for (int a = 0; a < NR; ++a)
        if (slot + P * a < rows) z.store((slot + P * a) * S, out[a]);
      __syncthreads();
    }
  }

  // The assembled matrix's factors.
  __device__ __forceinline__ void factorize() {
    run_lu<kPair>(LS_FACTOR, chunk_space(K.s.q, K.s.ctl));  // q is free
    tail();
  }

  // z = (I - c J)^-1 z on the vector section; q is free.
  __device__ __forceinline__ void solve() {
    run_lu<1>(LS_FORWARD, chunk_space(K.s.q, K.s.ctl));
    apply_tail();
    run_lu<1>(LS_BACKWARD, chunk_space(K.s.q, K.s.ctl));
  }

  // Rates of progress into q: q = keff x[a] x[b] x[c] (x[m] = 1).
  __device__ __forceinline__ void rates(const double (&keff)[NRS]) const {
    const Shared<double> x = xsh(), q = qsh();
    int n_rounds;
    const uint4* p = packets(LS_REACTIONS, n_rounds);
#pragma unroll
    for (int k = 0; k < NRS; ++k) {
      if (k >= K.p.nrs) break;
      const uint4 f = p[k * SPW];
      if (k * P + slot < K.p.R) {
        double v = keff[k] * x.load((f.x & 0xffffu) * S);
        if ((f.y >> 16) > 1) v *= x.load((f.x >> 16) * S);
        if ((f.y >> 16) > 2) v *= x.load((f.y & 0xffffu) * S);
        q.store(f.w * S, v);
      }
    }
  }

  // dq/dx . v into q.
  __device__ __forceinline__ void rate_derivatives(const double (&keff)[NRS]) const {
    const Shared<double> x = xsh(), q = qsh(), v{base() + K.s.v + s * 8u};
    int n_rounds;
    const uint4* p = packets(LS_REACTIONS, n_rounds);
#pragma unroll
    for (int k = 0; k < NRS; ++k) {
      if (k >= K.p.nrs) break;
      const uint4 f = p[k * SPW];
      if (k * P + slot < K.p.R) {
        const int a = (f.x & 0xffffu) * S, b = (f.x >> 16) * S, c = (f.y & 0xffffu) * S, n = f.y >> 16;
        double d = n > 0 ? v.load(a) : 0.0;
        if (n >= 2) {
          const double xa = x.load(a), xb = x.load(b);
          d = fma(d, xb, xa * v.load(b));
          if (n > 2) d = fma(d, x.load(c), xa * xb * v.load(c));
        }
        q.store(f.w * S, keff[k] * d);
      }
    }
  }

  // out[k] = sum of nu q over the slot's species.
  __device__ __forceinline__ void net(double (&out)[NPS]) const {
    const Shared<double> q = qsh();
    int n_rounds, e = 0;
    const uint4* p = packets(LS_NET, n_rounds);
    const int4 ends = reinterpret_cast<const int4*>(sm + K.s.prog + LS_COUNT * W * sizeof(int2))[warp];
    const int end[kLaneSegments] = {ends.x, ends.y, ends.z, ends.w};
#pragma unroll
    for (int k = 0; k < NPS; ++k) {
      double a0 = 0.0, a1 = 0.0;
#pragma unroll 2
      for (; e < end[k]; e += 2) {
        const uint4 u = p[0], w = p[SPW];
        p += 2 * SPW;
        a0 = fma(__hiloint2double(static_cast<int>(u.w), static_cast<int>(u.z)), q.load(u.x * S), a0);
        a1 = fma(__hiloint2double(static_cast<int>(w.w), static_cast<int>(w.z)), q.load(w.x * S), a1);
      }
      out[k] = a0 + a1;
    }
  }

  // dq/dx per factor slot into d, from the iterate in T precision.
  __device__ __forceinline__ void factor_slots(const T (&kt)[NRS]) const {
    const Shared<T> x{base() + (kRefine ? K.s.v : K.s.x) + s * static_cast<uint32_t>(sizeof(T))};
    const Shared<T> d{base() + K.s.q + s * static_cast<uint32_t>(sizeof(T))};
    int n_rounds;
    const uint4* p = packets(LS_REACTIONS, n_rounds);
#pragma unroll
    for (int k = 0; k < NRS; ++k) {
      if (k >= K.p.nrs) break;
      const uint4 f = p[k * SPW];
      if (k * P + slot < K.p.R) {
        const int n = f.y >> 16;
        const uint32_t o = f.z * S;
        if (n == 1) {
          d.store(o, kt[k]);
        } else if (n > 1) {
          const T a = x.load((f.x & 0xffffu) * S), b = x.load((f.x >> 16) * S);
          if (n == 2) {
            d.store(o, kt[k] * b);
            d.store(o + S, kt[k] * a);
          } else {
            const T c = x.load((f.y & 0xffffu) * S);
            d.store(o, kt[k] * b * c);
            d.store(o + S, kt[k] * a * c);
            d.store(o + 2 * S, kt[k] * a * b);
          }
        }
      }
    }
  }

  // ---- gas-aerosol problem ----
  // The section holds, per sample: simc [nS][4] (accommodation coefficient, mean free path, partitioning
  // constant, kg m-3 -> ppm), nc [nP], part [nP][5] (radius, mean molecular weight, mass, moles, r / 3V),
  // tr [nP nS][4] (condensation coefficient, and the factors of 1 / density, 1 / molecular weight and the
  // entry's own species in the transfer's derivative by a species of the particle), unit [nP nA].
  //
  // unit: what one kg m-3 in a particle is in the gas phase, number concentration x kg m-3 -> ppm of the species' own
  // molecular weight, as a power of two. The matrix is that of the scaled unknowns: a bound on multipliers means
  // nothing between rows in kg m-3 and rows in ppm, which are 1e5 and more apart, and powers of two leave every
  // digit of the factors as it was.
  __device__ __forceinline__ double* ext(int i) const { return reinterpret_cast<double*>(sm + K.s.ext) + i * S + s; }
  __device__ __forceinline__ int nc_at() const { return 4 * K.aero.nS; }
  __device__ __forceinline__ int part_at() const { return 4 * K.aero.nS + K.aero.nP; }
  __device__ __forceinline__ int tr_at() const { return 4 * K.aero.nS + 6 * K.aero.nP; }
  __device__ __forceinline__ int unit_at() const { return tr_at() + 4 * K.aero.nP * K.aero.nS; }
  // 1 / u for a power of two
  static __device__ __forceinline__ double inverse_unit(double u) {
    return __longlong_as_double(0x7fe0000000000000ll - __double_as_longlong(u));
  }
  static __device__ __forceinline__ double power_of_two_below(double v) {
    const int e = (__double2hiint(v) >> 20) & 0x7ff;  // 0, subnormal, infinite, NaN: no scaling
    return __hiloint2double((e < 1023 - 300 || e > 1023 + 300 ? 1023 : e) << 20, 0);
  }

  // Temperature and pressure terms and number concentrations of the new sample in lane c, by all threads.
  __device__ __forceinline__ void aero_setup_sample(int c, int smp, double p, double Tk) const {
    const AeroDev& A = K.aero;
    double* e = reinterpret_cast<double*>(sm + K.s.ext) + c;
    for (int is = threadIdx.x; is < A.nS; is += NT) {
      double sc[4];
      fp64::aero_entry_terms(A.sim_idx + 3 * is, A.sim_par + 7 * is, Tk, p, sc);
      for (int i = 0; i < 4; ++i) e[(4 * is + i) * S] = sc[i];
    }
    for (int ip = threadIdx.x; ip < A.nP; ip += NT)
      e[(nc_at() + ip) * S] = K.number_conc[static_cast<size_t>(smp) * A.nP + ip];
    for (int i = threadIdx.x; i < A.nP * A.nA; i += NT)
      e[(unit_at() + i) * S] = power_of_two_below(K.number_conc[static_cast<size_t>(smp) * A.nP + i / A.nA] *
                                                  (fp64::kAeroRuniv / A.mw[i % A.nA] * 1.0e6 * Tk / p));
  }
  __device__ __forceinline__ double ode(int i) const { return xs()[__ldg(K.p.pos + i) * S]; }

  // Radius, mean molecular weight and mass of the particles: src/core/impl/TChem_Impl_SingleParticleUtils.hpp:50-170.
  __device__ __forceinline__ void aero_particles() const {
    const AeroDev& A = K.aero;
    for (int ip = slot; ip < A.nP; ip += P) {
      const int first = A.m_gas + ip * A.nA;
      double volume = A.vol0, mass = A.mass0, moles = A.moles0;
      for (int k = 0; k < A.nA; ++k) {
        const double x = ode(first + k);
        volume += x / A.density[k];
        mass += x;
        moles += x / A.mw[k];
      }
      const double radius = pow(volume * 3.0 / 4.0 / fp64::kAeroPi, 1.0 / 3.0);
      const int o = part_at() + 5 * ip;
      *ext(o) = radius;
      *ext(o + 1) = mass / moles;
      *ext(o + 2) = mass;
      *ext(o + 3) = moles;
      *ext(o + 4) = radius / (3.0 * volume);
    }
  }

  // The (particle, entry) pairs' rows of q: src/core/impl/TChem_Impl_SIMPOL_phase_transfer.hpp:60-150, and the
  // terms of their derivatives.
  __device__ __forceinline__ void aero_transfers() const {
    const AeroDev& A = K.aero;
    double* q = qs();
    for (int e = slot; e < A.nP * A.nS; e += P) {
      const int ip = e / A.nS, is = e - ip * A.nS, o = part_at() + 5 * ip;
      const double alpha = *ext(4 * is), mfp = *ext(4 * is + 1), keq = *ext(4 * is + 2), D = A.sim_par[7 * is + 4];
      const double radius = *ext(o), avg_mw = *ext(o + 1), mass = *ext(o + 2), moles = *ext(o + 3);
      const double kn = mfp / radius;
      const double num = 0.75 * alpha * (1.0 + kn), den = kn * kn + (1.0 + 0.283 * alpha) * kn + 0.75 * alpha;
      const double ffs = num / den;
      double cond = 4.0 * fp64::kAeroPi * radius * D * ffs;
      double evap = cond * 1.0 * (keq * avg_mw / mass);
      const double xg = ode(A.sim_idx[3 * is + 1]), xa = ode(A.sim_idx[3 * is] + ip * A.nA);
      // d cond / dr: radius enters directly and through kn = mfp / radius
      const double dffs = (0.75 * alpha * den - num * (2.0 * kn + 1.0 + 0.283 * alpha)) / (den * den);
      const double dcond = 4.0 * fp64::kAeroPi * D * (ffs - kn * dffs), keq_m = keq / moles;
      const int t = tr_at() + 4 * e;
      *ext(t) = cond;
      *ext(t + 1) = dcond * *ext(o + 4) * (xg - keq_m * xa);
      *ext(t + 2) = cond * keq_m * xa / moles;
      *ext(t + 3) = -cond * keq_m;
      cond *= xg;
      evap *= xa;
      const double d = -evap + cond;
      q[(K.p.R + 2 * e) * S] = -*ext(nc_at() + ip) * d;
      q[(K.p.R + 2 * e + 1) * S] = d / *ext(4 * is + 3);
    }
  }

  // The pairs' slots of d.
  __device__ __forceinline__ void aero_slots() const {
    const AeroDev& A = K.aero;
    T* d = ds() + (K.p.D - 2 * A.nP * A.nS * (1 + A.nA)) * S;
    for (int i = slot; i < A.nP * A.nS * (1 + A.nA); i += P) {
      const int e = i / (1 + A.nA), c = i - e * (1 + A.nA), ip = e / A.nS, is = e - ip * A.nS, t = tr_at() + 4 * e;
      const int own = A.sim_idx[3 * is] - A.m_gas;
      double v = *ext(t);
      if (c > 0) {
        v = *ext(t + 1) / A.density[c - 1] + *ext(t + 2) / A.mw[c - 1];
        if (own == c - 1) v += *ext(t + 3);
        v *= inverse_unit(*ext(unit_at() + ip * A.nA + c - 1));
      }
      d[2 * i * S] = -*ext(nc_at() + ip) * v;
      d[(2 * i + 1) * S] = v / *ext(4 * is + 3) * *ext(unit_at() + ip * A.nA + own);
    }
  }

  // Entries of I - coef J.
  __device__ __forceinline__ void matrix(T coef) const {
    const Shared<T> A = lus(), d{base() + K.s.q + s * static_cast<uint32_t>(sizeof(T))};
    T acc = T(0);
    // x in T precision (in v's place) has been read; FP64 has no such section
    int n;
    Reader r = open<2>(LS_MATRIX, kRefine ? chunk_space(K.s.v, K.s.q) : make_uint2(K.s.stage, K.s.stage_bytes), n);
#pragma unroll 1
    for (; n > 0; n -= 2) {
      const uint4 w0 = r.a, w1 = r.b;
      // both packets' operands first
      T nu[2], dv[2], nv[2], ev[2];  // FP32 packets hold two contributions, FP64 packets one
      if constexpr (sizeof(T) == 4) {
        nu[0] = __uint_as_float(w0.z), nv[0] = __uint_as_float(w0.w);
        nu[1] = __uint_as_float(w1.z), nv[1] = __uint_as_float(w1.w);
        dv[0] = d.load((w0.y & 0xffffu) * S), ev[0] = d.load((w0.y >> 16) * S);
        dv[1] = d.load((w1.y & 0xffffu) * S), ev[1] = d.load((w1.y >> 16) * S);
      } else {
        nu[0] = __hiloint2double(static_cast<int>(w0.w), static_cast<int>(w0.z));
        nu[1] = __hiloint2double(static_cast<int>(w1.w), static_cast<int>(w1.z));
        dv[0] = d.load(w0.y * S);
        dv[1] = d.load(w1.y * S);
      }
      advance<2>(r);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const uint32_t h = i ? w1.x : w0.x;
        acc = Num<T>::mul_sub(nu[i], -dv[i], (h & LM_START) ? T(0) : acc);
        if (sizeof(T) == 4) acc = Num<T>::mul_sub(nv[i], -ev[i], acc);
        if (h & LM_END) A.store((h & 0x7fffu) * S, Num<T>::mul_sub(coef, acc, (h & LM_DIAG) ? T(1) : T(0)));
      }
    }
  }

  // 0.9 e^(-1/3) clamped to [0.2, 2]: a single-precision start and two Newton-Raphson passes of
  // r <- r + r (1 - e r^3) / 3, each of which squares the relative error (1e-6 at the start). The control
  // warp waits for this chain once per step; outside [0.05, 200] the clamp decides alone.
  static __device__ __forceinline__ double step_factor(double e) {
    if (!(e > 0.05)) return 2.0;
    if (e > 200.0) return 0.2;
    double r = static_cast<double>(exp2f(-log2f(static_cast<float>(e)) * (1.f / 3.f)));
#pragma unroll
    for (int i = 0; i < 2; ++i) r = fma(r * (1.0 / 3.0), fma(-e * r, r * r, 1.0), r);
    return fmax(0.2, fmin(2.0, 0.9 * r));
  }

  // The next try of sample i's step: clamps the step size, or ends the sample.
  __device__ __forceinline__ int begin_try(int i, int code) {
    const double d = 0.5 * (2.0 - sqrt(2.0));
    double dt = fmin(fmax(cd(D_DT, i), cd(D_DTMIN, i)), cd(D_DTMAX, i));
    const double left = cd(D_TEND, i) - cd(D_T, i);
    const bool last = dt >= left;
    if (last) dt = left;
    cd(D_DT, i) = dt;
    ci(I_LAST, i) = last ? 1 : 0;
    ci(I_STAGE, i) = 0;
    ci(I_NEWT, i) = 0;
    if (!(dt > 0.0)) {
      ci(I_STATUS, i) = TCHEM_GB_SAMPLE_DT_UNDERFLOW;
      return C_DONE;
    }
    cd(D_COEF, i) = d * dt;
    return code;
  }
  // The next step of sample i, or its end.
  __device__ __forceinline__ int begin_step(int i, int code) {
    if (!(ci(I_ITER, i) < ci(I_MAXITER, i) && cd(D_T, i) < cd(D_TEND, i))) return C_DONE;
    ci(I_TRY, i) = 0;
    return begin_try(i, code);
  }

  // A slot's value summed (or its maximum taken) over the warp's slots, in every lane.
  template <bool MAX>
  static __device__ __forceinline__ double over_warp(double v) {
#pragma unroll
    for (int o = S; o < 32; o <<= 1) {
      const double w = __shfl_xor_sync(kFullMask, v, o);
      v = MAX ? max_nonneg(v, w) : v + w;
    }
    return v;
  }
  // The larger of two non-negative numbers, which order as their bit patterns: integer compares instead
  // of FP64 ones.
  static __device__ __forceinline__ double max_nonneg(double a, double b) {
    return __longlong_as_double(max(__double_as_longlong(a), __double_as_longlong(b)));
  }

  // Sum (or maximum) over the warps of the W partial values at q[(base + warp) * S], by one warp; the
  // lane's sample is s.
  template <bool MAX>
  __device__ __forceinline__ double reduce(int base) const {
    const double* q = qs();
    double v = 0.0;
#pragma unroll
    for (int k = sl; k < W; k += SPW) {
      const double w = q[(base + k) * S];
      v = MAX ? max_nonneg(v, w) : v + w;
    }
    return over_warp<MAX>(v);
  }

  __device__ void run() {
    const AdvanceParams& A = K.a;
    const int mm = K.p.m;
    const int mg = AERO ? K.aero.m_gas : mm, nc = AERO ? K.n_gas - mg : A.state_dim - 3 - mm;  // gas, constant gas
    const double gamma = 2.0 - sqrt(2.0);
    const double cg = 1.0 / (gamma * (2.0 - gamma));
    const double cn = (1.0 - gamma) * (1.0 - gamma) / (gamma * (2.0 - gamma));
    const double kappa = (-3.0 * gamma * gamma + 4.0 * gamma - 2.0) / (12.0 * (2.0 - gamma));
    const double e0 = 1.0 / gamma, e1 = -1.0 / (gamma * (1.0 - gamma)), e2 = 1.0 / (1.0 - gamma);
    const int n_items = A.n_items_dev ? *A.n_items_dev : A.n_items;
    const bool control = warp == 0;
    const int zbase = K.p.vec * S;  // the vector section of lu

    // the slot's species: positions (mm: none) and, in the upper half, species numbers
    int sps[NPS];
#pragma unroll
    for (int k = 0; k < NPS; ++k) sps[k] = k < K.p.nps ? __ldg(K.p.species + k * P + slot) : mm;
    auto pos = [&](int k) { return sps[k] & 0xffff; };
    auto species = [&](int k) { return sps[k] >> 16; };
    auto column = [&](int k) { return 3 + (sps[k] >> 16) + (AERO && (sps[k] >> 16) >= mg ? nc : 0); };  // of the state row
    auto has = [&](int k) { return (sps[k] & 0xffff) < mm; };
    // the iterate itself is x
    double yn[NPS], fn[NPS], fg[NPS], rv[NPS], keff[NRS];
    [[maybe_unused]] double unit[NPS] = {};  // of the slot's rows (gas species: 1)
    auto to_matrix = [&](int k, double v) {
      if constexpr (AERO) v *= unit[k];
      return v;
    };
    auto from_matrix = [&](int k, double v) {
      if constexpr (AERO) v *= inverse_unit(unit[k]);
      return v;
    };
    T kt[NRS];
#pragma unroll
    for (int k = 0; k < NPS; ++k) {
      yn[k] = fn[k] = fg[k] = rv[k] = 0.0;
      if constexpr (AERO) unit[k] = 1.0;
      if (has(k)) xs()[pos(k) * S] = 0.0;
    }
#pragma unroll
    for (int k = 0; k < NRS; ++k) {
      keff[k] = 0.0;
      kt[k] = T(0);
    }
    // the resident streams and the small tables
    for (int id = 0; id < LS_COUNT; ++id)
      if (K.s.stream[id])
        for (int i = threadIdx.x; i < K.p.packet_count[id]; i += NT)
          reinterpret_cast<uint4*>(sm + K.s.stream[id])[i] = __ldg(K.p.packets[id] + i);
    for (int i = threadIdx.x; i < K.p.table_bytes / 16; i += NT)
      reinterpret_cast<uint4*>(sm + K.s.prog)[i] = __ldg(K.p.table + i);
    if (s == 0)
#pragma unroll
      for (int k = 0; k < NPS; ++k)
        if (has(k))
          reinterpret_cast<double2*>(sm + K.s.tol)[pos(k)] = make_double2(A.tol_time[2 * species(k)], A.tol_time[2 * species(k) + 1]);
    if (slot == 0) {
      xs()[mm * S] = 1.0;
      lu()[K.p.zero * S] = T(0);
      lu()[K.p.ms * S] = T(1);
      for (int k = K.p.vec + mm; k < K.p.n_entries; ++k) lu()[k * S] = T(0);  // tail rows beyond the species
    }
    if (control && sl == 0) {
      ci(I_CODE, s) = C_IDLE;
      ci(I_SMP, s) = -1;
      cd(D_COEF, s) = 0.0;
      ci(I_BAD, s) = 0;
    }
    if (threadIdx.x == 0) flag(0) = 1;  // some lane wants a sample
    const double* srcp = K.p.emis;
    int dead = 0;  // control lanes: the queue gave out
    __syncthreads();

    while (true) {
      // ---- new samples ----
      if (flag(0)) {
        bool fresh = false;
        if (control && sl == 0 && ci(I_CODE, s) == C_IDLE && !dead) {
          int smp = -1;
          while (true) {
            const int item = atomicAdd(A.queue, 1);
            if (item >= n_items) {
              dead = 1;
              break;
            }
            const int c = A.items ? A.items[item] : item;
            const tchem_gb_tadv ta = A.tadv[c];
            if (A.t_out[c] >= ta.tend) {
              A.status[c] = TCHEM_GB_SAMPLE_SKIPPED;
              if (A.stats) A.stats[c] = tchem_gb_sample_stats{};
              continue;
            }
            const int gm = A.mech_of_sample ? A.mech_of_sample[c] : 0;
            const int sm_slot = (gm >= 0 && gm < kMaxMechs) ? A.slot_of_mech[gm] : -1;
            if (sm_slot < 0) {
              A.status[c] = TCHEM_GB_SAMPLE_BAD_MECH;
              continue;
            }
            if (ta.dt < 0.0 || ta.jacobian_interval > 1 || ta.max_num_newton_iterations < 1) {
              A.status[c] = kStatusRedo;  // cases the general kernel handles
              atomicAdd(K.redo_count, 1);
              continue;
            }
            smp = c;
            cd(D_T, s) = ta.tbeg;
            cd(D_DT, s) = ta.dt;
            cd(D_TEND, s) = ta.tend;
            cd(D_DTMIN, s) = ta.dtmin;
            cd(D_DTMAX, s) = ta.dtmax;
            ci(I_MAXITER, s) = ta.num_time_iterations_per_interval;
            ci(I_MAXNEWT, s) = ta.max_num_newton_iterations;
            ci(I_ITER, s) = 0;
            ci(I_STEPS, s) = ci(I_REJ, s) = ci(I_NFAIL, s) = ci(I_NITS, s) = ci(I_NOK0, s) = ci(I_NATT, s) = 0;
            ci(I_STATUS, s) = TCHEM_GB_SAMPLE_OK;
            ci(I_SLOT, s) = sm_slot;
            ci(I_ACC, s) = 0;
            break;
          }
          ci(I_SMP, s) = smp;
          fresh = smp >= 0;
          if (fresh) ci(I_CODE, s) = C_FRESH;
        }
        __syncthreads();
        // rate constants of the new samples: all threads over (sample, reaction), through q
        bool any = false;
        for (int c = 0; c < S; ++c) {
          if (ci(I_CODE, c) != C_FRESH) continue;
          any = true;
          const int smp = ci(I_SMP, c);
          const double* row = A.state + static_cast<size_t>(smp) * A.state_dim;
          const double p = row[1], Tk = row[2], t_1 = 1.0 / Tk, conv = A.mech.conv_ppm * p * t_1;
          const double* rp = A.keff_in ? nullptr : A.rate_param[ci(I_SLOT, c)];
          double* q = reinterpret_cast<double*>(sm + K.s.q) + c;
          for (int r = threadIdx.x; r < K.p.R; r += NT) {
            double k;
            if (A.keff_in) {
              k = A.keff_in[static_cast<size_t>(smp) * K.p.R + r];
            } else {
              k = rate_constant(A.mech.rate_type[r], rp + 8 * r, A.mech.conv_exp[r], Tk, t_1, p, conv);
              for (int e = A.mech.cf_ptr[r]; e < A.mech.cf_ptr[r + 1]; ++e) k *= row[3 + mg + A.mech.cf_idx[e]];
            }
            if (A.k_scale) k *= A.k_scale[r];
            q[r * S] = k;
          }
          if constexpr (AERO) aero_setup_sample(c, smp, p, Tk);
        }
        __syncthreads();
        if (!any) {
          bool idle = true;
          for (int c = 0; c < S; ++c) idle = idle && ci(I_CODE, c) == C_IDLE;
          if (idle) break;  // every lane is idle and the queue is empty
        }
        if (ci(I_CODE, s) == C_FRESH) {
          const int smp = ci(I_SMP, s);
          const double* row = A.state + static_cast<size_t>(smp) * A.state_dim;
          int n_rounds;
          const uint4* rx = packets(LS_REACTIONS, n_rounds);
#pragma unroll
          for (int k = 0; k < NRS; ++k)
            if (k < K.p.nrs && k * P + slot < K.p.R) {
              keff[k] = qs()[rx[k * SPW].w * S];
              kt[k] = static_cast<T>(keff[k]);
            }
#pragma unroll
          for (int k = 0; k < NPS; ++k) {
            yn[k] = has(k) ? row[column(k)] : 0.0;
            if (has(k)) xs()[pos(k) * S] = yn[k];
            if constexpr (AERO) unit[k] = has(k) && species(k) >= mg ? *ext(unit_at() + species(k) - mg) : 1.0;
            fn[k] = fg[k] = rv[k] = 0.0;
          }
          if (A.keff_in) srcp = A.src_in + smp * A.src_stride;
        }
        __syncthreads();
        if (fresh) ci(I_CODE, s) = begin_step(s, C_FRESH);
        __syncthreads();
      }

      // ---- right-hand side at the iterate ----
      int code = ci(I_CODE, s);
      double coef = cd(D_COEF, s);
      if (threadIdx.x == 0) flag(0) = 0;
      if (code == C_RETRY) {
#pragma unroll
        for (int k = 0; k < NPS; ++k)
          if (has(k)) xs()[pos(k) * S] = yn[k];
      }
      if (slot == 0) qs()[K.p.Q * S] = 0.0;
      double src[NPS];
#pragma unroll
      for (int k = 0; k < NPS; ++k) src[k] = has(k) ? __ldg(srcp + species(k)) : 0.0;
      __syncthreads();
      rates(keff);
      if constexpr (AERO) {
        aero_particles();
        __syncthreads();
        aero_transfers();
      }
      const int step_pending = __syncthreads_or(code == C_STEP || code == C_DONE);
      double f[NPS];
      net(f);
#pragma unroll
      for (int k = 0; k < NPS; ++k)
        if (has(k)) f[k] += src[k];

      // ---- error test of the samples whose second stage converged ----
      if (step_pending) {
        __syncthreads();  // q is read
        const double dt = cd(D_DT, s);
#pragma unroll
        for (int k = 0; k < NPS; ++k)
          if (has(k)) {
            const double est = code == C_STEP ? 2.0 * kappa * dt * (e0 * fn[k] + e1 * fg[k] + e2 * f[k]) : 0.0;
            lu()[zbase + pos(k) * S] = static_cast<T>(to_matrix(k, est));
          }
        __syncthreads();
        solve();
        // the largest |est| / weight of the slot's species: the quotients are compared by cross products
        // (one division; as fmax does, a NaN quotient loses every comparison)
        double num = 0.0, den = 1.0;
        if (code == C_STEP) {
#pragma unroll
          for (int k = 0; k < NPS; ++k)
            if (has(k)) {
              const double est = fabs(from_matrix(k, static_cast<double>(lu()[zbase + pos(k) * S])));
              const double2 tol = reinterpret_cast<const double2*>(sm + K.s.tol)[pos(k)];
              const double wgt = tol.x + tol.y * fmax(fabs(yn[k]), fabs(xs()[pos(k) * S]));
              if (est * den > num * wgt) {
                num = est;
                den = wgt;
              }
            }
        }
        num = over_warp<true>(num > 0.0 ? num / den : 0.0);
        if (sl == 0) qs()[warp * S] = num;
        __syncthreads();
        if (control) {
          const double e = reduce<true>(0);
          if (sl == 0 && code == C_STEP) {
            ++ci(I_NATT, s);
            int next;
            const double h = cd(D_DT, s);
            if (!isfinite(e)) {
              ci(I_STATUS, s) = TCHEM_GB_SAMPLE_NONFINITE;
              ci(I_ACC, s) = 0;
              next = C_DONE;
            } else if ((e <= 1.0 || h <= cd(D_DTMIN, s)) && A.tape_dt && ci(I_STEPS, s) >= A.tape_cap) {
              ci(I_STATUS, s) = TCHEM_GB_SAMPLE_TAPE_FULL;
              ci(I_ACC, s) = 0;
              next = C_DONE;
            } else if (e <= 1.0 || h <= cd(D_DTMIN, s)) {
              const double t = ci(I_LAST, s) ? cd(D_TEND, s) : cd(D_T, s) + h;
              const double fac = step_factor(e);
              double hn = fmin(h * fac, cd(D_DTMAX, s));
              if (t + hn > cd(D_TEND, s)) hn = cd(D_TEND, s) - t;
              if (A.tape_dt) A.tape_dt[static_cast<size_t>(ci(I_SMP, s)) * A.tape_cap + ci(I_STEPS, s)] = h;
              cd(D_T, s) = t;
              cd(D_DT, s) = hn;
              ++ci(I_STEPS, s);
              ++ci(I_ITER, s);
              ci(I_ACC, s) = 1;
              next = begin_step(s, C_ACCEPT);
            } else {
              ++ci(I_REJ, s);
              ++ci(I_ITER, s);
              ci(I_ACC, s) = 0;
              cd(D_DT, s) = h * step_factor(e);  // e > 1: below 0.9
              next = begin_step(s, C_REJECT);
            }
            ci(I_CODE, s) = next;
          }
        }
        __syncthreads();
        if (A.tape_dt && code == C_STEP && ci(I_ACC, s)) {
          // checkpoint: the state at the start of the step just accepted
          const int n = ci(I_STEPS, s) - 1;
          if (n % kTapeSegment == 0) {
            double* ck = A.tape_ckpt + (static_cast<size_t>(ci(I_SMP, s)) * (A.tape_cap / kTapeSegment + 1) + n / kTapeSegment) * mm;
#pragma unroll
            for (int k = 0; k < NPS; ++k)
              if (has(k)) ck[species(k)] = yn[k];
          }
        }
        code = ci(I_CODE, s);
        coef = cd(D_COEF, s);
        if (code == C_DONE) {
          const int smp = ci(I_SMP, s), status = ci(I_STATUS, s);
          if (status == kStatusRedo) {
            if (slot == 0) {
              A.status[smp] = kStatusRedo;
              atomicAdd(K.redo_count, 1);
            }
          } else {
            const bool at_y = ci(I_ACC, s) != 0;  // else y_n: the last attempt was rejected, or no step was taken
            const double* row = A.state + static_cast<size_t>(smp) * A.state_dim;
            double* out = A.state_out + static_cast<size_t>(smp) * A.state_dim;
            for (int i = slot; i < nc; i += P) out[3 + mg + i] = row[3 + mg + i];
#pragma unroll
            for (int k = 0; k < NPS; ++k)
              if (has(k)) out[column(k)] = status != TCHEM_GB_SAMPLE_OK ? 0.0 : (at_y ? xs()[pos(k) * S] : yn[k]);
            if (slot == 0) {
              const double rho = row[0], p = row[1], Tk = row[2];
              out[0] = rho;
              out[1] = p;
              out[2] = Tk;
              A.t_out[smp] = status == TCHEM_GB_SAMPLE_OK ? cd(D_T, s) : cd(D_TEND, s);
              A.dt_out[smp] = status == TCHEM_GB_SAMPLE_OK ? cd(D_DT, s) : -1.0;
              A.status[smp] = status;
              if (A.tape_nsteps) A.tape_nsteps[smp] = ci(I_STEPS, s);
              if (A.stats) {
                tchem_gb_sample_stats st;
                st.n_steps = ci(I_STEPS, s);
                st.n_rejected = ci(I_REJ, s);
                st.n_newton_fail = ci(I_NFAIL, s);
                st.n_newton_iter = ci(I_NITS, s);
                st.n_lu = st.n_jac = ci(I_NITS, s);
                // as the algorithm counts them: f(y_0), one per iteration (and one Jacobian-vector
                // product per refinement), f(y_gamma) and f(y_{n+1})
                st.n_solve = (kRefine ? 2 : 1) * ci(I_NITS, s) + ci(I_NATT, s);
                st.n_rhs = 1 + (kRefine ? 2 : 1) * ci(I_NITS, s) + ci(I_NOK0, s) + ci(I_NATT, s);
                A.stats[smp] = st;
              }
            }
          }
        }
        if (code == C_ACCEPT) {
#pragma unroll
          for (int k = 0; k < NPS; ++k)
            if (has(k)) {
              yn[k] = xs()[pos(k) * S];
              fn[k] = f[k];
            }
        } else if (code == C_REJECT) {
#pragma unroll
          for (int k = 0; k < NPS; ++k) {
            f[k] = fn[k];
            if (has(k)) xs()[pos(k) * S] = yn[k];
          }
        }
        // outputs written before the lane is given away
        const bool rejected = AERO ? __syncthreads_or(code == C_REJECT) != 0 : (__syncthreads(), false);
        if constexpr (AERO) {
          // the transfers' terms are those of the rejected state; the matrix wants them at y_n again (the others'
          // come out as they were, and q is free)
          if (rejected) {
            aero_particles();
            __syncthreads();
            aero_transfers();
          }
        }
        if (control && sl == 0 && code == C_DONE) {
          ci(I_CODE, s) = C_IDLE;
          ci(I_SMP, s) = -1;
          cd(D_COEF, s) = 0.0;
          flag(0) = 1;
        }
      }

      // ---- where the stage starts ----
      if (code == C_STAGE) {
#pragma unroll
        for (int k = 0; k < NPS; ++k)
          if (has(k)) {
            fg[k] = f[k];
            rv[k] = cg * xs()[pos(k) * S] - cn * yn[k];
          }
      } else if (code != C_ITER) {
        if (code == C_FRESH) {
#pragma unroll
          for (int k = 0; k < NPS; ++k) fn[k] = f[k];
        }
#pragma unroll
        for (int k = 0; k < NPS; ++k)
          if (has(k)) rv[k] = yn[k] + coef * fn[k];
      }

      double g[NPS], dx[NPS];
#pragma unroll
      for (int k = 0; k < NPS; ++k) {
        g[k] = 0.0;
        if (has(k)) {
          const double y = xs()[pos(k) * S];
          g[k] = -((y - coef * f[k]) - rv[k]);
          lu()[zbase + pos(k) * S] = static_cast<T>(to_matrix(k, g[k]));
          if (kRefine) xt()[pos(k) * S] = static_cast<T>(y);
        }
      }
      bad = 0;
      {
        // zero the pattern behind the pivots and the one entry (the matrix stream writes every pivot)
        T* z = reinterpret_cast<T*>(sm + K.s.lu) + (K.p.ms + 1) * S;
        const int n = (K.p.zero - K.p.ms - 1) * S;
        if constexpr (S * sizeof(T) >= 16) {
          for (int i = threadIdx.x; i < n * static_cast<int>(sizeof(T)) / 16; i += NT)
            reinterpret_cast<uint4*>(z)[i] = make_uint4(0u, 0u, 0u, 0u);
        } else {
          for (int i = threadIdx.x; i < n; i += NT) z[i] = T(0);
        }
      }
      __syncthreads();
      factor_slots(kt);
      if constexpr (AERO) aero_slots();
      if (slot == 0) ds()[K.p.D * S] = T(0);
      __syncthreads();
      matrix(static_cast<T>(coef));
      if constexpr (kRefine) {
        // g waits in v, which matrix() no longer needs as chunk space, for the refinement
        __syncthreads();
#pragma unroll
        for (int k = 0; k < NPS; ++k)
          if (has(k)) vs()[pos(k) * S] = g[k];
      }
      __syncthreads();
      factorize();
      if (bad) ci(I_BAD, s) = 1;
      solve();
#pragma unroll
      for (int k = 0; k < NPS; ++k) dx[k] = has(k) ? from_matrix(k, static_cast<double>(lu()[zbase + pos(k) * S])) : 0.0;
      if constexpr (kRefine) {
        // FP64 residual of (I - c J) dx = g, correction through the FP32 factors
#pragma unroll
        for (int k = 0; k < NPS; ++k)
          if (has(k)) {
            g[k] = vs()[pos(k) * S];
            vs()[pos(k) * S] = dx[k];
          }
        if (slot == 0) qs()[K.p.Q * S] = 0.0;
        __syncthreads();
        rate_derivatives(keff);
        __syncthreads();
        double jd[NPS];
        net(jd);
#pragma unroll
        for (int k = 0; k < NPS; ++k)
          if (has(k)) lu()[zbase + pos(k) * S] = static_cast<T>(g[k] - (dx[k] - coef * jd[k]));
        __syncthreads();
        solve();
#pragma unroll
        for (int k = 0; k < NPS; ++k)
          if (has(k)) dx[k] += static_cast<double>(lu()[zbase + pos(k) * S]);
      }
      double sdx = 0.0, sy = 0.0;
#pragma unroll
      for (int k = 0; k < NPS; ++k)
        if (has(k)) {
          const double y = xs()[pos(k) * S] + dx[k];
          xs()[pos(k) * S] = y;
          sdx += dx[k] * dx[k];
          sy += y * y;
        }
      sdx = over_warp<false>(sdx);
      sy = over_warp<false>(sy);
      if (sl == 0) {
        qs()[warp * S] = sdx;
        qs()[(W + warp) * S] = sy;
      }
      __syncthreads();
      if (warp == 1) {  // ||y|| beside the control warp's ||dx||
        const double v = sqrt(reduce<false>(W));
        if (sl == 0) qs()[2 * W * S] = v;
        asm volatile("bar.arrive 1, 64;" ::: "memory");
      }
      if (control) {
        const double ndx = sqrt(reduce<false>(0));
        asm volatile("bar.sync 1, 64;" ::: "memory");
        const double ny = qs()[2 * W * S];
        if (sl == 0 && ci(I_SMP, s) >= 0) {
          int next = C_ITER;
          ++ci(I_NITS, s);
          const int it = ++ci(I_NEWT, s);
          const bool finite = isfinite(ndx) && isfinite(ny);
          if (ci(I_BAD, s)) {
            ci(I_BAD, s) = 0;
            ci(I_STATUS, s) = kStatusRedo;
            next = C_DONE;
          } else if (finite && ndx <= A.tol_newton[0] + A.tol_newton[1] * ny) {
            if (ci(I_STAGE, s) == 0) {
              ci(I_STAGE, s) = 1;
              ci(I_NEWT, s) = 0;
              ++ci(I_NOK0, s);
              next = C_STAGE;
            } else {
              next = C_STEP;
            }
          } else if (!finite || it >= ci(I_MAXNEWT, s)) {
            ++ci(I_NFAIL, s);
            cd(D_DT, s) *= 0.5;
            if (++ci(I_TRY, s) < 4) {
              next = begin_try(s, C_RETRY);
            } else {
              ci(I_STATUS, s) = TCHEM_GB_SAMPLE_NEWTON_FAIL;
              next = C_DONE;
            }
          }
          ci(I_CODE, s) = next;
        } else if (sl == 0) {
          ci(I_BAD, s) = 0;
        }
      }
      __syncthreads();
    }
  }
};

}  // namespace lanes
}  // namespace tchem_gb

namespace tchem_gb {
namespace lanes {

template <typename T, int S, int W, int CTAS, bool AERO>
__global__ void __launch_bounds__(32 * W, CTAS) trbdf2_lanes_kernel(const __grid_constant__ LaneParams K) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int SPW = 32 / S;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  Kernel<T, S, W, AERO> k{K, smem, lane % S, lane / S, warp * SPW + lane / S, warp, 0};
  k.run();
}

}  // namespace lanes
}  // namespace tchem_gb

#define TCHEM_GB_LANE_SHAPE(NAME, T, S, W, C, A)                                                       \
  namespace tchem_gb {                                                                              \
  const void* lane_kernel_##NAME() {                                                                \
    return reinterpret_cast<const void*>(&lanes::trbdf2_lanes_kernel<T, S, W, C, A>);                       \
  }                                                                                                 \
  cudaError_t launch_lanes_##NAME(const LaneParams& P, int grid, cudaStream_t stream) {              \
    lanes::trbdf2_lanes_kernel<T, S, W, C, A><<<grid, 32 * W, P.s.bytes, stream>>>(P);                      \
    return cudaGetLastError();                                                                      \
  }                                                                                                 \
  }
