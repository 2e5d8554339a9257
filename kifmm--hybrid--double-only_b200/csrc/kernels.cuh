// Device kernels of the KIFMM evaluator (sm_100a).  Included by plan.cu only.
//
// Data layout in HBM (all node-major, node = index into the BFS node array):
//   src4[i]      leaf-ordered sources (x, y, z, w), plain form double4
//   src4f[i]     mixed form: (x, y, z) - leaf centre, w      float4
//   trg4[i]      leaf-ordered targets (x, y, z, 0)            double4
//   ctr[n]       node centre and radius (cx, cy, cz, r)       double4
//   uden/dchk/dden[n*P + k]   upward equivalent density, downward check
//                potential, downward equivalent density      double
//   spec/effv[fb][n][32]      source / target spectra, frequency-blocked
//                (see spec_index)             double2 or float2 (mixed)
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

namespace kfmm {

constexpr double kOOFP = 1.0 / (4.0 * 3.14159265358979323846);

__device__ __forceinline__ unsigned smem_addr(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}

// The far field's kernels (transforms, Hadamard, level products) are launched as
// programmatic dependents of the kernel before them on the stream: a kernel lets
// its successor's blocks start as soon as all of its own have (chain_release), and
// waits, before it touches anything that an earlier kernel writes or reads, until
// that kernel is done (chain_wait).  What lies before the wait reads only what the
// plan's creation wrote.  Every block of every such kernel waits, so the order
// holds from end to end; launched in the ordinary way both are without effect.
// Device time of a solve, ordinary launches -> these: 20,011 points on a deep tree
// (32 such launches) 221 -> 162 us, 4,096 points 95 -> 78, 65,536 333 -> 309.  The
// pair kernels are launched in the ordinary way: their waiting blocks took the slots
// of what ran before them (65,536 points 358 -> 417 us when that was tried).
__device__ __forceinline__ void chain_release() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// ---------------------------------------------------------------------------
// P2P engine.  A job evaluates one set of targets against a list of source
// sets ("entries").  Targets: real points of a leaf (kind 0) or the UC (1) /
// DC (2) check surface of a node.  Entries: `count` sources, kind 0 = source
// points from leaf-order position `base` on (of leaf `node`; plain plans merge
// adjacent leaves' ranges), 1 = node's UE surface carrying uden, 2 = the node's
// DE surface carrying dden (base 0).  Output: out[job.out + i] = (or +=)
// 1/(4 pi) sum_j w_j / |t_i - s_j|, pairs with r == 0 skipped
// (fmm/omp.cc:259-283).
// ---------------------------------------------------------------------------
struct __align__(16) P2PEntry {
  int base, count, kind, node;
};

struct P2PJob {
  int tnode, tkind, tbeg, tcnt;
  int ebeg, eend, out, mode;  // mode 0 write, 1 add
  int ns;    // sources of all entries
  int plan;  // batched solves: whose arrays
  int copies;  // team jobs of at most 16 or 8 targets: 2 or 4 copies of them in a warp
};

struct P2PParams {
  const P2PJob* jobs;
  const P2PEntry* entries;
  const double4* src4;
  const double4* trg4;
  const double4* ctr;
  const double* uden;
  const double* dden;
  const double* sp_ue;  // 3 per point
  const double* sp_uc;
  const double* sp_de;
  const double* sp_dc;
  double* out;
  // near field: target i of a job goes to out[out_perm[J.out + i]], the original
  // order (no scatter pass afterwards); null: out[J.out + i]
  const int* out_perm;
  int P, Q;
};

// The mixed form's kernels take these besides (a separate struct: the plain
// form's kernel keeps its argument block, and ptxas its register allocation).
struct P2PMixedParams {
  P2PParams p;
  // leaf-order sources as FP32 offsets from their leaf's centre with the
  // density in FP32 (made once per upload); node centres in FP32
  const float4* src4f;
  const float4* ctrf;
  const float* spf_ue;  // the unit UE / DE surfaces in FP32, 3 per point
  const float* spf_de;
  // the entries as (kind << 28) | node for the row jobs' cursor, which reads the
  // leaf ranges itself (one 16-byte entry load instead costs registers there:
  // S2M of 4M points, NP 6, 0.397 -> 0.415 ms)
  const int* entry_ids;
  const int* src_beg;
  const int* src_num;
};
template <bool kMixed>
using P2PArgs = typename std::conditional<kMixed, P2PMixedParams, P2PParams>::type;
__device__ __forceinline__ const P2PParams& base_of(const P2PParams& a) { return a; }
__device__ __forceinline__ const P2PParams& base_of(const P2PMixedParams& a) { return a.p; }

__device__ __forceinline__ double3 surface_point(const double4 c, const double* sp, int k) {
  // centre + radius * unit-surface point, unfused as fmm/trans.cc:92-100
  double3 r;
  r.x = __dadd_rn(c.x, __dmul_rn(c.w, sp[3 * k]));
  r.y = __dadd_rn(c.y, __dmul_rn(c.w, sp[3 * k + 1]));
  r.z = __dadd_rn(c.z, __dmul_rn(c.w, sp[3 * k + 2]));
  return r;
}

// Mixed precision P2P (kMixed below): coordinates are taken relative to the
// target set's own node centre and rounded to FP32, so the FP32 differences
// keep ~1e-7 of the box size; 1/r comes from the FP32 reciprocal square root;
// terms are summed in FP32 over blocks of 32 sources and the block sums in
// FP64; the result is scaled by 1/(4 pi) in FP64.  Leaf sources are stored as
// FP32 offsets from their own leaf's centre (src4f); the offset between the
// leaf's and the target node's centres is exact in FP32 (centres are
// -1 + (2i + 1) 2^-d: the difference of two is a multiple of 2^-20 below 2 in
// magnitude for the depths <= 20 that plans accept), so a source costs one
// FP32 rounding more than a direct conversion, and half the bytes.

// ---------------------------------------------------------------------------
// Warp-autonomous P2P.  One warp owns one job of up to 32*kMaxSlots targets
// (slot k of lane l is target l + 32k) and walks the job's source sets on its
// own, without block barriers.  Sources are fetched 32 at a time, one per lane
// (coalesced), prepared in the lane, and written to the warp's own shared
// buffer; after __syncwarp every lane reads each source back as a broadcast.
// The next 32 sources are fetched into registers while the current ones are
// used.  Each source then meets the lane's `slots` targets: independent
// dependency chains per source.  r = 0 can only occur between a leaf's own
// sources and targets (equal coordinates always fall in the same leaf), so
// only the self entry carries the r > 0 test (fmm/omp.cc:280).
//
// The kernel is persistent: a grid of (SMs x resident blocks) warps takes jobs
// from an atomic counter; the host orders the jobs by decreasing cost, so the
// largest start first and the tail is short.
// ---------------------------------------------------------------------------
constexpr int kWarpJobsPerBlock = 4;
constexpr int kMaxSlots = 6;  // targets per lane: jobs hold up to 192 targets
#ifndef KFMM_P2P_MIXED_MINB
#define KFMM_P2P_MIXED_MINB 6  // resident blocks per SM asked of the mixed P2P kernel
#endif

// 1 / sqrt(r2) in FP64 for the pair sums.  The seed is the approximate reciprocal
// square root (PTX rsqrt.approx.ftz.f64, one MUFU operation), followed by one
// third-order Householder step for y^-2 = r2 (A. S. Householder, The Numerical
// Treatment of a Single Nonlinear Equation, 1970): with e = 1 - r2 y^2,
// y (1 + e/2 + 3 e^2 / 8) leaves 5/16 e^3.  Five FP64 operations where rsqrt()
// takes ten, and no branch, so several pairs' chains interleave; 1/(4 pi r) comes
// out within 1.24 eps as measured (tests/test_direct.py holds it to 3).  A pair is 12
// FP64 operations instead of 17: near field of 4M uniform points, NP 6, 15.6 -> 11.8
// ms.
// kGuard, for sets that can hold r = 0 (a leaf's own sources, the direct sum): pairs
// whose r2 is below the smallest normal number (r = 0, which fmm/omp.cc:280 skips;
// r < 1.5e-154), infinite or not a number give 0, by an integer test on the high word.
// It costs a tenth of the pair rate; rsqrt() in a branch for what lies below as well
// costs the direct sum another 12% (1,144 -> 1,279 us) and the 100,003-point NP 8 solve
// 6%.
// Other sets start the sum of squares from kTinyR2, so that r2 is neither zero nor
// subnormal there.
constexpr double kTinyR2 = 0x1p-1020;
template <bool kGuard>
__device__ __forceinline__ double pair_rsqrt(double r2) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(r2));
  const double e = fma(-r2, y * y, 1.0);
  y = fma(y * e, fma(e, 0.375, 0.5), y);
  if constexpr (kGuard) {
    constexpr unsigned kLo = 0x00100000u;  // high word of the smallest normal number
    const bool ok = (unsigned)__double2hiint(r2) - kLo < 0x7ff00000u - kLo;
    y = ok ? y : 0.0;
  }
  return y;
}

// `cnt` sources at every G-th place of buf.
template <int NS, bool kGuard, int G = 1>
__device__ __forceinline__ void pairs_fp64(const double (&tx)[NS], const double (&ty)[NS],
                                           const double (&tz)[NS], double (&acc)[NS],
                                           const double4* buf, int cnt) {
  constexpr int kUnroll = NS >= 4 ? 2 : NS >= 2 ? 4 : 8;  // chains in flight: 8 to 12
#pragma unroll kUnroll
  for (int k = 0; k < cnt; ++k) {
    const double4 s = buf[k * G];
#pragma unroll
    for (int t = 0; t < NS; ++t) {
      const double dx = tx[t] - s.x, dy = ty[t] - s.y, dz = tz[t] - s.z;
      const double r2 = fma(dz, dz, fma(dy, dy, kGuard ? dx * dx : fma(dx, dx, kTinyR2)));
      acc[t] = fma(s.w, pair_rsqrt<kGuard>(r2), acc[t]);
    }
  }
}

// Packed FP32 pairs (sm_100 f32x2 instructions): one instruction updates two
// targets.  t* hold two targets' coordinates; the source components arrive
// duplicated in both halves.
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  return ((unsigned long long)__float_as_uint(hi) << 32) | __float_as_uint(lo);
}
__device__ __forceinline__ float lo_of(unsigned long long v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float hi_of(unsigned long long v) {
  return __uint_as_float((unsigned)(v >> 32));
}

template <bool kGuard>
__device__ __forceinline__ unsigned long long pair_term2(unsigned long long tx,
                                                         unsigned long long ty,
                                                         unsigned long long tz, ulonglong2 sxy,
                                                         ulonglong2 szw, unsigned long long blk) {
  unsigned long long out;
  if (kGuard) {
    asm("{\n"
        " .reg .b64 dx, dy, dz, r2, inv;\n"
        " .reg .f32 a, b, ia, ib;\n"
        " .reg .pred pa, pb;\n"
        " sub.f32x2 dx, %1, %4;\n"
        " sub.f32x2 dy, %2, %5;\n"
        " sub.f32x2 dz, %3, %6;\n"
        " mul.f32x2 r2, dx, dx;\n"
        " fma.rn.f32x2 r2, dy, dy, r2;\n"
        " fma.rn.f32x2 r2, dz, dz, r2;\n"
        " mov.b64 {a, b}, r2;\n"
        " rsqrt.approx.ftz.f32 ia, a;\n"
        " rsqrt.approx.ftz.f32 ib, b;\n"
        " setp.gt.f32 pa, a, 0f00000000;\n"
        " setp.gt.f32 pb, b, 0f00000000;\n"
        " selp.f32 ia, ia, 0f00000000, pa;\n"
        " selp.f32 ib, ib, 0f00000000, pb;\n"
        " mov.b64 inv, {ia, ib};\n"
        " fma.rn.f32x2 %0, %7, inv, %8;\n"
        "}\n"
        : "=l"(out)
        : "l"(tx), "l"(ty), "l"(tz), "l"(sxy.x), "l"(sxy.y), "l"(szw.x), "l"(szw.y), "l"(blk));
  } else {
    asm("{\n"
        " .reg .b64 dx, dy, dz, r2, inv;\n"
        " .reg .f32 a, b, ia, ib;\n"
        " sub.f32x2 dx, %1, %4;\n"
        " sub.f32x2 dy, %2, %5;\n"
        " sub.f32x2 dz, %3, %6;\n"
        " mul.f32x2 r2, dx, dx;\n"
        " fma.rn.f32x2 r2, dy, dy, r2;\n"
        " fma.rn.f32x2 r2, dz, dz, r2;\n"
        " mov.b64 {a, b}, r2;\n"
        " rsqrt.approx.ftz.f32 ia, a;\n"
        " rsqrt.approx.ftz.f32 ib, b;\n"
        " mov.b64 inv, {ia, ib};\n"
        " fma.rn.f32x2 %0, %7, inv, %8;\n"
        "}\n"
        : "=l"(out)
        : "l"(tx), "l"(ty), "l"(tz), "l"(sxy.x), "l"(sxy.y), "l"(szw.x), "l"(szw.y), "l"(blk));
  }
  return out;
}

// Scalar FP32 pair, for the odd target of a lane with an odd slot count.
template <bool kGuard>
__device__ __forceinline__ float pair_term1(float tx, float ty, float tz, float sx, float sy,
                                            float sz, float w, float blk) {
  float out;
  if (kGuard) {
    asm("{\n"
        " .reg .f32 dx, dy, dz, r2, inv;\n"
        " .reg .pred pa;\n"
        " sub.f32 dx, %1, %4;\n"
        " sub.f32 dy, %2, %5;\n"
        " sub.f32 dz, %3, %6;\n"
        " mul.f32 r2, dx, dx;\n"
        " fma.rn.f32 r2, dy, dy, r2;\n"
        " fma.rn.f32 r2, dz, dz, r2;\n"
        " rsqrt.approx.ftz.f32 inv, r2;\n"
        " setp.gt.f32 pa, r2, 0f00000000;\n"
        " selp.f32 inv, inv, 0f00000000, pa;\n"
        " fma.rn.f32 %0, %7, inv, %8;\n"
        "}\n"
        : "=f"(out)
        : "f"(tx), "f"(ty), "f"(tz), "f"(sx), "f"(sy), "f"(sz), "f"(w), "f"(blk));
  } else {
    asm("{\n"
        " .reg .f32 dx, dy, dz, r2, inv;\n"
        " sub.f32 dx, %1, %4;\n"
        " sub.f32 dy, %2, %5;\n"
        " sub.f32 dz, %3, %6;\n"
        " mul.f32 r2, dx, dx;\n"
        " fma.rn.f32 r2, dy, dy, r2;\n"
        " fma.rn.f32 r2, dz, dz, r2;\n"
        " rsqrt.approx.ftz.f32 inv, r2;\n"
        " fma.rn.f32 %0, %7, inv, %8;\n"
        "}\n"
        : "=f"(out)
        : "f"(tx), "f"(ty), "f"(tz), "f"(sx), "f"(sy), "f"(sz), "f"(w), "f"(blk));
  }
  return out;
}

// NS targets per lane: NS / 2 packed pairs, plus one scalar target when NS is
// odd (the high half of the last packed register is then unused).  Terms are
// summed in FP32 over blocks of 32 sources (one chunk); the block sums are
// accumulated in FP64 (acc), which keeps the long sum close to a compensated
// FP32 sum and leaves the FP32 pipe to the pair terms.  (The FP32 -> FP64
// conversions take XU slots beside the reciprocal square roots: blocks of 16
// measured 0.11 ms slower at 4M points, with a 2% smaller rel-L2 error.)
// buf: per source {x,x},{y,y} then {z,z},{w,w} (two ulonglong2 per source).
template <int NS, bool kGuard, int G = 1>
__device__ __forceinline__ void pairs_mixed(const unsigned long long (&tx)[(NS + 1) / 2],
                                            const unsigned long long (&ty)[(NS + 1) / 2],
                                            const unsigned long long (&tz)[(NS + 1) / 2],
                                            double (&acc)[NS], const ulonglong2* buf, int cnt) {
  constexpr int NP2 = NS / 2, ODD = NS & 1, kBlock = 32;
  for (int k = 0; k < cnt; k += kBlock) {
    const int m = min(kBlock, cnt - k);
    unsigned long long blk[NP2 > 0 ? NP2 : 1];
    float blk1 = 0.f;
#pragma unroll
    for (int t = 0; t < NP2; ++t) blk[t] = 0ull;
    auto step = [&](int u) {
      const ulonglong2 a = buf[2 * G * (k + u)], b = buf[2 * G * (k + u) + 1];
#pragma unroll
      for (int t = 0; t < NP2; ++t) blk[t] = pair_term2<kGuard>(tx[t], ty[t], tz[t], a, b, blk[t]);
      if (ODD)
        blk1 = pair_term1<kGuard>(lo_of(tx[NP2]), lo_of(ty[NP2]), lo_of(tz[NP2]), lo_of(a.x),
                                  lo_of(a.y), lo_of(b.x), lo_of(b.y), blk1);
    };
    if (G == 1 && m == kBlock) {
      constexpr int kUnroll = NS > 4 ? 2 : 4;  // bounds the live pair temporaries
#pragma unroll kUnroll
      for (int u = 0; u < kBlock; ++u) step(u);
    } else if (G > 1) {
#pragma unroll 4
      for (int u = 0; u < m; ++u) step(u);
    } else {
      for (int u = 0; u < m; ++u) step(u);
    }
#pragma unroll
    for (int t = 0; t < NP2; ++t) {
      acc[2 * t] += (double)lo_of(blk[t]);
      acc[2 * t + 1] += (double)hi_of(blk[t]);
    }
    if (ODD) acc[NS - 1] += (double)blk1;
  }
}

// Target i of job J (i < J.tcnt), absolute FP64 coordinates.
__device__ __forceinline__ double3 job_target(const P2PParams& p, const P2PJob& J,
                                              const double4 org, int i) {
  if (J.tkind == 0) {
    const double4 w = p.trg4[J.tbeg + i];
    return make_double3(w.x, w.y, w.z);
  }
  return surface_point(org, J.tkind == 1 ? p.sp_uc : p.sp_dc, J.tbeg + i);
}

// Cursor over a job's entries, 32 sources at a time: entry e, sources
// [c0, c0 + 32).  It keeps the entry node's centre relative to the target
// node's centre in FP32 (dlt, exact) and the entry node's radius (a power of
// two).
struct EntryCursor {
  int e, eend, c0, kind, node, count, base;
  float3 dlt;
  float rad;
  __device__ __forceinline__ void open(const P2PMixedParams& a, const float4 orgf) {
    for (; e < eend; ++e) {
      const int ent = a.entry_ids[e];
      kind = ent >> 28;
      node = ent & 0x0fffffff;
      count = kind == 0 ? a.src_num[node] : a.p.P;
      base = kind == 0 ? a.src_beg[node] : 0;
      if (count > 0) break;
    }
    if (e < eend) {
      const float4 k = a.ctrf[node];
      dlt = make_float3(k.x - orgf.x, k.y - orgf.y, k.z - orgf.z);
      rad = k.w;
    }
  }
  __device__ __forceinline__ void advance(const P2PMixedParams& a, const float4 orgf) {
    c0 += 32;
    if (c0 >= count) {
      ++e;
      c0 = 0;
      open(a, orgf);
    }
  }
  // Source c0 + lane of the current entry relative to the entry node's
  // centre: the leaf point's stored offset, or rad * (FP32 unit-surface
  // point), which is exact.  dlt is added when the chunk is written to the
  // warp's buffer, so this load stays in flight across the pair loop.
  __device__ __forceinline__ float4 source(const P2PMixedParams& a, int lane) const {
    const int idx = c0 + lane;
    if (kind == 0) return a.src4f[base + idx];
    const float* sp = (kind == 1 ? a.spf_ue : a.spf_de) + 3 * idx;
    const double w = (kind == 1 ? a.p.uden : a.p.dden)[(size_t)node * a.p.P + idx];
    return make_float4(rad * sp[0], rad * sp[1], rad * sp[2], (float)w);
  }
};

// Mixed form of a row job (see warp-autonomous P2P above): slot k of lane l
// is target l + 32k; each chunk of 32 sources goes through the warp's shared
// buffer in the target node's FP32 frame and is read back as broadcasts.
template <int NS>
__device__ __forceinline__ void row_job_mixed(const P2PMixedParams& a, const P2PJob& J, int lane,
                                              void* wbuf) {
  const P2PParams& p = a.p;
  const double4 org = p.ctr[J.tnode];
  const float4 orgf = a.ctrf[J.tnode];
  constexpr int NP2C = (NS + 1) / 2;
  unsigned long long tx[NP2C], ty[NP2C], tz[NP2C];
  {
    float q[NS][3];
#pragma unroll
    for (int t = 0; t < NS; ++t) {
      const int i = lane + 32 * t;
      double3 v = make_double3(org.x, org.y, org.z);
      if (i < J.tcnt) v = job_target(p, J, org, i);
      q[t][0] = (float)(v.x - org.x);
      q[t][1] = (float)(v.y - org.y);
      q[t][2] = (float)(v.z - org.z);
    }
#pragma unroll
    for (int t = 0; t < NP2C; ++t) {
      const int u = 2 * t + 1 < NS ? 2 * t + 1 : 2 * t;
      tx[t] = pack2(q[2 * t][0], q[u][0]);
      ty[t] = pack2(q[2 * t][1], q[u][1]);
      tz[t] = pack2(q[2 * t][2], q[u][2]);
    }
  }
  EntryCursor c{J.ebeg, J.eend, 0, 0, 0, 0, 0, make_float3(0.f, 0.f, 0.f), 0.f};
  c.open(a, orgf);
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (c.e < c.eend && lane < min(32, c.count)) s = c.source(a, lane);
  double acc[NS];
#pragma unroll
  for (int t = 0; t < NS; ++t) acc[t] = 0.0;
  ulonglong2* buf = (ulonglong2*)wbuf;
  while (c.e < c.eend) {
    const int cnt = min(32, c.count - c.c0);
    const bool guard = c.kind == 0 && J.tkind == 0 && c.node == J.tnode;
    if (lane < cnt) {
      const float x = s.x + c.dlt.x, y = s.y + c.dlt.y, z = s.z + c.dlt.z;
      buf[2 * lane] = make_ulonglong2(pack2(x, x), pack2(y, y));
      buf[2 * lane + 1] = make_ulonglong2(pack2(z, z), pack2(s.w, s.w));
    }
    __syncwarp();
    c.advance(a, orgf);
    if (c.e < c.eend && lane < min(32, c.count - c.c0)) s = c.source(a, lane);
    if (guard) pairs_mixed<NS, true>(tx, ty, tz, acc, buf, cnt);
    else pairs_mixed<NS, false>(tx, ty, tz, acc, buf, cnt);
    __syncwarp();
  }
#pragma unroll
  for (int t = 0; t < NS; ++t) {
    const int i = lane + 32 * t;
    if (i < J.tcnt) {
      const double r = kOOFP * acc[t];
      double* o = p.out + (p.out_perm ? p.out_perm[J.out + i] : J.out + i);
      if (J.mode) *o += r;
      else *o = r;
    }
  }
}

// A warp's walk over its share [lo, hi) of a job's sources, 32 at a time.  The
// job's entries are read 32 at once, one per lane, cut to the share and staged in
// the warp's shared memory (the mixed form with each entry node's centre relative
// to the target node's, exact in FP32, and its radius), so that going from one
// entry to the next costs one shared load and no dependent global loads.
template <bool kMixed>
struct __align__(16) EntryStage {
  P2PEntry ent[32];
  float4 off[kMixed ? 32 : 1];
};

template <bool kMixed>
struct Walk {
  int e, eend, lo, hi;  // next entry to stage; the share, relative to its first source
  int i, m, c0;         // entry i of the m staged ones, its sources from c0 on
  P2PEntry q;           // entry i
  __device__ __forceinline__ bool refill(const P2PArgs<kMixed>& a, const float4 orgf, int lane,
                                         EntryStage<kMixed>* st) {
    while (e < eend && hi > 0) {
      P2PEntry t{0, 0, 0, 0};
      if (e + lane < eend) t = base_of(a).entries[e + lane];
      int end = t.count;
#pragma unroll
      for (int d = 1; d < 32; d *= 2) {
        const int v = __shfl_up_sync(0xffffffffu, end, d);
        if (lane >= d) end += v;
      }
      const int start = end - t.count, from = max(start, lo), n = min(end, hi) - from;
      const unsigned keep = __ballot_sync(0xffffffffu, n > 0);
      const int all = __shfl_sync(0xffffffffu, end, 31);
      e += 32;
      lo -= all;
      hi -= all;
      if (keep) {
        __syncwarp();
        if (n > 0) {
          const int slot = __popc(keep & ((1u << lane) - 1u));
          st->ent[slot] = P2PEntry{t.base + from - start, n, t.kind, t.node};
          if constexpr (kMixed) {
            const float4 k = a.ctrf[t.node];
            st->off[slot] = make_float4(k.x - orgf.x, k.y - orgf.y, k.z - orgf.z, k.w);
          }
        }
        __syncwarp();
        i = 0;
        m = __popc(keep);
        c0 = 0;
        q = st->ent[0];
        return true;
      }
    }
    return false;
  }
  // the next 32 sources; false at the end
  __device__ __forceinline__ bool advance(const P2PArgs<kMixed>& a, const float4 orgf, int lane,
                                          EntryStage<kMixed>* st) {
    c0 += 32;
    if (c0 < q.count) return true;
    if (++i < m) {
      c0 = 0;
      q = st->ent[i];
      return true;
    }
    return refill(a, orgf, lane, st);
  }
};

// Source c0 + lane of the walk's entry.  Plain form: absolute coordinates.
__device__ __forceinline__ double4 walk_source(const P2PParams& p, const Walk<false>& w, int lane) {
  const int idx = w.q.base + w.c0 + lane;
  if (w.q.kind == 0) return p.src4[idx];
  const double3 s = surface_point(p.ctr[w.q.node], w.q.kind == 1 ? p.sp_ue : p.sp_de, idx);
  return make_double4(s.x, s.y, s.z,
                      (w.q.kind == 1 ? p.uden : p.dden)[(size_t)w.q.node * p.P + idx]);
}
// Mixed form: relative to the entry node's centre (the leaf point's stored
// offset, or radius * FP32 unit-surface point, which is exact); the entry's
// offset is added when the chunk is written to the warp's buffer, so this load
// stays in flight across the pair loop.
__device__ __forceinline__ float4 walk_source(const P2PMixedParams& a, const Walk<true>& w,
                                              int lane, const EntryStage<true>* st) {
  const int idx = w.q.base + w.c0 + lane;
  if (w.q.kind == 0) return a.src4f[idx];
  const float* sp = (w.q.kind == 1 ? a.spf_ue : a.spf_de) + 3 * idx;
  const double v = (w.q.kind == 1 ? a.p.uden : a.p.dden)[(size_t)w.q.node * a.p.P + idx];
  const float rad = st->off[w.i].w;
  return make_float4(rad * sp[0], rad * sp[1], rad * sp[2], (float)v);
}

// The warps of a team (one CTA) share a job's sources; their sums meet in `red`
// and are added in warp order.
constexpr int kTeam = kWarpJobsPerBlock;
constexpr int kTeamRows = 4;  // targets per lane: a team's jobs hold up to 128
struct TeamSums {
  double v[kTeam][32 * kTeamRows];
};

__device__ __forceinline__ void store_sum(const P2PJob& J, double* out, const int* perm, int i,
                                          double sum) {
  double* o = out + (perm ? perm[J.out + i] : J.out + i);
  const double r = kOOFP * sum;
  if (J.mode) *o += r;
  else *o = r;
}

template <int NS, int G, bool kIsTeam>
__device__ __forceinline__ void store_job(const P2PJob& J, double* out, const int* perm,
                                          double (&acc)[NS], int lane, TeamSums* red) {
#pragma unroll
  for (int d = 32 / G; d < 32; d *= 2) acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], d);
  if constexpr (!kIsTeam) {
#pragma unroll
    for (int t = 0; t < NS; ++t) {
      const int i = lane + 32 * t;
      if (i < J.tcnt) store_sum(J, out, perm, i, acc[t]);
    }
  } else {
    const int wid = threadIdx.x >> 5;
#pragma unroll
    for (int t = 0; t < NS; ++t) red->v[wid][lane + 32 * t] = acc[t];
    __syncthreads();
    for (int i = threadIdx.x; i < J.tcnt; i += 32 * kTeam) {
      double s = red->v[0][i];
#pragma unroll
      for (int w = 1; w < kTeam; ++w) s += red->v[w][i];
      store_sum(J, out, perm, i, s);
    }
  }
}

// A warp's part of a job: slot k of lane l is target l + 32k (G = 1).  Jobs of G =
// 2 or 4 copies hold at most 32 / G targets, copy g meeting every G-th source (one
// slot; chunks are then padded with sources of zero weight).
template <bool kIsTeam, bool kMixed>
__device__ __forceinline__ Walk<kMixed> walk_of(const P2PJob& J) {
  Walk<kMixed> w{};
  w.e = J.ebeg;
  w.eend = J.eend;
  w.hi = J.ns;
  if constexpr (kIsTeam) {
    const int wid = threadIdx.x >> 5, chunks = (J.ns + 31) >> 5;
    w.lo = 32 * ((chunks * wid) / kTeam);
    w.hi = min(J.ns, 32 * ((chunks * (wid + 1)) / kTeam));
  }
  return w;
}

template <int NS, int G>
__device__ __forceinline__ void team_job_mixed(const P2PMixedParams& a, const P2PJob& J, int lane,
                                               void* wbuf, EntryStage<true>* st, TeamSums* red) {
  const P2PParams& p = a.p;
  const double4 org = p.ctr[J.tnode];
  const float4 orgf = a.ctrf[J.tnode];
  constexpr int NP2C = (NS + 1) / 2;
  unsigned long long tx[NP2C], ty[NP2C], tz[NP2C];
  {
    float q[NS][3];
#pragma unroll
    for (int t = 0; t < NS; ++t) {
      const int i = G > 1 ? lane % (32 / G) : lane + 32 * t;
      double3 v = make_double3(org.x, org.y, org.z);
      if (i < J.tcnt) v = job_target(p, J, org, i);
      q[t][0] = (float)(v.x - org.x);
      q[t][1] = (float)(v.y - org.y);
      q[t][2] = (float)(v.z - org.z);
    }
#pragma unroll
    for (int t = 0; t < NP2C; ++t) {
      const int u = 2 * t + 1 < NS ? 2 * t + 1 : 2 * t;
      tx[t] = pack2(q[2 * t][0], q[u][0]);
      ty[t] = pack2(q[2 * t][1], q[u][1]);
      tz[t] = pack2(q[2 * t][2], q[u][2]);
    }
  }
  Walk<true> w = walk_of<true, true>(J);
  bool more = w.refill(a, orgf, lane, st);
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (more && lane < w.q.count) s = walk_source(a, w, lane, st);
  double acc[NS];
#pragma unroll
  for (int t = 0; t < NS; ++t) acc[t] = 0.0;
  ulonglong2* buf = (ulonglong2*)wbuf;
  while (more) {
    int cnt = min(32, w.q.count - w.c0);
    const bool guard = w.q.kind == 0 && J.tkind == 0 && w.q.node == J.tnode;
    if (lane < cnt) {
      const float4 o = st->off[w.i];
      const float x = s.x + o.x, y = s.y + o.y, z = s.z + o.z;
      buf[2 * lane] = make_ulonglong2(pack2(x, x), pack2(y, y));
      buf[2 * lane + 1] = make_ulonglong2(pack2(z, z), pack2(s.w, s.w));
    } else if (G > 1) {
      // outside every target's box, weight zero
      buf[2 * lane] = make_ulonglong2(pack2(8.f, 8.f), pack2(8.f, 8.f));
      buf[2 * lane + 1] = make_ulonglong2(pack2(8.f, 8.f), 0ull);
    }
    __syncwarp();
    more = w.advance(a, orgf, lane, st);
    if (more && lane < w.q.count - w.c0) s = walk_source(a, w, lane, st);
    if constexpr (G > 1) {
      cnt = (cnt + G - 1) / G;
      const ulonglong2* mine = buf + 2 * (lane / (32 / G));
      if (guard) pairs_mixed<NS, true, G>(tx, ty, tz, acc, mine, cnt);
      else pairs_mixed<NS, false, G>(tx, ty, tz, acc, mine, cnt);
    } else {
      if (guard) pairs_mixed<NS, true>(tx, ty, tz, acc, buf, cnt);
      else pairs_mixed<NS, false>(tx, ty, tz, acc, buf, cnt);
    }
    __syncwarp();
  }
  store_job<NS, G, true>(J, p.out, p.out_perm, acc, lane, red);
}

// Plain FP64 form: the same walk, sources staged as double4.
template <int NS, int G, bool kIsTeam>
__device__ __forceinline__ void warp_job_fp64(const P2PParams& p, const P2PJob& J, int lane,
                                              void* wbuf, EntryStage<false>* st, TeamSums* red) {
  const double4 org = p.ctr[J.tnode];
  double tx[NS], ty[NS], tz[NS], acc[NS];
#pragma unroll
  for (int t = 0; t < NS; ++t) {
    const int i = G > 1 ? lane % (32 / G) : lane + 32 * t;
    double3 v = make_double3(org.x, org.y, org.z);
    if (i < J.tcnt) v = job_target(p, J, org, i);
    tx[t] = v.x;
    ty[t] = v.y;
    tz[t] = v.z;
    acc[t] = 0.0;
  }
  Walk<false> w = walk_of<kIsTeam, false>(J);
  const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
  bool more = w.refill(p, none, lane, st);
  double4 s = make_double4(0.0, 0.0, 0.0, 0.0);
  if (more && lane < w.q.count) s = walk_source(p, w, lane);
  double4* buf = (double4*)wbuf;
  while (more) {
    const int cnt = min(32, w.q.count - w.c0);
    const bool guard = w.q.kind == 0 && J.tkind == 0 && w.q.node == J.tnode;
    if (lane < cnt) buf[lane] = s;
    else if (G > 1) buf[lane] = make_double4(0.0, 0.0, 0.0, 0.0);
    __syncwarp();
    more = w.advance(p, none, lane, st);
    if (more && lane < w.q.count - w.c0) s = walk_source(p, w, lane);
    const double4* mine = G > 1 ? buf + lane / (32 / G) : buf;
    if (guard) pairs_fp64<NS, true, G>(tx, ty, tz, acc, mine, (cnt + G - 1) / G);
    else pairs_fp64<NS, false, G>(tx, ty, tz, acc, mine, (cnt + G - 1) / G);
    __syncwarp();
  }
  store_job<NS, G, kIsTeam>(J, p.out, p.out_perm, acc, lane, red);
}

// Shared memory of one P2P warp: its chunk of 32 sources and its staged entries.
template <bool kMixed>
struct __align__(16) P2PWarpSmem {
  unsigned char chunk[32 * 32];
  EntryStage<kMixed> st;
};

// One warp per job: the mixed form walks with its cursor (row_job_mixed), the plain
// form as a team of one.
template <bool kMixed>
using P2PRowSmem = typename std::conditional<kMixed, unsigned char[32 * 32], P2PWarpSmem<false>>::type;

template <bool kMixed, int NS>
__device__ __forceinline__ void warp_job(const P2PArgs<kMixed>& a, const P2PJob& J, int lane,
                                         void* ws) {
  if constexpr (kMixed) {
    row_job_mixed<NS>(a, J, lane, ws);
  } else {
    P2PWarpSmem<false>* w = (P2PWarpSmem<false>*)ws;
    warp_job_fp64<NS, 1, false>(a, J, lane, w->chunk, &w->st, nullptr);
  }
}

template <bool kMixed>
__device__ __forceinline__ void run_job(const P2PArgs<kMixed>& a, const P2PJob& J, int lane,
                                        void* ws) {
  switch ((J.tcnt + 31) >> 5) {
    case 1: warp_job<kMixed, 1>(a, J, lane, ws); break;
    case 2: warp_job<kMixed, 2>(a, J, lane, ws); break;
    case 3: warp_job<kMixed, 3>(a, J, lane, ws); break;
    case 4: warp_job<kMixed, 4>(a, J, lane, ws); break;
    case 5: warp_job<kMixed, 5>(a, J, lane, ws); break;
    default: warp_job<kMixed, kMaxSlots>(a, J, lane, ws); break;
  }
}

template <bool kMixed, int NS, int G>
__device__ __forceinline__ void team_job(const P2PArgs<kMixed>& a, const P2PJob& J, int lane,
                                         P2PWarpSmem<kMixed>* ws, TeamSums* red) {
  if constexpr (kMixed) team_job_mixed<NS, G>(a, J, lane, ws->chunk, &ws->st, red);
  else warp_job_fp64<NS, G, true>(a, J, lane, ws->chunk, &ws->st, red);
}

template <bool kMixed>
__device__ __forceinline__ void run_team_job(const P2PArgs<kMixed>& a, const P2PJob& J, int lane,
                                             P2PWarpSmem<kMixed>* ws, TeamSums* red) {
  switch ((J.tcnt + 31) >> 5) {
    case 1:
      if (J.copies == 4) team_job<kMixed, 1, 4>(a, J, lane, ws, red);
      else if (J.copies == 2) team_job<kMixed, 1, 2>(a, J, lane, ws, red);
      else team_job<kMixed, 1, 1>(a, J, lane, ws, red);
      break;
    case 2: team_job<kMixed, 2, 1>(a, J, lane, ws, red); break;
    case 3: team_job<kMixed, 3, 1>(a, J, lane, ws, red); break;
    default: team_job<kMixed, kTeamRows, 1>(a, J, lane, ws, red); break;
  }
}

// Persistent: each warp takes jobs from *next_job until none are left.  The
// counter is zeroed on the stream before every launch.  kMinBlocks: resident
// blocks per SM asked of ptxas; the plan runs the mixed near field with 5
// (96 registers, no spills) when W-list surfaces carry more than 1% of its
// pairs: measured 8-11% faster on ellipsoid-surface clouds, 1-2% slower than
// 6 on uniform ones, whatever the NP.
template <bool kMixed, int kMinBlocks = kMixed ? KFMM_P2P_MIXED_MINB : 4>
__global__ void __launch_bounds__(32 * kWarpJobsPerBlock, kMinBlocks)
p2p_warp_kernel(P2PArgs<kMixed> a, int njobs, int* next_job) {
  __shared__ __align__(16) P2PRowSmem<kMixed> smem[kWarpJobsPerBlock];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (;;) {
    int j = 0;
    if (lane == 0) j = atomicAdd(next_job, 1);
    j = __shfl_sync(0xffffffffu, j, 0);
    if (j >= njobs) return;
    const P2PJob J = base_of(a).jobs[j];  // a register copy: the output stores may alias
    run_job<kMixed>(a, J, lane, &smem[wid]);
  }
}

// One job per CTA, its sources shared by the CTA's four warps; blocks start in
// job order, largest first.  A job's time is a quarter of what one warp takes, so
// near fields with few jobs per resident warp neither wait for the longest of
// them nor leave warps idle: 65,536 points NP 4 plain 0.95 -> 0.16 ms, 1M points
// NP 6 mixed 2.17 -> 1.94 ms.  Resident blocks asked of ptxas: plain 4 (119
// registers; 5 and 6 measured 2% slower at 4M points), mixed 8 (64 registers; 5 to
// 7 measured 1-5% slower at 1M and 4M).
constexpr int kTeamBlocksFp64 = 4, kTeamBlocksMixed = 8;

template <bool kMixed>
__global__ void __launch_bounds__(32 * kTeam, kMixed ? kTeamBlocksMixed : kTeamBlocksFp64)
p2p_team_kernel(P2PArgs<kMixed> a) {
  __shared__ P2PWarpSmem<kMixed> smem[kTeam];
  __shared__ TeamSums red;
  const P2PJob J = base_of(a).jobs[blockIdx.x];
  run_team_job<kMixed>(a, J, threadIdx.x & 31, &smem[threadIdx.x >> 5], &red);
}

// The near fields of many plans in one launch (batched solves): job j is of the
// plan whose arrays params[jobs[j].plan] describes.  32 solves of 4,096 to 262,144
// points, mixed: 0.91 ms.
template <bool kMixed>
__global__ void __launch_bounds__(32 * kTeam, kMixed ? kTeamBlocksMixed : kTeamBlocksFp64)
p2p_team_batch_kernel(const P2PArgs<kMixed>* params, const P2PJob* jobs) {
  __shared__ P2PWarpSmem<kMixed> smem[kTeam];
  __shared__ TeamSums red;
  const P2PJob J = jobs[blockIdx.x];
  run_team_job<kMixed>(params[J.plan], J, threadIdx.x & 31, &smem[threadIdx.x >> 5], &red);
}

// The same with one warp per job (mixed plans with jobs enough).
__global__ void __launch_bounds__(32 * kWarpJobsPerBlock, KFMM_P2P_MIXED_MINB)
p2p_fused_kernel(const P2PMixedParams* params, const P2PJob* jobs, int njobs, int* next_job) {
  __shared__ __align__(16) unsigned char smem[kWarpJobsPerBlock][32 * 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (;;) {
    int j = 0;
    if (lane == 0) j = atomicAdd(next_job, 1);
    j = __shfl_sync(0xffffffffu, j, 0);
    if (j >= njobs) return;
    const P2PJob J = jobs[j];
    run_job<true>(params[J.plan], J, lane, smem[wid]);
  }
}

// ---------------------------------------------------------------------------
// Level GEMM on FP64 tensor cores (mma.sync m8n8k4 DMMA):
//   C[:, j] = alpha_j * A * B[:, j]   (+ C[:, j] when accumulate)
// A: M x K column-major (lda = M).  Column j of B starts at B + boff[j]
// (K contiguous values), column j of C at C + coff[j] (M values).
// ---------------------------------------------------------------------------
struct GemmArgs {
  const double* A;
  int M, K;
  const double* B;
  const int* boff;
  double* C;
  const int* coff;
  const double* alpha;  // per column, or NULL -> alpha_const
  double alpha_const;
  int ncol;
  int accumulate;
};

__device__ __forceinline__ void dmma_884(double& d0, double& d1, double a, double b) {
  asm volatile(
      "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
      : "+d"(d0), "+d"(d1)
      : "d"(a), "d"(b));
}

// A block computes rows [m0, m0 + mrows) of C (mrows <= 160, a multiple of 8)
// for kGemmBN columns.  8 warps = 4 (rows) x 2 (columns); each warp owns 5 x 4
// m8n8 tiles, i.e. 20 DMMA per 4-deep k step for 9 shared loads.  16-deep
// slices of A and B stream into a 3-stage shared-memory ring by asynchronous
// 16-byte copies (cp.async, zero-filled outside the matrices), so no
// registers hold data in flight and two blocks fit on an SM.  Requires M, K
// and every column offset even (16-byte aligned pairs of doubles); the host
// checks this when it builds a batch.
constexpr int kGemmRows = 160, kGemmBN = 64, kGemmBK = 16, kGemmThreads = 256;
constexpr int kGemmStages = 3;
constexpr int kGemmAStride = kGemmRows + 8;  // doubles; 8 and 4 (mod 16): every bank pair
constexpr int kGemmBStride = kGemmBK + 4;    // hit exactly twice by a warp's fragment reads
constexpr int kGemmStageDoubles = kGemmBK * kGemmAStride + kGemmBN * kGemmBStride;
constexpr size_t kGemmSmemBytes = sizeof(double) * kGemmStages * kGemmStageDoubles;

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_addr(smem)),
               "l"(gmem), "r"(valid ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// kAcc: the launch accumulates onto C (its epilogue reads C; see there).
template <bool kAcc>
__global__ void __launch_bounds__(kGemmThreads, 2) gemm_fp64_dmma_kernel(GemmArgs g, int mrows) {
  extern __shared__ __align__(16) double gsm[];
  __shared__ int boff_s[kGemmBN];
  __shared__ int coff_s[kAcc ? kGemmBN : 1];
  __shared__ double alpha_s[kAcc ? kGemmBN : 1];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp >> 1, wn = warp & 1;
  const int m0 = blockIdx.x * mrows, n0 = blockIdx.y * kGemmBN;
  chain_release();
  const int mend = min(g.M, m0 + mrows);
  const int nslices = (g.K + kGemmBK - 1) / kGemmBK;
  if (tid < kGemmBN) {
    const bool in = n0 + tid < g.ncol;
    boff_s[tid] = in ? g.boff[n0 + tid] : -1;
    if constexpr (kAcc) {
      coff_s[tid] = in ? g.coff[n0 + tid] : 0;
      alpha_s[tid] = in ? (g.alpha ? g.alpha[n0 + tid] : g.alpha_const) : 0.0;
    }
  }
  double acc[5][4][2];
#pragma unroll
  for (int i = 0; i < 5; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  __syncthreads();
  chain_wait();
  auto issue = [&](int s) {
    double* As = gsm + (s % kGemmStages) * kGemmStageDoubles;
    double* Bs = As + kGemmBK * kGemmAStride;
    const int k0 = s * kGemmBK;
#pragma unroll
    for (int r = 0; r < kGemmRows * kGemmBK / 2 / kGemmThreads; ++r) {
      const int q = tid + r * kGemmThreads;
      const int k = q / (kGemmRows / 2), m = 2 * (q % (kGemmRows / 2));
      const int gm = m0 + m, gk = k0 + k;
      const bool ok = gm < mend && gk < g.K;
      cp_async16(As + k * kGemmAStride + m, ok ? g.A + (size_t)gk * g.M + gm : g.A, ok);
    }
#pragma unroll
    for (int r = 0; r < kGemmBN * kGemmBK / 2 / kGemmThreads; ++r) {
      const int q = tid + r * kGemmThreads;
      const int n = q / (kGemmBK / 2), k = 2 * (q % (kGemmBK / 2));
      const int gk = k0 + k, bo = boff_s[n];
      const bool ok = bo >= 0 && gk < g.K;
      cp_async16(Bs + n * kGemmBStride + k, ok ? g.B + (size_t)bo + gk : g.B, ok);
    }
  };
#pragma unroll
  for (int s = 0; s < kGemmStages - 1; ++s) {
    if (s < nslices) issue(s);
    cp_async_commit();
  }
  for (int s = 0; s < nslices; ++s) {
    cp_async_wait<kGemmStages - 2>();
    __syncthreads();
    if (s + kGemmStages - 1 < nslices) issue(s + kGemmStages - 1);
    cp_async_commit();
    const double* As = gsm + (s % kGemmStages) * kGemmStageDoubles;
    const double* Bs = As + kGemmBK * kGemmAStride;
#pragma unroll
    for (int kk = 0; kk < kGemmBK; kk += 4) {
      double af[5], bf[4];
#pragma unroll
      for (int mi = 0; mi < 5; ++mi)
        af[mi] = As[(kk + (lane & 3)) * kGemmAStride + wm * 40 + mi * 8 + (lane >> 2)];
#pragma unroll
      for (int ni = 0; ni < 4; ++ni)
        bf[ni] = Bs[(wn * 32 + ni * 8 + (lane >> 2)) * kGemmBStride + kk + (lane & 3)];
#pragma unroll
      for (int mi = 0; mi < 5; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) dmma_884(acc[mi][ni][0], acc[mi][ni][1], af[mi], bf[ni]);
    }
  }
  cp_async_wait<0>();
  if constexpr (!kAcc) {
#pragma unroll
    for (int mi = 0; mi < 5; ++mi)
#pragma unroll
      for (int ni = 0; ni < 4; ++ni)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int m = m0 + wm * 40 + mi * 8 + (lane >> 2);
          const int n = n0 + wn * 32 + ni * 8 + (lane & 3) * 2 + h;
          if (m < mend && n < g.ncol) {
            const double a = g.alpha ? g.alpha[n] : g.alpha_const;
            g.C[(size_t)g.coff[n] + m] = a * acc[mi][ni][h];
          }
        }
  } else {
    // Accumulating epilogue, one row of tiles (8 outputs a thread) at a time:
    // the outputs to accumulate onto are all read before any is written
    // (distinct columns never share memory), so the eight loads overlap instead
    // of each waiting behind the previous store (the accumulating down-pass
    // products at 4M points, NP=6: 0.28 -> 0.25 ms).
#pragma unroll
    for (int mi = 0; mi < 5; ++mi) {
      const int m = m0 + wm * 40 + mi * 8 + (lane >> 2);
      double old[4][2];
#pragma unroll
      for (int ni = 0; ni < 4; ++ni)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int nl = wn * 32 + ni * 8 + (lane & 3) * 2 + h;
          old[ni][h] = m < mend && n0 + nl < g.ncol ? g.C[(size_t)coff_s[nl] + m] : 0.0;
        }
#pragma unroll
      for (int ni = 0; ni < 4; ++ni)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int nl = wn * 32 + ni * 8 + (lane & 3) * 2 + h, n = n0 + nl;
          if (m < mend && n < g.ncol) {
            const double v = alpha_s[nl] * acc[mi][ni][h];
            g.C[(size_t)coff_s[nl] + m] = old[ni][h] + v;
          }
        }
    }
  }
}

// The same product in small tiles, operands straight from global memory (L2)
// into the fragments: a CTA computes 32 rows x 16 wn columns, its 8 warps being wn
// column groups times wk = 8 / wn shares of K, whose sums meet in shared memory.
// No pipeline to fill, no split-K pass: what bounds a level product of a few
// hundred columns is the latency of its start and of the passes after it; with
// more columns it is the L1's rate, so the fragments are read 16 bytes a lane: a
// load of A holds rows 2r and 2r + 1 of one k (rows of two m8 tiles), a load of B
// holds k 2c and 2c + 1 of one column (two k steps, of the even and the odd k).
// Up and down products of a solve, split-K and a reduction pass -> 8-byte loads, 40
// x 16 -> this: 20,011 points on a deep tree 346 -> 140 -> 94 us, 65,536 points NP 4
// plain 141 -> 73 -> 52, 4M on the ellipsoid surface NP 4 678 -> 439 -> 303.
constexpr int kSmallRows = 32, kSmallCols = 16, kSmallWarps = 8;
constexpr int kSmallStride = kSmallRows + 2;

__global__ void __launch_bounds__(32 * kSmallWarps, 2) gemm_fp64_small_kernel(GemmArgs g, int wn) {
  __shared__ double red[kSmallWarps][kSmallCols * kSmallStride];  // [warp][col][row]
  __shared__ int coff_s[kSmallCols * kSmallWarps];  // the epilogue's, read before the wait
  __shared__ double alpha_s[kSmallCols * kSmallWarps];
  chain_release();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wk = kSmallWarps / wn, cg = warp % wn, ks = warp / wn;
  const int m0 = blockIdx.x * kSmallRows, n0 = blockIdx.y * (kSmallCols * wn);
  const int r = lane >> 2, c = lane & 3;
  // this warp's K range, a multiple of 8 but for the end
  const int eights = (g.K + 7) / 8;
  const int k0 = 8 * (eights * ks / wk), k1 = min(g.K, 8 * (eights * (ks + 1) / wk));
  const double* ap[2];
#pragma unroll
  for (int i = 0; i < 2; ++i)  // rows beyond the matrix repeat its last two (not stored)
    ap[i] = g.A + (size_t)(k0 + 2 * c) * g.M + min(g.M - 2, m0 + 16 * i + 2 * r);
  const double* bp[2];
#pragma unroll
  for (int j = 0; j < 2; ++j)
    bp[j] = g.B + g.boff[min(g.ncol - 1, n0 + cg * kSmallCols + 8 * j + r)] + k0 + 2 * c;
  for (int q = threadIdx.x; q < wn * kSmallCols; q += 32 * kSmallWarps) {
    const bool in = n0 + q < g.ncol;
    coff_s[q] = in ? g.coff[n0 + q] : 0;
    alpha_s[q] = in && g.alpha ? g.alpha[n0 + q] : g.alpha_const;
  }
  double acc[4][2][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  chain_wait();
  constexpr int U = 2;  // eights of K in flight
  for (int k = k0; k < k1; k += 8 * U) {
    double2 af[U][2][2], bf[U][2];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool in = k + 8 * u + 2 * c < k1;  // K is even
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i)
          af[u][j][i] = in ? __ldg((const double2*)(ap[i] + (size_t)(8 * u + j) * g.M))
                           : make_double2(0.0, 0.0);
#pragma unroll
      for (int j = 0; j < 2; ++j)
        bf[u][j] = in ? *(const double2*)(bp[j] + 8 * u) : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) ap[i] += (size_t)(8 * U) * g.M;
#pragma unroll
    for (int j = 0; j < 2; ++j) bp[j] += 8 * U;
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int o = 0; o < 2; ++o)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 2; ++j)
            dmma_884(acc[i][j][0], acc[i][j][1], i & 1 ? af[u][o][i >> 1].y : af[u][o][i >> 1].x,
                     o ? bf[u][j].y : bf[u][j].x);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        red[warp][(8 * j + 2 * c + h) * kSmallStride + 16 * (i >> 1) + 2 * r + (i & 1)] =
            acc[i][j][h];
  __syncthreads();
  // outputs: 32 consecutive rows of a column by a warp, two columns at a time (the
  // outputs to accumulate onto are read before either is written)
  const int m = m0 + lane;
  if (m >= g.M) return;
  for (int q0 = warp; q0 < wn * kSmallCols; q0 += 2 * kSmallWarps) {
    double* o[2];
    double old[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int q = q0 + h * kSmallWarps;  // 16 wn columns: both exist
      o[h] = n0 + q < g.ncol ? g.C + (size_t)coff_s[q] + m : nullptr;
      old[h] = o[h] && g.accumulate ? *o[h] : 0.0;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (!o[h]) continue;
      const int q = q0 + h * kSmallWarps, e = (q % kSmallCols) * kSmallStride + lane;
      double s = red[q / kSmallCols][e];
      for (int z = 1; z < wk; ++z) s += red[q / kSmallCols + z * wn][e];
      s *= alpha_s[q];
      *o[h] = g.accumulate ? old[h] + s : s;
    }
  }
}

// ---------------------------------------------------------------------------
// V list.  Grids: the (2np)^3 regular grid, x fastest; surface sample (i,j,k)
// sits at (x,y,z) = (i,j,k) + np/2 (fmm/trans.cc:336-358, 395-418).
// Spectrum index (kz * n + ky) * (np + 1) + kx (r2c halves x).
// Both transforms are pruned to the np^3 block that holds the surface.
// ---------------------------------------------------------------------------
// Spectra are stored frequency-blocked: spec[(fb * nn + node) * kFB + f % kFB]
// with fb = f / kFB, so one block of frequencies for every box (nn * 256 B)
// is contiguous and stays resident in L2 while the Hadamard kernel works on it.
constexpr int kFB = 32;
__host__ __device__ __forceinline__ size_t spec_index(int f, int node, int nn) {
  return ((size_t)(f / kFB) * nn + node) * kFB + (f % kFB);
}

struct FFTParams {
  int np, P, F, nn;
  int nboxes;           // entries of nodes
  const int* nodes;     // nodes to transform
  const int* depth;
  const int* surf_idx;  // np^3 -> surface index or -1, index (i*np + j)*np + k
  const int* surf_ijk;  // P x 3
  const double* cs;     // cos(2 pi m / n), m < n
  const double* sn;     // sin(2 pi m / n)
  const double* pln;    // uden (forward) or dchk target (inverse) base
  double* plnout;
  const void* specin;   // double2 (FP64 plans) or float2 (mixed plans)
  void* specout;
  // the forward transform also zeroes the downward check potentials (nn * P, even)
  // and the solve's error flag
  double* zero;
  int* error;
};

constexpr int kFFTThreads = 128;
constexpr int kMaxNP = 8;

// Multiplication by (-i)^e.
__device__ __forceinline__ double2 rot_mi(double2 v, int e) {
  switch (e & 3) {
    case 0: return v;
    case 1: return make_double2(v.y, -v.x);
    case 2: return make_double2(-v.x, -v.y);
    default: return make_double2(-v.y, v.x);
  }
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) {
  return make_double2(a.x + b.x, a.y + b.y);
}

// Pruned forward DFT of length N = 2 NP whose input is non-zero at positions
// H .. H + NP - 1 only (the surface block, H = NP / 2):
//   X[q] = sum_k v[k] w^(q (k + H)),  w = exp(-2 pi i / N),  q < N.
// Decimation in the output index: with Q = NP / 2 (NP even) and q = m + jQ,
// w^(jQ (k + H)) = (-i)^(j (k + H)) depends on k mod 4 only, so four partial
// sums per m over k of one residue mod 4 give all four outputs m + jQ:
// NP * NP / 2 complex multiply-adds instead of 2 NP^2.  For odd NP the split
// is on q = m + jNP, k mod 2: NP^2.  Twiddles come from the tables cs, sn
// (cos, sin of 2 pi m / N) at compile-time indices.
template <int NP>
__device__ __forceinline__ void dft_fwd_pruned(const double2 (&v)[NP], double2 (&X)[2 * NP],
                                               const double* cs, const double* sn) {
  constexpr int N = 2 * NP, H = NP / 2;
  constexpr int R = NP % 2 == 0 ? 4 : 2, Q = N / R;
#pragma unroll
  for (int m = 0; m < Q; ++m) {
    double2 S[R];
#pragma unroll
    for (int c = 0; c < R; ++c) S[c] = make_double2(0.0, 0.0);
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      const int e = (m * (k + H)) % N;
      double2& a = S[k % R];
      a.x = fma(v[k].x, cs[e], fma(v[k].y, sn[e], a.x));
      a.y = fma(v[k].y, cs[e], fma(-v[k].x, sn[e], a.y));
    }
#pragma unroll
    for (int j = 0; j < R; ++j) {
      double2 o = make_double2(0.0, 0.0);
#pragma unroll
      for (int c = 0; c < R; ++c) o = cadd(o, rot_mi(S[c], (4 / R) * j * (c + H)));
      X[m + j * Q] = o;
    }
  }
}

// Pruned inverse DFT of length N = 2 NP evaluated at positions H .. H+NP-1:
//   y[k] = sum_q X[q] w^(-q (k + H)),  k < NP.
// With q = m + jQ as above, the inner sum over j only depends on (k + H) mod
// R: R combinations of the X[m + jQ] per m, then NP * Q multiply-adds.
template <int NP>
__device__ __forceinline__ void dft_inv_pruned(const double2 (&X)[2 * NP], double2 (&y)[NP],
                                               const double* cs, const double* sn) {
  constexpr int N = 2 * NP, H = NP / 2;
  constexpr int R = NP % 2 == 0 ? 4 : 2, Q = N / R;
#pragma unroll
  for (int k = 0; k < NP; ++k) y[k] = make_double2(0.0, 0.0);
#pragma unroll
  for (int m = 0; m < Q; ++m) {
    double2 T[R];  // T[c] = sum_j X[m + jQ] (+i)^((4/R) j c), c = (k + H) mod R
#pragma unroll
    for (int c = 0; c < R; ++c) {
      double2 o = make_double2(0.0, 0.0);
#pragma unroll
      for (int j = 0; j < R; ++j) o = cadd(o, rot_mi(X[m + j * Q], -(4 / R) * j * c));
      T[c] = o;
    }
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      const int e = (m * (k + H)) % N;
      const double2 t = T[(k + H) % R];
      y[k].x = fma(t.x, cs[e], fma(-t.y, sn[e], y[k].x));
      y[k].y = fma(t.y, cs[e], fma(t.x, sn[e], y[k].y));
    }
  }
}

// Boxes per block: as many as fit in ~44 KB of static shared memory (at most
// 3), so that every pass keeps most of the block's threads busy.
template <int NP>
__host__ __device__ constexpr int fft_boxes_per_block() {
  constexpr int N = 2 * NP, NK = NP + 1;
  constexpr int fwd = NP * NP * NP * 8 + NP * NP * NK * 16 + NP * N * NK * 16;
  constexpr int b = 44000 / fwd;
  return b < 1 ? 1 : (b > 3 ? 3 : b);
}

// Pruned 3-D transforms, compiled per NP so every loop over the np^3 surface
// block unrolls and every twiddle index is a constant (the twiddle loads are
// then warp-wide broadcasts).  A block transforms fft_boxes_per_block<NP>()
// boxes.  Each pass gives one thread one line of one box's grid: the x pass a
// (z, y) row, the y pass a (z, kx) column, the z pass a (ky, kx) column, and
// each thread produces all outputs of its line from the <= np non-zero
// inputs.
// Five resident blocks per SM (shared memory allows five at NP = 6): with
// the next group's values held in registers the unbounded kernel takes 168
// registers and three blocks, measured slower on small and surface clouds.
template <int NP, class C>
__global__ void __launch_bounds__(kFFTThreads, 5) fft_src_np_kernel(FFTParams p) {
  constexpr int N = 2 * NP, H = NP / 2, NK = NP + 1, B = fft_boxes_per_block<NP>();
  __shared__ double den[B][NP * NP * NP];
  __shared__ double2 X[B][NP * NP * NK];
  __shared__ double2 Y[B][NP * N * NK];
  __shared__ double cs[N], sn[N];
  constexpr int P = NP * NP * NP - (NP - 2) * (NP - 2) * (NP - 2);
  constexpr int R = (B * P + kFFTThreads - 1) / kFFTThreads;  // surface values per thread
  __shared__ int node_s[B];
  __shared__ double scale_s[B];
  __shared__ int cell_s[P];  // surface point -> cell of the np^3 block
  const int tid = threadIdx.x;
  const int ngroups = (p.nboxes + B - 1) / B;
  if (tid < N) {
    cs[tid] = p.cs[tid];
    sn[tid] = p.sn[tid];
  }
  chain_release();
  for (int q = tid; q < P; q += kFFTThreads)
    cell_s[q] = (p.surf_ijk[3 * q] * NP + p.surf_ijk[3 * q + 1]) * NP + p.surf_ijk[3 * q + 2];
  // Persistent: the block takes groups of B boxes in turn.  The P surface
  // values of the next group (consecutive threads, consecutive values) and
  // its nodes' scales are loaded into registers while this group is
  // transformed, so the passes do not wait for global memory.
  chain_wait();
  {
    const size_t n2 = (size_t)p.nn * P / 2;
    double2* z = (double2*)p.zero;
    for (size_t q = (size_t)blockIdx.x * kFFTThreads + tid; q < n2; q += (size_t)gridDim.x * kFFTThreads)
      z[q] = make_double2(0.0, 0.0);
    if (blockIdx.x == 0 && tid == 0) *p.error = 0;
  }
  double pre[R];
  int nx_node = -1;
  double nx_scale = 0.0;
  auto fetch = [&](int grp) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int q = tid + r * kFFTThreads, bb = q / P, s = q % P, b = grp * B + bb;
      pre[r] = 0.0;
      if (q < B * P && grp < ngroups && b < p.nboxes) pre[r] = p.pln[(size_t)p.nodes[b] * p.P + s];
    }
    if (tid < B) {
      const int b = grp * B + tid;
      nx_node = grp < ngroups && b < p.nboxes ? p.nodes[b] : -1;
      nx_scale = nx_node >= 0 ? ldexp(1.0, p.depth[nx_node]) : 0.0;
    }
  };
  fetch(blockIdx.x);
  for (int grp = blockIdx.x; grp < ngroups; grp += gridDim.x) {
    __syncthreads();  // the previous group's passes are done with the shared arrays
    if (tid < B) {
      node_s[tid] = nx_node;
      scale_s[tid] = nx_scale;
    }
    for (int q = tid; q < B * NP * NP * NP; q += kFFTThreads) (&den[0][0])[q] = 0.0;
    __syncthreads();
    // the group's surface values into the boxes' np^3 blocks
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int q = tid + r * kFFTThreads, bb = q / P, s = q % P;
      if (q < B * P && node_s[bb] >= 0) den[bb][cell_s[s]] = pre[r] * scale_s[bb];
    }
    fetch(grp + gridDim.x);
    __syncthreads();
    // x: row (k = z, j = y), outputs kx
    for (int q = tid; q < B * NP * NP; q += kFFTThreads) {
      const int bb = q / (NP * NP), t = q % (NP * NP);
      const int k = t / NP, j = t % NP;
      double v[NP];
#pragma unroll
      for (int i = 0; i < NP; ++i) v[i] = den[bb][(i * NP + j) * NP + k];
#pragma unroll
      for (int kx = 0; kx < NK; ++kx) {
        double ar = 0, ai = 0;
#pragma unroll
        for (int i = 0; i < NP; ++i) {
          const int m = (kx * (i + H)) % N;
          ar = fma(v[i], cs[m], ar);
          ai = fma(-v[i], sn[m], ai);
        }
        X[bb][(k * NP + j) * NK + kx] = make_double2(ar, ai);
      }
    }
    __syncthreads();
    // y: column (k, kx), outputs ky
    for (int q = tid; q < B * NP * NK; q += kFFTThreads) {
      const int bb = q / (NP * NK), t = q % (NP * NK);
      const int k = t / NK, kx = t % NK;
      double2 v[NP], o[N];
#pragma unroll
      for (int j = 0; j < NP; ++j) v[j] = X[bb][(k * NP + j) * NK + kx];
      dft_fwd_pruned<NP>(v, o, cs, sn);
#pragma unroll
      for (int ky = 0; ky < N; ++ky) Y[bb][(k * N + ky) * NK + kx] = o[ky];
    }
    __syncthreads();
    // z: column (ky, kx), outputs kz -> spectrum
    C* out = (C*)p.specout;
    for (int q = tid; q < B * N * NK; q += kFFTThreads) {
      const int bb = q / (N * NK), t = q % (N * NK);
      const int node = node_s[bb];
      if (node < 0) continue;
      const int ky = t / NK, kx = t % NK;
      double2 v[NP], o[N];
#pragma unroll
      for (int k = 0; k < NP; ++k) v[k] = Y[bb][(k * N + ky) * NK + kx];
      dft_fwd_pruned<NP>(v, o, cs, sn);
#pragma unroll
      for (int kz = 0; kz < N; ++kz) {
        C e;
        e.x = o[kz].x;
        e.y = o[kz].y;
        out[spec_index((kz * N + ky) * NK + kx, node, p.nn)] = e;
      }
    }
  }
}

// spectrum -> c2r -> gather at the DC surface, scaled by 1/(2np)^3
// (omp.cc:482-533, trans.cc:383-418).  Writes plnout[node*P + s].
template <int NP, class C>
__global__ void __launch_bounds__(kFFTThreads) ifft_trg_np_kernel(FFTParams p) {
  constexpr int N = 2 * NP, H = NP / 2, NK = NP + 1, B = fft_boxes_per_block<NP>();
  __shared__ double2 Z[B][NP * N * NK];
  __shared__ double2 W[B][NP * NP * NK];
  __shared__ double cs[N], sn[N];
  __shared__ int node_s[B];
  const int tid = threadIdx.x;
  const int b0 = blockIdx.x * B;
  if (tid < N) {
    cs[tid] = p.cs[tid];
    sn[tid] = p.sn[tid];
  }
  if (tid < B) node_s[tid] = b0 + tid < p.nboxes ? p.nodes[b0 + tid] : -1;
  chain_release();
  __syncthreads();
  chain_wait();
  // z inverse: column (ky, kx), outputs z in the surface block; every
  // spectrum entry is read exactly once, straight from global memory
  // (consecutive threads, consecutive entries)
  const C* in = (const C*)p.specin;
  for (int q = tid; q < B * N * NK; q += kFFTThreads) {
    const int bb = q / (N * NK), t = q % (N * NK);
    const int node = node_s[bb];
    if (node < 0) continue;
    const int ky = t / NK, kx = t % NK;
    double2 v[N], acc[NP];
#pragma unroll
    for (int kz = 0; kz < N; ++kz) {
      const C e = in[spec_index((kz * N + ky) * NK + kx, node, p.nn)];
      v[kz] = make_double2(e.x, e.y);
    }
    dft_inv_pruned<NP>(v, acc, cs, sn);
#pragma unroll
    for (int k = 0; k < NP; ++k) Z[bb][(k * N + ky) * NK + kx] = acc[k];
  }
  __syncthreads();
  // y inverse: column (k, kx), outputs y in the surface block
  for (int q = tid; q < B * NP * NK; q += kFFTThreads) {
    const int bb = q / (NP * NK), t = q % (NP * NK);
    if (node_s[bb] < 0) continue;
    const int k = t / NK, kx = t % NK;
    double2 v[N], acc[NP];
#pragma unroll
    for (int ky = 0; ky < N; ++ky) v[ky] = Z[bb][(k * N + ky) * NK + kx];
    dft_inv_pruned<NP>(v, acc, cs, sn);
#pragma unroll
    for (int j = 0; j < NP; ++j) W[bb][(k * NP + j) * NK + kx] = acc[j];
  }
  __syncthreads();
  // x: Hermitian half -> real, at the surface points only
  constexpr double inv_g = 1.0 / (double)(N * N * N);
  constexpr int P = NP * NP * NP - (NP - 2) * (NP - 2) * (NP - 2);
  for (int q = tid; q < B * P; q += kFFTThreads) {
    const int bb = q / P, s = q % P;
    const int node = node_s[bb];
    if (node < 0) continue;
    const int i = p.surf_ijk[3 * s], j = p.surf_ijk[3 * s + 1], k = p.surf_ijk[3 * s + 2];
    const double2* w = &W[bb][(k * NP + j) * NK];
    const int x = i + H;
    double acc = w[0].x + ((x & 1) ? -w[NP].x : w[NP].x);
    int m = 0;
#pragma unroll
    for (int kx = 1; kx < NP; ++kx) {
      m += x;
      if (m >= N) m -= N;
      acc += 2.0 * (w[kx].x * cs[m] - w[kx].y * sn[m]);
    }
    p.plnout[(size_t)node * p.P + s] = acc * inv_g;
  }
}

// M2L Hadamard accumulation over sibling groups.  A group is the 8 children
// of one parent; their V lists all lie in the 6x6x6 window of same-depth
// positions 2*parent + [-2,3]^3 (fmm/input.cc:311-339), each member taking
// the window entries at Chebyshev distance >= 2 from itself.  Window entry w
// = (wx + 6 wy + 36 wz); member c = 4 cx + 2 cy + cz; offset delta = w - 2 -
// (cx,cy,cz) selects translation spectrum (dx+3) + 7 (dy+3) + 49 (dz+3)
// (fmm/omp_sse_block.cc:581-593).
// Spectra in blocks of kFB = 32 frequencies, lane = frequency.  A window's rows in
// x meet, for each of the 4 (cy, cz) member pairs, one row of 7 translation
// spectra.  Pairs of sibling groups whose parents are x-neighbours (parent x even
// and x + 1) share one 8 x 6 x 6 window, so each translation value serves both.
// One launch takes the windows of both kinds (blocks [0, pairs.chunks) the pairs').
struct HadSet {
  int nwin = 0, win_per_block = 1, chunks = 0;
  int split = 1;  // warps that share a window (then one window per team of warps)
  const int* win = nullptr;      // nwin x (4 + 2H) x 6 x 6 node ids, x fastest (-1 = absent)
  const int* members = nullptr;  // nwin x 8H node ids (-1 = no V list)
  // per window: bit wy + 6 wz set if the row has an entry
  const unsigned long long* rows = nullptr;
};

// Groups whose windows are mostly empty (clouds on surfaces): their present
// entries one by one.  Entry (node, k): the source spectrum of `node` meets
// translation spectrum k - 49 cz - 7 cy - cx for member (cx, cy, cz), so an entry
// costs 8 translation loads and 8 multiply-adds whatever its place, where a row of
// a dense window costs 28 loads and 48 a group.
struct HadSparse {
  int n = 0, per_block = 1, chunks = 0;
  const int* ptr = nullptr;      // n + 1
  const int2* ent = nullptr;
  const int* members = nullptr;  // n x 8
};
__device__ __forceinline__ constexpr int had_member_offset(int c) {
  return 49 * (c & 1) + 7 * ((c >> 1) & 1) + (c >> 2);
}

// The rows of a window that warp `part` of `split` takes.
__device__ __forceinline__ unsigned long long had_rows_of(int part, int split) {
  if (split == 1) return ~0ull;
  unsigned long long m = 0ull;
  for (int r = part; r < 36; r += split) m |= 1ull << r;
  return m;
}

// A row of the translation table at (dy, dz) with |dy| <= 1 and |dz| <= 1:
// its entries dx = -1, 0, 1 (k = 2, 3, 4 of the row) are adjacent offsets,
// whose spectra are zero (they are not V-list interactions), so the FP64
// kernel skips those loads and multiply-adds: 27 of the 216 per member.
// (The FP32 kernels below are FMA-bound with their loads scheduled across the
// rows; there a branch per row costs more than the skipped work.)
__device__ __forceinline__ bool near_row(int dy, int dz) {
  return dy >= -1 && dy <= 1 && dz >= -1 && dz <= 1;
}

// ---------------------------------------------------------------------------
// Mixed-form Hadamard, one CTA per SM.  The translation spectra of one block of
// 32 frequencies ([fb][343][32] complex FP32, 87,808 B) are brought into
// shared memory by bulk asynchronous copies (TMA, cp.async.bulk) that
// complete on an mbarrier.  A complex multiply-add is two packed FP32 FMAs on
// the translation value as loaded and the source value duplicated:
//   A += {tr, ti} * {sr, sr},  B += {tr, ti} * {si, si},
//   re = A.x - B.y,  im = A.y + B.x
// so a lane reads 8 B of shared memory per 12/7 multiply-adds and spends no
// instruction on rearranging it.  The products of each half of the window
// (z-planes 0-2 and 3-5, 108 per member of which up to 27 are zero) are
// summed in FP32 and the two half sums added in FP64.
// Warps are autonomous: each loads its own group's window into its slice of
// shared memory.
constexpr int kHad32Threads = 512;
constexpr int kHad32Warps = kHad32Threads / 32;
constexpr unsigned kHad32TileBytes = 343u * kFB * 8u;  // 87,808
constexpr int kHadCopies = 7;                           // 49 offsets each
constexpr long long kMbarSpinLimit = 1ll << 24;          // bounded waits

struct Had32Params {
  int nn, ngroups, groups_per_block;
  const int* win;
  const int* members;
  const unsigned long long* rows;  // per window: bit wy + 6 wz set if the row has an entry
  const float2* tile;  // [fb][343][32] translation spectra
  const float2* spec;
  float2* effv;
  int* error;  // set to 1 when the tile copy does not complete
  long long wait_limit;  // tries of the tile-copy wait (kMbarSpinLimit by default)
};

__device__ __forceinline__ bool mbar_try_wait(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ bool mbar_wait_bounded(unsigned bar, unsigned parity,
                                                  long long limit = kMbarSpinLimit) {
  for (long long i = 0; i < limit; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

// Bulk-copies kBytes of a translation tile from src into dst in 7 copies of 49
// offsets (one thread issues, all wait on the mbarrier with a bounded spin of `limit`
// tries).  Returns false in every thread of the block, after setting *error,
// if the copy did not complete; thread 0 then waits (with the full default
// bound) for the copy still in flight to land before the block exits.
template <unsigned kBytes>
__device__ __forceinline__ bool had_load_tile(const void* tile, unsigned char* dst,
                                              unsigned long long* bar, int* error,
                                              long long limit) {
  chain_release();
  const unsigned b = smem_addr(bar);
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(b) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(b),
                 "r"(kBytes)
                 : "memory");
    const unsigned char* src = (const unsigned char*)tile;
    constexpr unsigned chunk = kBytes / kHadCopies;
#pragma unroll 1
    for (int c = 0; c < kHadCopies; ++c)
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, "
          "[%3];\n" ::"r"(smem_addr(dst + c * chunk)),
          "l"(src + (size_t)c * chunk), "r"(chunk), "r"(b)
          : "memory");
  }
  chain_wait();  // the tile's copy runs meanwhile
  const bool ready = mbar_wait_bounded(b, 0, limit);
  if (!__syncthreads_and(ready)) {
    if (threadIdx.x == 0) {
      atomicExch(error, 1);
      mbar_wait_bounded(b, 0);  // let copies still in flight land before exiting
    }
    return false;
  }
  return true;
}

// Plain FP64 form, one CTA per SM: the frequency block's 343 translation spectra
// (175,616 B) are brought into shared memory by bulk asynchronous copies, a warp
// takes one window of H sibling groups (H = 2: an x-pair), all 8 H members'
// sums in registers.  Bound by the FP64 pipe and the latency of its operations: a
// row of H = 2 is 384 multiply-adds a lane (192 cycles of the SM's pipe) against
// 112 shared-memory wavefronts of translation values and 32 of sources; with one
// group a window the wavefronts outweighed the multiply-adds.  4M uniform points,
// NP 6: 3.98 ms one group a window through L1, 2.96 ms with 8 warps (pipe 42%
// busy, fixed-latency waits the first stall), 2.63 ms with 12 (168 registers).
// Where there are fewer windows than warps on the device, `split` warps share a
// window, each taking every split-th of its rows; their sums meet in shared
// memory (over the tile, once every warp is done with it) and are added in order.
constexpr int kHad64Threads = 384;
constexpr int kHad64Warps = kHad64Threads / 32;
constexpr unsigned kHad64TileBytes = 343u * kFB * 16u;  // 175,616

struct Had64Params {
  int nn;
  HadSet pairs, singles;
  HadSparse sparse;
  const double2* tile;  // [fb][343][32], zero for |delta|_inf <= 1 and f >= F
  const double2* spec;
  double2* effv;
  int* error;            // set to 1 when the tile copy does not complete
  long long wait_limit;  // tries of the tile-copy wait (kMbarSpinLimit by default)
};

template <int H>
__device__ __forceinline__ void had64_windows(const Had64Params& p, const HadSet& q, int chunk,
                                              int (*win)[288], int (*mem)[16],
                                              unsigned char* had32_dyn) {
  constexpr int WX = 4 + 2 * H, C = 8 * H;
  const double2* tsm = (const double2*)had32_dyn;
  const int f = threadIdx.x & 31, slot = threadIdx.x >> 5;
  const int teams = kHad64Warps / q.split, part = slot % q.split;
  const int g0 = chunk * q.win_per_block;
  const int g1 = min(q.nwin, g0 + q.win_per_block);
  const size_t fbase = (size_t)blockIdx.y * p.nn;
  const double2* spec = p.spec + fbase * kFB + f;
  const unsigned long long mine = had_rows_of(part, q.split);
  double ar[C], ai[C];
  for (int g = g0 + slot / q.split; g < g1; g += teams) {
    for (int k = f; k < 36 * WX; k += 32) win[slot][k] = q.win[(size_t)g * (36 * WX) + k];
    if (f < C) mem[slot][f] = q.members[(size_t)g * C + f];
    __syncwarp();
    const int* w = win[slot];
    unsigned long long rows = q.rows[g] & mine;
#pragma unroll
    for (int c = 0; c < C; ++c) ar[c] = ai[c] = 0.0;
    double2 nxt[WX];
    auto fetch = [&](int r) {
#pragma unroll
      for (int x = 0; x < WX; ++x) {
        const int sid = w[r * WX + x];
        nxt[x] = sid >= 0 ? spec[(size_t)sid * kFB] : make_double2(0.0, 0.0);
      }
    };
    int row = rows ? __ffsll((long long)rows) - 1 : 36;
    if (row < 36) fetch(row);
    while (row < 36) {
      rows &= rows - 1;
      const int next = rows ? __ffsll((long long)rows) - 1 : 36;
      double2 srow[WX];
#pragma unroll
      for (int x = 0; x < WX; ++x) srow[x] = nxt[x];
      if (next < 36) fetch(next);
      const int wy = row % 6, wz = row / 6;
#pragma unroll
      for (int cyz = 0; cyz < 4; ++cyz) {
        const int cy = cyz >> 1, cz = cyz & 1;
        const double2* trow = tsm + ((wz + 1 - cz) * 49 + (wy + 1 - cy) * 7) * kFB + f;
        auto row_body = [&](auto near) {
          constexpr bool kNear = decltype(near)::value;
#pragma unroll
          for (int k = 0; k < 7; ++k) {
            if (kNear && k >= 2 && k <= 4) continue;
            const double2 t = trow[k * kFB];
            // the products with t.x of all members first, then those with t.y: the
            // two a sum receives are then 2 H x 2 operations apart, not adjacent
#pragma unroll
            for (int part = 0; part < 2; ++part)
#pragma unroll
              for (int h = 0; h < H; ++h)
#pragma unroll
                for (int cx = 0; cx < 2; ++cx) {
                  const int wx = k - 1 + cx;
                  if (wx < 0 || wx > 5) continue;
                  const int c = h * 8 + cx * 4 + cy * 2 + cz;
                  const double2 v = srow[wx + 2 * h];
                  ar[c] = part == 0 ? fma(t.x, v.x, ar[c]) : fma(-t.y, v.y, ar[c]);
                  ai[c] = part == 0 ? fma(t.x, v.y, ai[c]) : fma(t.y, v.x, ai[c]);
                }
          }
        };
        if (near_row(wy - 2 - cy, wz - 2 - cz)) row_body(std::true_type{});
        else row_body(std::false_type{});
      }
      row = next;
    }
    if (q.split == 1) {
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const int m = mem[slot][c];
        if (m >= 0) p.effv[(fbase + m) * kFB + f] = make_double2(ar[c], ai[c]);
      }
    }
    __syncwarp();
  }
  if (q.split > 1) {  // one window per team
    __syncthreads();
    double2* sums = (double2*)had32_dyn;
    const bool have = g0 + slot / q.split < g1;
    if (have)
#pragma unroll
      for (int c = 0; c < C; ++c) sums[(slot * C + c) * 32 + f] = make_double2(ar[c], ai[c]);
    __syncthreads();
    if (!have) return;
    for (int c = part; c < C; c += q.split) {
      const int m = mem[slot][c];
      if (m < 0) continue;
      double2 s = sums[((slot - part) * C + c) * 32 + f];
      for (int k = 1; k < q.split; ++k) {
        const double2 v = sums[((slot - part + k) * C + c) * 32 + f];
        s.x += v.x;
        s.y += v.y;
      }
      p.effv[(fbase + m) * kFB + f] = s;
    }
  }
}

// Sparse groups, one per warp at a time: entries read 32 at once, one per lane, and
// handed round; the next entries' spectra are loaded while the current ones are
// multiplied.
__device__ __forceinline__ void had64_sparse(const Had64Params& p, int chunk,
                                             const double2* tsm) {
  const HadSparse& q = p.sparse;
  const int f = threadIdx.x & 31, slot = threadIdx.x >> 5;
  const size_t fbase = (size_t)blockIdx.y * p.nn;
  const double2* spec = p.spec + fbase * kFB + f;
  const int g1 = min(q.n, (chunk + 1) * q.per_block);
  for (int g = chunk * q.per_block + slot; g < g1; g += kHad64Warps) {
    const int end = q.ptr[g + 1];
    double ar[8], ai[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) ar[c] = ai[c] = 0.0;
    for (int e0 = q.ptr[g]; e0 < end; e0 += 32) {
      const int n = min(32, end - e0);
      const int2 mine = f < n ? q.ent[e0 + f] : make_int2(0, 0);
      constexpr int U = 4;
      double2 nxt[U];
      auto fetch = [&](int i) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int node = __shfl_sync(0xffffffffu, mine.x, i + u);
          nxt[u] = i + u < n ? spec[(size_t)node * kFB] : make_double2(0.0, 0.0);
        }
      };
      fetch(0);
      for (int i = 0; i < n; i += U) {
        double2 v[U];
        const double2* t[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          v[u] = nxt[u];
          const int k = __shfl_sync(0xffffffffu, mine.y, i + u);
          t[u] = tsm + (i + u < n ? k : had_member_offset(7)) * kFB + f;
        }
        if (i + U < n) fetch(i + U);
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const double2 w = t[u][-had_member_offset(c) * kFB];
            ar[c] = fma(-w.y, v[u].y, fma(w.x, v[u].x, ar[c]));
            ai[c] = fma(w.y, v[u].x, fma(w.x, v[u].y, ai[c]));
          }
      }
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int m = q.members[(size_t)g * 8 + c];
      if (m >= 0) p.effv[(fbase + m) * kFB + f] = make_double2(ar[c], ai[c]);
    }
  }
}

__global__ void __launch_bounds__(kHad64Threads, 1) hadamard_fp64_kernel(Had64Params p) {
  extern __shared__ __align__(128) unsigned char had32_dyn[];
  __shared__ int win[kHad64Warps][288];
  __shared__ int mem[kHad64Warps][16];
  __shared__ __align__(8) unsigned long long bar;
  if (!had_load_tile<kHad64TileBytes>(p.tile + (size_t)blockIdx.y * 343 * kFB, had32_dyn, &bar,
                                      p.error, p.wait_limit))
    return;
  const int chunk = blockIdx.x;
  const int single = chunk - p.pairs.chunks, sparse = single - p.singles.chunks;
  if (single < 0) had64_windows<2>(p, p.pairs, chunk, win, mem, had32_dyn);
  else if (sparse < 0) had64_windows<1>(p, p.singles, single, win, mem, had32_dyn);
  else had64_sparse(p, sparse, (const double2*)had32_dyn);
}

__global__ void __launch_bounds__(kHad32Threads, 1) hadamard_fp32_kernel(Had32Params p) {
  extern __shared__ __align__(128) unsigned char had32_dyn[];
  __shared__ int win[kHad32Warps][216];
  __shared__ int mem[kHad32Warps][8];
  __shared__ __align__(8) unsigned long long bar;
  const unsigned long long* tsm = (const unsigned long long*)had32_dyn;
  const int fb = blockIdx.y;
  const int f = threadIdx.x & 31, slot = threadIdx.x >> 5;
  const int g0 = blockIdx.x * p.groups_per_block;
  const int g1 = min(p.ngroups, g0 + p.groups_per_block);
  const size_t fbase = (size_t)fb * p.nn;
  if (!had_load_tile<kHad32TileBytes>(p.tile + (size_t)fb * 343 * kFB, had32_dyn, &bar, p.error,
                                      p.wait_limit))
    return;
  for (int g = g0 + slot; g < g1; g += kHad32Warps) {
    for (int q = f; q < 216; q += 32) win[slot][q] = p.win[(size_t)g * 216 + q];
    if (f < 8) mem[slot][f] = p.members[(size_t)g * 8 + f];
    __syncwarp();
    const int* w = win[slot];
    const unsigned long long* spec = (const unsigned long long*)p.spec + fbase * kFB + f;
    unsigned long long rows = p.rows[g];  // rows with no entry are not visited
    unsigned long long A[8], B[8];
    double ar[8], ai[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      A[c] = B[c] = 0ull;
      ar[c] = ai[c] = 0.0;
    }
    auto fold = [&]() {  // the half window's FP32 sums into FP64
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        ar[c] += (double)lo_of(A[c]) - (double)hi_of(B[c]);
        ai[c] += (double)hi_of(A[c]) + (double)lo_of(B[c]);
        A[c] = B[c] = 0ull;
      }
    };
    int row = rows ? __ffsll((long long)rows) - 1 : 36;
    unsigned long long nxt[6];
    if (row < 36) {
#pragma unroll
      for (int wx = 0; wx < 6; ++wx) {
        const int sid = w[row * 6 + wx];
        nxt[wx] = sid >= 0 ? spec[(size_t)sid * kFB] : 0ull;
      }
    }
    bool folded = false;
    while (row < 36) {
      rows &= rows - 1;
      const int next = rows ? __ffsll((long long)rows) - 1 : 36;
      unsigned long long sr[6], si[6];  // {sr, sr}, {si, si}
#pragma unroll
      for (int wx = 0; wx < 6; ++wx) {
        sr[wx] = pack2(lo_of(nxt[wx]), lo_of(nxt[wx]));
        si[wx] = pack2(hi_of(nxt[wx]), hi_of(nxt[wx]));
      }
      if (next < 36) {
#pragma unroll
        for (int wx = 0; wx < 6; ++wx) {
          const int sid = w[next * 6 + wx];
          nxt[wx] = sid >= 0 ? spec[(size_t)sid * kFB] : 0ull;
        }
      }
      const int wy = row % 6, wz = row / 6;
      if (!folded && wz >= 3) {  // end of z-planes 0-2 of the window
        fold();
        folded = true;
      }
#pragma unroll
      for (int cyz = 0; cyz < 4; ++cyz) {
        const int cy = cyz >> 1, cz = cyz & 1;
        const unsigned long long* trow =
            tsm + ((wz - 2 - cz + 3) * 49 + (wy - 2 - cy + 3) * 7) * kFB + f;
        unsigned long long t[7];
#pragma unroll
        for (int k = 0; k < 7; ++k) t[k] = trow[k * kFB];
#pragma unroll
        for (int wx = 0; wx < 6; ++wx)
#pragma unroll
          for (int cx = 0; cx < 2; ++cx) {
            const int c = cx * 4 + cy * 2 + cz;
            const unsigned long long tk = t[wx - cx + 1];
            asm("fma.rn.f32x2 %0, %2, %3, %0;\n"
                "fma.rn.f32x2 %1, %2, %4, %1;\n"
                : "+l"(A[c]), "+l"(B[c])
                : "l"(tk), "l"(sr[wx]), "l"(si[wx]));
          }
      }
      row = next;
    }
    fold();
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int m = mem[slot][c];
      if (m >= 0) p.effv[(fbase + m) * kFB + f] = make_float2((float)ar[c], (float)ai[c]);
    }
    __syncwarp();
  }
}

// Pairs of sibling groups whose parents are x-neighbours (parent x even and
// x + 1) share one 8 x 6 x 6 window: a row of 8 source spectra meets each
// row of 7 translation values for both groups, 24 multiply-adds per 7 shared
// loads, which halves the shared-memory traffic per multiply-add.  The 16
// members' FP32 sums of the first half-window are kept in FP64 in the warp's
// slice of shared memory and added to the second half's at the end.  12 warps
// per CTA (up to 168 registers a thread).
//
// Rows whose 8 entries are all absent (windows at the domain's faces, and
// the many empty boxes around clouds on surfaces) are not visited: the plan
// gives each window a mask of its rows that hold an entry (4M points on the
// ellipsoid surface: 1.19 -> 0.65 ms; uniform cube: -2%).  The four centre
// rows, where every member pair meets the zero translation values of the
// adjacent offsets, run as separate runs of a body that skips them (1.527
// -> 1.510 ms at 4M, NP=6); elsewhere they are multiplied like the others:
// row bodies specialised on which member pairs meet an adjacent row (ten
// variants, dispatched per row) were measured 14% slower on the uniform cube.
constexpr int kHadPairThreads = 384;
constexpr int kHadPairWarps = kHadPairThreads / 32;
constexpr size_t kHadPairSumBytes = sizeof(double) * kHadPairWarps * 16 * 2 * 32;
constexpr size_t kHadPairSmemBytes = kHad32TileBytes + kHadPairSumBytes;

struct HadPairParams {
  int nn, npairs, pairs_per_block;
  const int* win;      // npairs x 288: x8 + 8 * (wy + 6 * wz), -1 = absent
  const int* members;  // npairs x 16: group 0 members, then group 1
  const unsigned long long* rows;  // npairs: bit wy + 6 wz set if the row has an entry
  const float2* tile;
  const float2* spec;
  float2* effv;
  int* error;
  long long wait_limit;
};

// One window row for the 4 (cy, cz) member pairs.  trow0 points at the
// translation row of offset (dy, dz) = (wy - 2, wz - 2) for lane f; member
// pair (cy, cz) uses the row cz * 49 + cy * 7 spectra lower.
__device__ __forceinline__ void had_pair_row(unsigned long long (&A)[16],
                                             unsigned long long (&B)[16],
                                             const unsigned long long (&sr)[8],
                                             const unsigned long long (&si)[8],
                                             const unsigned long long* trow0) {
#pragma unroll
  for (int cyz = 0; cyz < 4; ++cyz) {
    const int cy = cyz >> 1, cz = cyz & 1;
    const unsigned long long* trow = trow0 - (cz * 49 + cy * 7) * kFB;
    unsigned long long t[7];
#pragma unroll
    for (int k = 0; k < 7; ++k) t[k] = trow[k * kFB];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int wx = 0; wx < 6; ++wx)
#pragma unroll
        for (int cx = 0; cx < 2; ++cx) {
          const int k = wx - cx + 1;
          const int c = h * 8 + cx * 4 + cy * 2 + cz;
          asm("fma.rn.f32x2 %0, %2, %3, %0;\n"
              "fma.rn.f32x2 %1, %2, %4, %1;\n"
              : "+l"(A[c]), "+l"(B[c])
              : "l"(t[k]), "l"(sr[wx + 2 * h]), "l"(si[wx + 2 * h]));
        }
  }
}

// A centre row of the window (wy and wz in {2, 3}): every member pair (cy, cz)
// meets it at |dy|, |dz| <= 1, so its translation values k = 2..4 (dx = -1,
// 0, 1: adjacent offsets, zero spectra) are neither loaded nor multiplied.
__device__ __forceinline__ void had_pair_row_centre(unsigned long long (&A)[16],
                                                    unsigned long long (&B)[16],
                                                    const unsigned long long (&sr)[8],
                                                    const unsigned long long (&si)[8],
                                                    const unsigned long long* trow0) {
#pragma unroll
  for (int cyz = 0; cyz < 4; ++cyz) {
    const int cy = cyz >> 1, cz = cyz & 1;
    const unsigned long long* trow = trow0 - (cz * 49 + cy * 7) * kFB;
    unsigned long long t[7];
#pragma unroll
    for (int k = 0; k < 7; ++k)
      if (k < 2 || k > 4) t[k] = trow[k * kFB];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int wx = 0; wx < 6; ++wx)
#pragma unroll
        for (int cx = 0; cx < 2; ++cx) {
          const int k = wx - cx + 1;
          if (k >= 2 && k <= 4) continue;
          const int c = h * 8 + cx * 4 + cy * 2 + cz;
          asm("fma.rn.f32x2 %0, %2, %3, %0;\n"
              "fma.rn.f32x2 %1, %2, %4, %1;\n"
              : "+l"(A[c]), "+l"(B[c])
              : "l"(t[k]), "l"(sr[wx + 2 * h]), "l"(si[wx + 2 * h]));
        }
  }
}

__global__ void __launch_bounds__(kHadPairThreads, 1) hadamard_fp32_pair_kernel(HadPairParams p) {
  extern __shared__ __align__(128) unsigned char had32_dyn[];
  __shared__ int win[kHadPairWarps][288];
  __shared__ int mem[kHadPairWarps][16];
  __shared__ __align__(8) unsigned long long bar;
  const unsigned long long* tsm = (const unsigned long long*)had32_dyn;
  const int fb = blockIdx.y;
  const int f = threadIdx.x & 31, slot = threadIdx.x >> 5;
  double* sums = (double*)(had32_dyn + kHad32TileBytes) + (size_t)slot * 16 * 2 * 32 + f;
  const int g0 = blockIdx.x * p.pairs_per_block;
  const int g1 = min(p.npairs, g0 + p.pairs_per_block);
  const size_t fbase = (size_t)fb * p.nn;
  const unsigned long long* spec = (const unsigned long long*)p.spec + fbase * kFB + f;
  if (!had_load_tile<kHad32TileBytes>(p.tile + (size_t)fb * 343 * kFB, had32_dyn, &bar, p.error,
                                      p.wait_limit))
    return;
  for (int g = g0 + slot; g < g1; g += kHadPairWarps) {
    for (int q = f; q < 288; q += 32) win[slot][q] = p.win[(size_t)g * 288 + q];
    if (f < 16) mem[slot][f] = p.members[(size_t)g * 16 + f];
    __syncwarp();
    const int* w = win[slot];
    unsigned long long rows = p.rows[g];
    unsigned long long A[16], B[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) A[c] = B[c] = 0ull;
    // the first half-window's sums go to shared memory (FP64) once its rows
    // are done
    auto flush = [&]() {
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        sums[(2 * c) * 32] = (double)lo_of(A[c]) - (double)hi_of(B[c]);
        sums[(2 * c + 1) * 32] = (double)hi_of(A[c]) + (double)lo_of(B[c]);
        A[c] = B[c] = 0ull;
      }
    };
    // Rows in four runs: the first half-window's other rows, its centre rows
    // (14, 15), the flush, the second half's centre rows (20, 21), then its
    // other rows; the centre rows skip the zero adjacent offsets.
    constexpr unsigned long long kLow = (1ull << 18) - 1;  // z-planes 0-2
    constexpr unsigned long long kCentre = (1ull << 14) | (1ull << 15) | (1ull << 20) | (1ull << 21);
    auto run_rows = [&](int run) {
      return rows & (run < 2 ? kLow : ~kLow) & (run == 1 || run == 2 ? kCentre : ~kCentre);
    };
    auto first_after = [&](int run) {  // first row of the runs after `run`, 36 if none
      for (int q = run + 1; q < 4; ++q) {
        const unsigned long long mm = run_rows(q);
        if (mm) return __ffsll((long long)mm) - 1;
      }
      return 36;
    };
    // the next row's source spectra are loaded while the current row is
    // multiplied, across the runs' boundaries too
    unsigned long long nxt[8];
    auto fetch = [&](int r) {
#pragma unroll
      for (int x = 0; x < 8; ++x) {
        const int sid = w[r * 8 + x];
        nxt[x] = sid >= 0 ? spec[(size_t)sid * kFB] : 0ull;
      }
    };
    {
      const int r0 = first_after(-1);
      if (r0 < 36) fetch(r0);
    }
#pragma unroll 1
    for (int run = 0; run < 4; ++run) {
      if (run == 2) flush();
      unsigned long long m = run_rows(run);
      int row = m ? __ffsll((long long)m) - 1 : 36;
      auto walk = [&](auto centre) {
        while (row < 36) {
          m &= m - 1;
          const int next = m ? __ffsll((long long)m) - 1 : 36;
          const int ahead = next < 36 ? next : first_after(run);
          unsigned long long sr[8], si[8];  // {sr, sr}, {si, si}
#pragma unroll
          for (int x = 0; x < 8; ++x) {
            sr[x] = pack2(lo_of(nxt[x]), lo_of(nxt[x]));
            si[x] = pack2(hi_of(nxt[x]), hi_of(nxt[x]));
          }
          if (ahead < 36) fetch(ahead);
          const int wy = row % 6, wz = row / 6;
          const unsigned long long* trow0 = tsm + ((wz + 1) * 49 + (wy + 1) * 7) * kFB + f;
          if constexpr (decltype(centre)::value) had_pair_row_centre(A, B, sr, si, trow0);
          else had_pair_row(A, B, sr, si, trow0);
          row = next;
        }
      };
      if (run == 1 || run == 2) walk(std::true_type{});
      else walk(std::false_type{});
    }
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      const int m = mem[slot][c];
      if (m >= 0)
        p.effv[(fbase + m) * kFB + f] =
            make_float2((float)(sums[(2 * c) * 32] + ((double)lo_of(A[c]) - (double)hi_of(B[c]))),
                        (float)(sums[(2 * c + 1) * 32] + ((double)hi_of(A[c]) + (double)lo_of(B[c]))));
    }
    __syncwarp();
  }
}

// Sparse groups as in the FP64 form, two CTAs per SM; each 32 entries' FP32 sums
// are added in FP64.
constexpr int kHadSparseThreads = 256;
constexpr int kHadSparseWarps = kHadSparseThreads / 32;

struct HadSparse32Params {
  int nn;
  HadSparse sparse;
  const float2* tile;
  const float2* spec;
  float2* effv;
  int* error;
  long long wait_limit;
};

__global__ void __launch_bounds__(kHadSparseThreads, 2)
hadamard_fp32_sparse_kernel(HadSparse32Params p) {
  extern __shared__ __align__(128) unsigned char had32_dyn[];
  __shared__ __align__(8) unsigned long long bar;
  const unsigned long long* tsm = (const unsigned long long*)had32_dyn;
  const HadSparse& q = p.sparse;
  const int f = threadIdx.x & 31, slot = threadIdx.x >> 5, chunk = blockIdx.x;
  const size_t fbase = (size_t)blockIdx.y * p.nn;
  if (!had_load_tile<kHad32TileBytes>(p.tile + (size_t)blockIdx.y * 343 * kFB, had32_dyn, &bar,
                                      p.error, p.wait_limit))
    return;
  const unsigned long long* spec = (const unsigned long long*)p.spec + fbase * kFB + f;
  const int g1 = min(q.n, (chunk + 1) * q.per_block);
  for (int g = chunk * q.per_block + slot; g < g1; g += kHadSparseWarps) {
    const int end = q.ptr[g + 1];
    double ar[8], ai[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) ar[c] = ai[c] = 0.0;
    for (int e0 = q.ptr[g]; e0 < end; e0 += 32) {
      const int n = min(32, end - e0);
      const int2 mine = f < n ? q.ent[e0 + f] : make_int2(0, 0);
      unsigned long long A[8], B[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) A[c] = B[c] = 0ull;
      constexpr int U = 4;
      unsigned long long nxt[U];
      auto fetch = [&](int i) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int node = __shfl_sync(0xffffffffu, mine.x, i + u);
          nxt[u] = i + u < n ? spec[(size_t)node * kFB] : 0ull;
        }
      };
      fetch(0);
      for (int i = 0; i < n; i += U) {
        unsigned long long sr[U], si[U];
        const unsigned long long* t[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          sr[u] = pack2(lo_of(nxt[u]), lo_of(nxt[u]));
          si[u] = pack2(hi_of(nxt[u]), hi_of(nxt[u]));
          const int k = __shfl_sync(0xffffffffu, mine.y, i + u);
          t[u] = tsm + (i + u < n ? k : had_member_offset(7)) * kFB + f;
        }
        if (i + U < n) fetch(i + U);
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const unsigned long long w = t[u][-had_member_offset(c) * kFB];
            asm("fma.rn.f32x2 %0, %2, %3, %0;\n"
                "fma.rn.f32x2 %1, %2, %4, %1;\n"
                : "+l"(A[c]), "+l"(B[c])
                : "l"(w), "l"(sr[u]), "l"(si[u]));
          }
      }
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        ar[c] += (double)lo_of(A[c]) - (double)hi_of(B[c]);
        ai[c] += (double)hi_of(A[c]) + (double)lo_of(B[c]);
      }
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int m = q.members[(size_t)g * 8 + c];
      if (m >= 0) p.effv[(fbase + m) * kFB + f] = make_float2((float)ar[c], (float)ai[c]);
    }
  }
}

#include "hadamard_tc.cuh"

// ---------------------------------------------------------------------------
// Point reordering (fmm/evaluate.cc:14-52 on the host in the reference); the near
// field stores original order itself (copy_trg_val, fmm/cuda.cu:2543-2565).
// ---------------------------------------------------------------------------
// Points to leaf order, driven from the original order: point k (read
// coalesced) goes to leaf-order position inv[k], one full 32-byte record
// (and, for mixed plans, a 16-byte record of FP32 offsets from the point's
// leaf centre, leaf[i]) per store; gathering instead reads 8 bytes from four
// random places per point.
//
// A coordinate beyond 2^510 is brought back to it, and a source that has one weighs
// nothing: its r^2 would be infinite, where pair_rsqrt gives NaN without its guard,
// while such a pair adds nothing (a source can be parked at infinity).
__global__ void scatter_points_kernel(int n, const int* inv, const double* x, const double* y,
                                      const double* z, const double* w, double4* out) {
  constexpr double kFar = 0x1p510;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    double4 v = make_double4(x[k], y[k], z[k], w ? w[k] : 0.0);
    bool far = false;
    auto near = [&](double& c) {
      if (fabs(c) > kFar) {
        c = copysign(kFar, c);
        far = true;
      }
    };
    near(v.x);
    near(v.y);
    near(v.z);
    if (far) v.w *= 0.0;  // NaN when the weight is not finite
    out[inv[k]] = v;
  }
}

// Mixed plans keep only the FP32 offsets (src4f); leaf[k]: source k's leaf.
__global__ void scatter_sources_mixed_kernel(int n, const int* inv, const int* leaf,
                                             const double* x, const double* y, const double* z,
                                             const double* w, const double4* ctr, float4* outf) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const double4 c = ctr[leaf[k]];
    outf[inv[k]] =
        make_float4((float)(x[k] - c.x), (float)(y[k] - c.y), (float)(z[k] - c.z), (float)w[k]);
  }
}

// Leaf-order view of original-order potentials (introspection).
__global__ void gather_pot_kernel(int n, const int* perm, const double* pot_orig,
                                  double* pot_leaf) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    pot_leaf[i] = pot_orig[perm[i]];
}

// error[1] |= error[0]: the per-solve flag of a bounded wait folded into the
// flag kfmm_evaluate_wait reports for every solve queued since the last wait.
__global__ void error_fold_kernel(int* error) {
  if (error[0]) error[1] = 1;
}

// The error flags of a batch's plans, side by side.
__global__ void gather_flags_kernel(int n, const int* const* flags, int* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = *flags[i];
}

// Direct sum (ulist__direct_evaluation) over SoA device arrays, any coordinates.
// Bound by the FP64 pipe (12 operations a pair, pair_rsqrt).  A warp takes 32
// targets, one per lane, and every (kSplit x cluster size)-th chunk of 32 sources,
// staged in its slice of shared memory and read back as broadcasts, the next
// chunk prefetched into registers; a CTA's 16 warps are 16 / kSplit target tiles
// times kSplit shares of the sources.  The shares are added in a fixed order, a
// CTA's through shared memory and a cluster's through distributed shared memory,
// so there is no scratch array, no atomic and one launch.  1,000 targets x 1,048,576
// sources: one thread per target 92.6 ms (8 blocks), this 1.14 ms (0.92e12 pairs/s
// of 1.5e12; its 256 blocks leave 40 of 296 slots empty).
constexpr int kDirectWarps = 16;
constexpr int kDirectCluster = 8;

template <int kSplit>
__global__ void __launch_bounds__(32 * kDirectWarps, 2)
direct_fp64_kernel(int nt, const double* tx, const double* ty, const double* tz, double* pot,
                   int ns, const double* sx, const double* sy, const double* sz,
                   const double* den) {
  __shared__ double4 stage[kDirectWarps][32];
  __shared__ double part[kDirectWarps][32];
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int nrank = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tile = (int)(blockIdx.x / nrank) * (kDirectWarps / kSplit) + warp / kSplit;
  const long long i = (long long)tile * 32 + lane;
  double x[1] = {0.0}, y[1] = {0.0}, z[1] = {0.0}, acc[1] = {0.0};
  if (i < nt) {
    x[0] = tx[i];
    y[0] = ty[i];
    z[0] = tz[i];
  }
  const int nchunks = (int)(((long long)ns + 31) / 32), step = kSplit * nrank;
  double4 s = make_double4(0.0, 0.0, 0.0, 0.0);
  auto fetch = [&](int c) {
    const int b = 32 * c;
    if (c < nchunks && lane < ns - b)
      s = make_double4(sx[b + lane], sy[b + lane], sz[b + lane], den[b + lane]);
  };
  if ((long long)tile * 32 < nt) {  // warp-uniform
    int c = rank * kSplit + warp % kSplit;
    fetch(c);
    for (; c < nchunks; c += step) {
      stage[warp][lane] = s;
      __syncwarp();
      fetch(c + step);
      pairs_fp64<1, true>(x, y, z, acc, stage[warp], min(32, ns - 32 * c));
      __syncwarp();
    }
  }
  if constexpr (kSplit == 1) {
    if (i < nt) pot[i] += kOOFP * acc[0];
  } else {
    part[warp][lane] = acc[0];
    __syncthreads();
    if (warp % kSplit == 0) {
      double sum = part[warp][lane];
#pragma unroll
      for (int w = 1; w < kSplit; ++w) sum += part[warp + w][lane];
      part[warp][lane] = sum;
    }
    cluster.sync();
    if (rank == 0 && warp % kSplit == 0 && i < nt) {
      double sum = 0.0;
      for (int r = 0; r < nrank; ++r) sum += cluster.map_shared_rank(&part[warp][lane], r)[0];
      pot[i] += kOOFP * sum;
    }
    cluster.sync();  // the other blocks' shared memory stays until it is read
  }
}

}  // namespace kfmm
