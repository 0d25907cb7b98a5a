// Sequential K-SVD dictionary update (updateDictionary,
// cuda_svd_denoiser.cu:285-362) on a maintained residual.
//
// The residual R = Y - X D (one n-vector per patch) is formed once before the
// sweep.  For atom j with support Omega_j (c entries, only the first 1024
// with the Q1 cap) the columns of the reference's error matrix are then
//     e_p = r_p + x_{j,p} d_j            (p in Omega_j)
// which equals y_p - sum_{s != j} x_{s,p} d_s with every earlier atom of the
// sweep already updated (the reference's Gauss-Seidel order, :309-361).  The
// top left singular vector u of E = [e_p] (gesvdj's U[:,0], :328-346) is
// found by power iteration on E itself, w = E (E^T u), warm-started from the
// old atom; u is signed so that u . d_j(old) >= 0; then
//     d_j <- u,  x_{j,p} <- u . e_p (= sigma v_p, :349-358),
//     r_p <- e_p - x_{j,p} u,
// with x_{j,p} = 0 (and r_p <- e_p) for entries beyond the cap.
//
// One persistent cooperative kernel walks the atoms.  An atom's entries are
// split over `active` CTAs (about slice_target entries each); each keeps its
// columns in shared memory (those beyond the capacity are re-read from the
// residual on every pass).  A power step is one pass over the local columns
// producing a partial w, then an all-reduce: each CTA writes its partial (as
// tagged words, or as a plain row behind a counter) and sums all CTAs'
// partials in the same fixed order, so every CTA holds the same u and takes
// the same convergence decision.  A CTA alone on its atom needs no exchange.
// An atom's CTAs wait for the previous atom's CTAs to finish their residual
// stores before reading the residual; since those in turn waited for the atom
// before, every earlier atom of the sweep is complete by then.  CTAs with no entries in an atom skip it.  All
// waits are bounded.
#include <cuda_runtime.h>

#include "device_util.cuh"
#include "ksvd_internal.cuh"

namespace ksvd {

constexpr int kUrThreads = 512;
constexpr int kUrWarps = kUrThreads / 32;
constexpr int kUrDefaultSlice = 64;   // entries per CTA before another CTA joins an atom (default)
constexpr int kUrMaxIters = 200;
constexpr float kUrTol = 2.0e-7f;     // max |u_new - u_old| to stop
constexpr size_t kUrSmemMax = 232448 - 256;  // opt-in shared memory per block, less the static part

__host__ __device__ inline int ur_n4(int n) { return (n + 3) & ~3; }

// Row stride of the resident columns (floats): a multiple of 4 whose float4
// count is odd, so that the 8 rows a quarter-warp reads with 16-byte loads
// sit in distinct banks.
__host__ __device__ inline int ur_es(int n) { return 4 * ((ur_n4(n) / 4) | 1); }

// Column groups of the w pass, and groups of partials of the all-reduce: the
// order in which w is summed.
__host__ __device__ inline int ur_groups(int n) {
  const int g = kUrThreads / (ur_n4(n) / 4);
  return g > 16 ? 16 : (g < 1 ? 1 : g);
}

// Row stride of the transposed u (floats): 16-byte rows in distinct banks.
__host__ __device__ inline int ur_ft(int n) { return 4 * (((ur_n4(n) / 4 + 3) / 4) | 1); }

// Shared memory: [cap x es] columns | row[2][cap] | xold[2][cap] | slices of the
// next atoms (int4 [kUrTab]) | transposed u[4][ft] | u[n4] | dold[2][n4] | wsum[n4] |
// wred[groups x n4] | streamed columns: [16 x n4].  The capacity also decides which columns are
// streamed, hence the order of their sums; it is the one of a layout of 24
// bytes a column and 35 rows.
constexpr int kUrTab = 128;

int update_res_capacity(int n) {
  const size_t per = size_t(ur_es(n)) * 4 + 24;
  const size_t fixed = size_t(35) * ur_n4(n) * 4;
  if (fixed + per * 16 > kUrSmemMax) return 0;
  return int((kUrSmemMax - fixed) / per) & ~3;
}

size_t update_res_smem_bytes(int n, int cap) {
  return size_t(cap) * (size_t(ur_es(n)) * 4 + 16) + kUrTab * 16 + size_t(4) * ur_ft(n) * 4 +
         size_t(4 + ur_groups(n) + kUrWarps) * ur_n4(n) * 4;
}

// Bounded spin of thread 0 until *ctr >= target.  False on timeout or when an
// error is already flagged.
KSVD_DEV bool ur_wait_count(const unsigned* ctr, unsigned target, GridBarrier* flags) {
  if (ld_acquire_u32(ctr) >= target) return true;
  const unsigned long long t0 = globaltimer_ns();
  while (ld_acquire_u32(ctr) < target) {
    if (ld_relaxed_i32(&flags->err) != DEVERR_NONE) return false;
    if (globaltimer_ns() - t0 > kBarrierTimeoutNs) {
      atomicCAS(&flags->err, DEVERR_NONE, DEVERR_TIMEOUT);
      return false;
    }
    __nanosleep(20);
  }
  return true;
}

__host__ __device__ inline int ur_active(int c, int G, int target) {
  const int a = (c + target - 1) / target;
  return a < G ? a : G;
}

// residual_kernel: R = Y - X D, one warp per patch (every patch, or those of
// a device-side list).  The patch's atoms and
// coefficients sit in lanes 0..L-1 and are broadcast by shuffles; each lane
// forms 16-byte pieces of the row with the support atoms' loads in flight
// together (same FMA order as r = y - sum_s x_s d_s, s ascending).  last[p]
// (optional) receives the highest atom of the patch's support (-1 if none):
// the sweep visits atoms in ascending order, so no atom after that one reads
// the patch's residual row again in the sweep.
__global__ void __launch_bounds__(256) residual_kernel(const float* __restrict__ Y, int64_t N, int n,
                                                       const float* __restrict__ D, int K, int L,
                                                       const int32_t* __restrict__ idx,
                                                       const float* __restrict__ coef, float* __restrict__ R,
                                                       int* __restrict__ last, int vec4,
                                                       const int64_t* __restrict__ list,
                                                       const unsigned long long* __restrict__ count) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = int64_t(gridDim.x) * (blockDim.x >> 5);
  int64_t total = N;  // every patch, or list[0 .. *count)
  if (list) {
    const unsigned long long c = *count;
    total = c < static_cast<unsigned long long>(N) ? int64_t(c) : N;
  }
  for (int64_t w = int64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); w < total; w += warps) {
    const int64_t p = list ? list[w] : w;
    int a = -1;
    float x = 0.0f;
    if (lane < L) {
      a = __ldg(idx + p * L + lane);
      x = __ldg(coef + p * L + lane);
      if (a < 0 || a >= K || x == 0.0f) a = -1;
    }
    if (last) {
      int top = a;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
      if (lane == 0) last[p] = top;
    }
    if (vec4) {
      const int F = n >> 2;
      const float4* y4 = reinterpret_cast<const float4*>(Y + p * n);
      float4* r4 = reinterpret_cast<float4*>(R + p * n);
      for (int f0 = 0; f0 < F; f0 += 32) {
        const int f = f0 + lane;
        const bool in = f < F;
        float4 r = in ? __ldg(y4 + f) : make_float4(0.f, 0.f, 0.f, 0.f);
        for (int s0 = 0; s0 < L; s0 += 8) {
          float4 dv[8];
          float xs[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const int as = __shfl_sync(0xffffffffu, a, (s0 + u) & 31);
            xs[u] = __shfl_sync(0xffffffffu, x, (s0 + u) & 31);
            const bool use = in && s0 + u < L && as >= 0;
            dv[u] = use ? __ldg(reinterpret_cast<const float4*>(D + int64_t(as) * n) + f)
                        : make_float4(0.f, 0.f, 0.f, 0.f);
            if (!use) xs[u] = 0.0f;
          }
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            if (xs[u] != 0.0f) {
              r.x = fmaf(-xs[u], dv[u].x, r.x);
              r.y = fmaf(-xs[u], dv[u].y, r.y);
              r.z = fmaf(-xs[u], dv[u].z, r.z);
              r.w = fmaf(-xs[u], dv[u].w, r.w);
            }
          }
        }
        if (in) r4[f] = r;
      }
    } else {
      for (int i0 = 0; i0 < n; i0 += 32) {
        const int i = i0 + lane;
        const bool in = i < n;
        float r = in ? Y[p * n + i] : 0.0f;
        for (int s = 0; s < L; ++s) {
          const int as = __shfl_sync(0xffffffffu, a, s & 31);
          const float xs = __shfl_sync(0xffffffffu, x, s & 31);
          if (in && as >= 0) r = fmaf(-xs, __ldg(D + int64_t(as) * n + i), r);
        }
        if (in) R[p * n + i] = r;
      }
    }
  }
}

// Arrive on a counter with release semantics: after a __syncthreads(), the
// writes of every thread of the CTA are visible to whoever acquires the count.
KSVD_DEV void red_release_add(unsigned* p, unsigned v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// A partial travels between CTAs as 16-byte words {three floats, tag}: each word is
// one 128-bit access, so a reader that finds the tag of the step it waits for
// has the three values with it.  No counter, fence or second read follows the
// store (a release on a counter, its poll and the read of the partials took
// two L2 round trips more per power step).
__host__ __device__ inline int ur_words(int n) { return (ur_n4(n) + 2) / 3; }

KSVD_DEV void st_word(uint4* p, float x, float y, float z, unsigned tag) {
  const unsigned long long lo = (static_cast<unsigned long long>(__float_as_uint(y)) << 32) | __float_as_uint(x);
  const unsigned long long hi = (static_cast<unsigned long long>(tag) << 32) | __float_as_uint(z);
  asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(p), "l"(lo),
               "l"(hi)
               : "memory");
}

KSVD_DEV uint4 ld_word(const uint4* p) {
  unsigned long long lo, hi;
  asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
               : "=l"(lo), "=l"(hi)
               : "l"(p)
               : "memory");
  return make_uint4(unsigned(lo), unsigned(lo >> 32), unsigned(hi), unsigned(hi >> 32));
}

// CTAs whose partials travel as words: at most this many a group of partials
// (more go behind a counter, see `counted`).
constexpr int kUrWordRounds = 2;

// Sum of the words p[0], p[stride], ... (count of them) in ascending order, once
// they show the tag: up to kUrWordRounds are polled together (re-reading one word
// after the other would cost an L2 round trip each; eight at a time cost every
// instantiation 12 to 50 bytes of spilled registers).  w of the result: 1, or 0
// when the time is over or an error is flagged elsewhere.
KSVD_DEV float4 ur_gather(const uint4* p, size_t stride, int count, unsigned tag, GridBarrier* flags) {
  constexpr int kB = kUrWordRounds;
  float4 a = make_float4(0.f, 0.f, 0.f, 1.f);
  for (int i = 0; i < count; i += kB) {
    uint4 v[kB];
#pragma unroll
    for (int k = 0; k < kB; ++k) v[k] = (i + k < count) ? ld_word(p + (i + k) * stride) : make_uint4(0u, 0u, 0u, tag);
    unsigned spins = 0;
    unsigned long long t0 = 0;
    for (;;) {
      bool ready = true;
#pragma unroll
      for (int k = 0; k < kB; ++k) ready = ready && v[k].w == tag;
      if (ready) break;
#pragma unroll
      for (int k = 0; k < kB; ++k)
        if (v[k].w != tag) v[k] = ld_word(p + (i + k) * stride);
      if ((++spins & 63u) == 0u) {
        const unsigned long long t = globaltimer_ns();
        if (t0 == 0) t0 = t;
        if (t - t0 > kBarrierTimeoutNs) atomicCAS(&flags->err, DEVERR_NONE, DEVERR_TIMEOUT);
        if (ld_relaxed_i32(&flags->err) != DEVERR_NONE) {
          a.w = 0.0f;
          return a;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < kB; ++k) {
      a.x += __uint_as_float(v[k].x);
      a.y += __uint_as_float(v[k].y);
      a.z += __uint_as_float(v[k].z);
    }
  }
  return a;
}

// Phase timer of one thread: the time since the last mark goes to `slot`.
__device__ __noinline__ void ur_lap(unsigned long long* ph, int slot) {
  const unsigned long long t = globaltimer_ns();
  ph[slot] += t - ph[8];
  ph[8] = t;
}

// One launch sweeps one or several problems (images): group g owns the CTAs
// [cta_begin, cta_begin + ctas) and walks its own atoms with its own buffers,
// counters and partials.  Groups whose ranges share CTAs run one after the
// other on those CTAs, in the order of the table; a group only waits for its
// own CTAs, and every CTA takes its groups in the same (table) order, so the
// lowest unfinished group always has all its CTAs and the launch cannot
// deadlock.
//
// What bounds the sweep is the latency of K atoms in sequence, each a handful
// of dependent steps (128 x 128 image, 8 x 8 patches, 256 atoms: 10 us an atom,
// 14.5 with one thread per column, warp 0 finishing each step and a counter for
// every exchange; 1000 x 777, 10 x 11 patches: 16 us, 25 before), so all that is not needed for the next step is kept off
// them: the slices of the atoms are tabulated, an atom's entries, old
// coefficients and old atom arrive during the atom before, e = r + x d_old is
// formed inside the first pass over the columns, and every warp finishes a
// power step for itself from the summed w.  The sums are in a fixed order
// (dot_u, the column groups, the groups of partials), whatever thread makes them.
template <int NW>
__global__ void __launch_bounds__(kUrThreads, 1)
    update_res_kernel(const __grid_constant__ UpdBatch batch, GridBarrier* flags, DevStats* stats, int timers) {
  extern __shared__ __align__(16) unsigned char ursm[];
  __shared__ int s_ok;
  __shared__ __align__(8) unsigned long long s_mbar;  // completion of the residual-row bulk copies
  __shared__ unsigned long long s_ph[9];  // phase times of this CTA (slots 0..7), the last mark
  constexpr int KF = (NW + 3) / 4;        // float4 per lane of a row of up to 32 NW features
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned mpar = 0;  // parity of the next phase of s_mbar
  if (tid == 0) {
    mbar_init(&s_mbar, 1);
    fence_mbar_init();
  }

  // phase times gather in shared memory and are flushed once at the end
  const bool timer = (timers != 0 && blockIdx.x == 0 && tid == 0);
  if (timer)
    for (int k = 0; k < 8; ++k) s_ph[k] = 0ull;
  if (timer) s_ph[8] = globaltimer_ns();
  auto lap = [&](int slot) {
    if (timer) ur_lap(s_ph, slot);
  };

  // every group whose CTA range holds this CTA, in the order of the table
  for (int gi = 0; gi < batch.ngroups; ++gi) {
    const UpdGroup& grp = batch.g[gi];
    if (int(blockIdx.x) < grp.cta_begin || int(blockIdx.x) >= grp.cta_begin + grp.ctas) continue;
    // bulk copies of this group may land where the previous one, of another
    // layout, kept its tables (fill_tab's barrier follows)
    fence_proxy_async_smem();
    float* const R = grp.R;
    float* const D = grp.D;
    float* const coef = grp.coef;
    const int* __restrict__ const entries = grp.entries;
    const int* __restrict__ const last = grp.last;
    const int n = grp.n, K = grp.K, L = grp.L, q1_cap = grp.q1_cap, cap = grp.cap;
    const int slice_target = grp.slice_target > 0 ? grp.slice_target : kUrDefaultSlice;
    const int n4 = ur_n4(n), es = ur_es(n), W = ur_words(n), Gr = ur_groups(n);
    const int F = n4 / 4, es4 = es / 4;  // float4 per row of u / w, per resident column
    const int G = grp.ctas, b = int(blockIdx.x) - grp.cta_begin;
    uint4* const words = static_cast<uint4*>(grp.gw);  // [2][G][W] partials, by parity of the step
    unsigned* const done_cnt = reinterpret_cast<unsigned*>(words + size_t(2) * G * W);
    unsigned* const iter_cnt = done_cnt + K;
    float* const raw = reinterpret_cast<float*>(words + size_t(2) * G * W + (K + 1) / 2);  // [2][G][n4] plain partials
    float* const Es = reinterpret_cast<float*>(ursm);
    float4* const Es4 = reinterpret_cast<float4*>(ursm);
    int* const row_b = reinterpret_cast<int*>(ursm + size_t(cap) * es * 4);  // [2][cap] patches
    float* const xold_b = reinterpret_cast<float*>(row_b + 2 * cap);         // [2][cap]
    int4* const tab = reinterpret_cast<int4*>(xold_b + 2 * cap);
    float* const ut = reinterpret_cast<float*>(tab + kUrTab);  // [4][ft] ut[c][f] = u[4 f + c]
    const int ft = ur_ft(n);
    float* const u = ut + 4 * ft;
    float* const dbuf = u + n4;        // [2][n4] old atom: this one's and the next one's
    float* const wsum = dbuf + 2 * n4;
    float* const wred = wsum + n4;     // [Gr][n4] sums over column groups, over groups of partials
    float* const wstr = wred + Gr * n4;  // [16][n4] sums over the streamed columns of a warp
    float* const xrow = wstr;            // [Gr][n4] sums over groups of partials
    const int x_g = tid / W, x_f = tid - x_g * W;  // this thread's first group and word
    const int s_q = tid / F, s_f = tid - s_q * F;  // its first column and float4 of the row stores, the stride
    const int d_q = kUrThreads / F, d_f = kUrThreads - d_q * F;
    float4* const u4 = reinterpret_cast<float4*>(u);
    const float4* const wsum4 = reinterpret_cast<const float4*>(wsum);
    // w pass: a warp per column group with its lanes over the features, or a
    // float4 of a group per thread.  The former needs a group for most warps (n <=
    // 224; with 8 groups, 512 x 512, 16 x 16, the local pass takes 2.1 ms a sweep
    // against 1.3) and runs 32 NW features, NW of the launch's widest patch (the
    // latter with 144 features: 1.3 ms at 2048 x 2048 against 1.1).
    const bool lanes_w = 2 * Gr > kUrWarps && NW == (n + 31) / 32;
    // bulk copies need 16-byte aligned rows of a multiple of 16 bytes
    const bool tma = (n & 3) == 0 && (reinterpret_cast<uintptr_t>(R) & 15) == 0;

    // this CTA's slice [sb, sb + m) of each of the next kUrTab atoms' c entries:
    // first entry, m (-1: no part in the atom), entries that enter the power
    // iteration, CTAs on the atom (0: unused atom)
    auto fill_tab = [&](int a0) {
      __syncthreads();
      for (int t = tid; t < kUrTab && a0 + t < K; t += kUrThreads) {
        const int beg = __ldg(grp.atom_ptr + a0 + t), c = __ldg(grp.atom_ptr + a0 + t + 1) - beg;
        const int active = c > 0 ? ur_active(c, G, slice_target) : 0;
        int sb = 0, m = -1, mc = 0;
        if (b < active) {
          sb = int(int64_t(c) * b / active);
          m = int(int64_t(c) * (b + 1) / active) - sb;
          const int c_eff = (q1_cap && c > 1024) ? 1024 : c;
          mc = max(0, min(m, c_eff - sb));
        }
        tab[t] = make_int4(beg + sb, m, mc, active);
      }
      __syncthreads();
    };
    // patches and old coefficients of the first `cnt` columns of a slice into meta
    // buffer `slot`, in three steps (thread t: column t, so the loads of one step
    // may be in flight while the block does something else).  A patch's
    // complement marks a residual row that is not stored back: a is the last
    // atom of the patch's support.
    struct Meta {
      int en, pt, lt;
      float x;
    };
    auto meta_entry = [&](Meta& md, int first, int cnt, int t) {
      md.en = t < cnt ? __ldg(entries + first + t) : -1;
    };
    auto meta_rest = [&](Meta& md) {
      md.x = md.en >= 0 ? __ldcg(coef + md.en) : 0.0f;
      md.pt = md.en >= 0 ? md.en / L : 0;
      md.lt = (md.en >= 0 && last != nullptr) ? __ldg(last + md.pt) : -1;
    };
    auto meta_store = [&](const Meta& md, int slot, int a, int t) {
      if (md.en >= 0) {
        row_b[slot * cap + t] = md.lt != a ? md.pt : ~md.pt;
        xold_b[slot * cap + t] = md.x;
      }
    };
    auto row_of = [](int p) -> int64_t { return p >= 0 ? p : ~p; };
    // u . e_q for a resident column: four chains, chain c over the features
    // 4 f + c, one per lane of four; (a0 + a1) + (a2 + a3) in every lane.  With
    // `form`, e = r + x d is formed in place first.  The four lanes' words of a
    // column and the eight columns of a warp sit in distinct banks, and u comes
    // four features of a chain at a time from its transposed copy.
    auto dot_u = [&](int q, bool in, bool form, float x) -> float {
      float* const er = Es + size_t(q) * es + (lane & 3);
      const float4* const uc = reinterpret_cast<const float4*>(ut + (lane & 3) * ft);
      float a = 0.0f;
      if (in) {
        auto term = [&](int f, float w) {
          float e = er[4 * f];
          if (form) {
            e = fmaf(x, w, e);
            er[4 * f] = e;
          }
          a = fmaf(e, w, a);
        };
        int f = 0;
#pragma unroll 2
        for (; f + 4 <= F; f += 4) {
          const float4 w = uc[f >> 2];
          float e0 = er[4 * f], e1 = er[4 * f + 4], e2 = er[4 * f + 8], e3 = er[4 * f + 12];
          if (form) {
            e0 = fmaf(x, w.x, e0);
            e1 = fmaf(x, w.y, e1);
            e2 = fmaf(x, w.z, e2);
            e3 = fmaf(x, w.w, e3);
            er[4 * f] = e0;
            er[4 * f + 4] = e1;
            er[4 * f + 8] = e2;
            er[4 * f + 12] = e3;
          }
          a = fmaf(e0, w.x, a);
          a = fmaf(e1, w.y, a);
          a = fmaf(e2, w.z, a);
          a = fmaf(e3, w.w, a);
        }
        for (; f < F; ++f) term(f, ut[(lane & 3) * ft + f]);
      }
      a += __shfl_xor_sync(0xffffffffu, a, 1);
      a += __shfl_xor_sync(0xffffffffu, a, 2);
      return a;
    };
    const int q_l = warp * 8 + (lane >> 2);  // this lane's column of 128

    int jprev = -1, aprev = 0;
    int slot = 0;        // meta and old-atom buffer of the current atom
    int meta_atom = -1;  // atom whose meta is in buffer `slot`
    for (int j = 0; j < K; ++j) {
      if (j % kUrTab == 0) fill_tab(j);
      const int4 sl = tab[j % kUrTab];
      const int first = sl.x, m = sl.y, mc = sl.z, active = sl.w;
      if (active == 0) continue;
      const int jp = jprev, ap = aprev;
      jprev = j;
      aprev = active;
      if (m < 0) continue;
      const int mres = min(m, cap);
      const int mcr = min(mc, cap);   // resident columns in the power iteration
      const bool streamed = mc > cap;  // some enter from the residual
      const bool alone = active == 1;
      // Partials of many CTAs: as plain rows behind a counter, which one thread
      // polls, instead of as tagged words that every thread polls.  Tagged words
      // save a release and a round trip a step (1.8 against 2.1 us with 9 CTAs,
      // 144 features), but each carries a quarter more bytes and the polls of many
      // CTAs slow the stores they wait for (3.2 against 3.0 us with 141 CTAs).  In
      // between it hardly matters: with the line at 1, 2, 3 or 4 words a group, sweeps
      // with 3 to 61 CTAs an atom and 64 to 484 features differ by 1.5% at most
      // (512 x 512, 16 x 16, 19 CTAs: 4.49, 4.48, 4.45, 4.46 ms).
      const bool counted = active > kUrWordRounds * Gr;
      float* const v_s = xold_b + slot * cap;  // old coefficients, then per-column scalars
      const int* const row_s = row_b + slot * cap;
      const float* const dold = dbuf + slot * n4;
      const float4* const dold4 = reinterpret_cast<const float4*>(dold);

      // ---- entries, old coefficients and the old atom: never written by other
      // atoms, so read before the wait (or during the previous atom)
      if (meta_atom != j) {
        for (int t = tid; t < mres; t += kUrThreads) {
          Meta md;
          meta_entry(md, first, mres, t);
          meta_rest(md);
          meta_store(md, slot, j, t);
        }
        for (int i = tid; i < n4; i += kUrThreads) {
          const float d = (i < n) ? __ldcg(D + int64_t(j) * n + i) : 0.0f;
          dbuf[slot * n4 + i] = d;
          ut[(i & 3) * ft + (i >> 2)] = d;
        }
        __syncthreads();
      }
      lap(7);
      // the previous atom's residual rows (what this CTA stored alone needs no wait)
      if (jp >= 0 && (ap > 1 || b > 0)) {
        if (tid == 0) s_ok = ur_wait_count(done_cnt + jp, unsigned(ap), flags) ? 1 : 0;
        __syncthreads();
        if (!s_ok) return;
      }
      lap(0);

      // ---- residual rows ----------------------------------------------------
      bool ok = true;
      if (tma) {
        // bulk copies (the residual was written by other CTAs through the generic
        // proxy: acquire above, proxy fence here)
        if (tid == 0) mbar_arrive_expect_tx(&s_mbar, unsigned(mres) * unsigned(n) * 4u);
        asm volatile("fence.proxy.async.global;" ::: "memory");
        for (int q = tid; q < mres; q += kUrThreads)
          bulk_g2s(Es + size_t(q) * es, R + row_of(row_s[q]) * n, unsigned(n) * 4u, &s_mbar);
      } else {
        for (int q = warp; q < mres; q += 2 * kUrWarps) {
          const int q1 = q + kUrWarps;
          const float* ra = R + row_of(row_s[q]) * n;
          const float* rb = R + (q1 < mres ? row_of(row_s[q1]) : 0) * n;
          float r0[NW], r1[NW];
#pragma unroll
          for (int k = 0; k < NW; ++k) {
            const int i = lane + 32 * k;
            r0[k] = i < n ? __ldcg(ra + i) : 0.0f;
            r1[k] = i < n && q1 < mres ? __ldcg(rb + i) : 0.0f;
          }
#pragma unroll
          for (int k = 0; k < NW; ++k) {
            const int i = lane + 32 * k;
            if (i < n4) Es[size_t(q) * es + i] = r0[k];
            if (i < n4 && q1 < mres) Es[size_t(q1) * es + i] = r1[k];
          }
        }
      }

      // the entry of this thread's column, for its new coefficient
      const int c_en = (lane & 3) == 0 && q_l < mres ? __ldg(entries + first + q_l) : 0;

      // the next non-empty atom; if this CTA works on it, its meta is fetched
      // while this one is worked on
      int jn = j + 1;
      while (jn < K && jn % kUrTab != 0 && tab[jn % kUrTab].w == 0) ++jn;
      int nact = 2;  // its CTAs (beyond the table: assume several)
      bool prefetch = false;
      Meta nm{-1, 0, -1, 0.0f};
      float nd = 0.0f;
      if (jn < K && jn % kUrTab != 0) {
        const int4 ns = tab[jn % kUrTab];
        nact = ns.w;
        prefetch = ns.y >= 0 && min(ns.y, cap) <= kUrThreads;
        if (prefetch) {
          meta_entry(nm, ns.x, min(ns.y, cap), tid);
          nd = (tid < n) ? __ldcg(D + int64_t(jn) * n + tid) : 0.0f;
        }
      }
      lap(1);
      if (tma) {
        ok = mbar_wait(&s_mbar, mpar, kBarrierTimeoutNs);
        mpar ^= 1u;
        if (!ok) atomicCAS(&flags->err, DEVERR_NONE, DEVERR_TIMEOUT);  // the block returns after the next step's sum
      } else {
        __syncthreads();
      }

      // Streamed columns, a warp per two (q and q + kUrWarps, both >= cap): their
      // entries (-1: index >= lim) and old coefficients, then the residual rows
      // (zeros for -1) and e = r + x d.  The pass is bound by the latency of these
      // dependent loads, so the next pair's entries and coefficients are fetched
      // while this pair's rows arrive (4096 x 4096, 16 x 16, 512 atoms: 87 -> 44 ms a
      // sweep).
      struct Pair {
        int ea, eb;
        float xa, xb;
      };
      auto stream_meta = [&](int q, int lim) {
        Pair p;
        p.ea = (q < lim) ? __ldg(entries + first + q) : -1;
        p.eb = (q + kUrWarps < lim) ? __ldg(entries + first + q + kUrWarps) : -1;
        p.xa = (p.ea >= 0) ? __ldcg(coef + p.ea) : 0.0f;
        p.xb = (p.eb >= 0) ? __ldcg(coef + p.eb) : 0.0f;
        return p;
      };
      auto stream_cols = [&](const Pair& p, float (&e0)[NW], float (&e1)[NW]) {
        const float* ra = R + int64_t(p.ea >= 0 ? p.ea / L : 0) * n;
        const float* rb = R + int64_t(p.eb >= 0 ? p.eb / L : 0) * n;
#pragma unroll
        for (int k = 0; k < NW; ++k) {
          const int i = lane + 32 * k;
          e0[k] = (i < n && p.ea >= 0) ? __ldcg(ra + i) : 0.0f;
          e1[k] = (i < n && p.eb >= 0) ? __ldcg(rb + i) : 0.0f;
        }
      };
      auto stream_form = [&](const Pair& p, float (&e0)[NW], float (&e1)[NW]) {
#pragma unroll
        for (int k = 0; k < NW; ++k) {
          const int i = lane + 32 * k;
          if (i < n) {
            e0[k] = fmaf(p.xa, dold[i], e0[k]);
            e1[k] = fmaf(p.xb, dold[i], e1[k]);
          }
        }
      };

      // ---- power iteration ---------------------------------------------------
      float4 uo[KF];  // u in the registers of every warp: float4 lane + 32 k
#pragma unroll
      for (int k = 0; k < KF; ++k)
        uo[k] = (lane + 32 * k < F) ? dold4[lane + 32 * k] : make_float4(0.f, 0.f, 0.f, 0.f);
      int iters = 0;
      float dprev = 0.0f;  // the previous step's change
      for (int it = 0; it < kUrMaxIters; ++it) {
        // v_q = u . e_q (u is d_old in the first step)
        const float* const uc = it == 0 ? dold : u;
        if (it == 0) {
          for (int q0 = 0; q0 + warp * 8 < mres; q0 += kUrThreads / 4) {
            const int q = q0 + q_l;
            const bool in = q < mres;
            const float v = dot_u(q, in, true, in ? v_s[q] : 0.0f);
            if (in && (lane & 3) == 0) v_s[q] = v;
          }
        } else {
          for (int q0 = 0; q0 + warp * 8 < mcr; q0 += kUrThreads / 4) {
            const int q = q0 + q_l;
            const float v = dot_u(q, q < mcr, false, 0.0f);
            if (q < mcr && (lane & 3) == 0) v_s[q] = v;
          }
        }
        if (streamed) {  // columns beyond the capacity: a warp per two columns
          float wacc[NW];
#pragma unroll
          for (int k = 0; k < NW; ++k) wacc[k] = 0.0f;
          Pair next = stream_meta(cap + warp, mc);
          for (int q = cap + warp; q < mc; q += 2 * kUrWarps) {
            float e0[NW], e1[NW];
            const Pair p = next;
            stream_cols(p, e0, e1);
            next = stream_meta(q + 2 * kUrWarps, mc);
            stream_form(p, e0, e1);
            float d0 = 0.0f, d1 = 0.0f;
#pragma unroll
            for (int k = 0; k < NW; ++k) {
              const float w = lane + 32 * k < n ? uc[lane + 32 * k] : 0.0f;
              d0 = fmaf(w, e0[k], d0);
              d1 = fmaf(w, e1[k], d1);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
              d0 += __shfl_xor_sync(0xffffffffu, d0, o);
              d1 += __shfl_xor_sync(0xffffffffu, d1, o);
            }
#pragma unroll
            for (int k = 0; k < NW; ++k) wacc[k] = fmaf(d1, e1[k], fmaf(d0, e0[k], wacc[k]));
          }
#pragma unroll
          for (int k = 0; k < NW; ++k) {
            const int i = lane + 32 * k;
            if (i < n4) wstr[warp * n4 + i] = wacc[k];
          }
        }
        __syncthreads();
        // w = sum_q v_q e_q: the columns q = g, g + Gr, ... of group g in order
        if (lanes_w) {  // a warp per group, lanes over the features
          if (warp < Gr) {
            float acc[NW];
#pragma unroll
            for (int k = 0; k < NW; ++k) acc[k] = 0.0f;
#pragma unroll 2
            for (int q = warp; q < mcr; q += Gr) {
              const float v = v_s[q];
              const float* const eq = Es + size_t(q) * es + lane;
#pragma unroll
              for (int k = 0; k < NW; ++k)
                if (32 * k + lane < n4) acc[k] = fmaf(v, eq[32 * k], acc[k]);
            }
#pragma unroll
            for (int k = 0; k < NW; ++k)
              if (32 * k + lane < n4) wred[warp * n4 + 32 * k + lane] = acc[k];
          }
        } else if (s_q < Gr) {  // a float4 of a group per thread
          float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
          for (int q = s_q; q < mcr; q += Gr) {
            const float v = v_s[q];
            const float4 e = Es4[q * es4 + s_f];
            acc.x = fmaf(v, e.x, acc.x);
            acc.y = fmaf(v, e.y, acc.y);
            acc.z = fmaf(v, e.z, acc.z);
            acc.w = fmaf(v, e.w, acc.w);
          }
          reinterpret_cast<float4*>(wred)[s_q * F + s_f] = acc;
        }
        __syncthreads();
        lap(2);
        // the CTA's w, an element per thread; with several CTAs three elements
        // are packed into a word by the first of their threads
        const unsigned tag = (unsigned(j) << 8) + unsigned(it) + 1u;
        {
          uint4* const wp = words + (size_t(it & 1) * G + b) * W;
          for (int i0 = warp * 30; i0 < 3 * W; i0 += kUrWarps * 30) {
            const int i = i0 + lane;
            float s = 0.0f;
            if (lane < 30 && i < n4) {
              s = wred[i];
#pragma unroll 8
              for (int g = 1; g < Gr; ++g) s += wred[g * n4 + i];
              if (streamed)
#pragma unroll
                for (int w = 0; w < kUrWarps; ++w) s += wstr[w * n4 + i];
            }
            if (alone) {
              if (lane < 30 && i < n4) wsum[i] = s;
            } else {
              const float y = __shfl_down_sync(0xffffffffu, s, 1), z = __shfl_down_sync(0xffffffffu, s, 2);
              if (counted) {
                if (lane < 30 && i < n4) __stcg(raw + (size_t(it & 1) * G + b) * n4 + i, s);
              } else if (lane < 30 && lane % 3 == 0 && i / 3 < W) {
                st_word(wp + i / 3, s, y, z, tag);
              }
            }
          }
        }
        if (counted) {
          __syncthreads();
          if (tid == 0) red_release_add(iter_cnt + j, 1u);
        }
        if (it == 0 && prefetch) meta_rest(nm);
        if (counted) {
          // group g sums rows g, g + Gr, ... of float4 column f
          if (tid == 0) s_ok = ur_wait_count(iter_cnt + j, unsigned(it + 1) * unsigned(active), flags) ? 1 : 0;
          __syncthreads();
          if (!s_ok) return;
          const int g = s_q, f = s_f;
          if (g < Gr) {
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
            const float4* const base = reinterpret_cast<const float4*>(raw + size_t(it & 1) * G * n4) + f;
            constexpr int kB = 11;  // loads in flight
#pragma unroll 1
            for (int bb0 = g; bb0 < active; bb0 += Gr * kB) {
              float4 v[kB];
#pragma unroll
              for (int k = 0; k < kB; ++k) {
                const int bb = bb0 + k * Gr;
                v[k] = (bb < active) ? __ldcg(base + size_t(bb) * F) : make_float4(0.f, 0.f, 0.f, 0.f);
              }
#pragma unroll
              for (int k = 0; k < kB; ++k) {
                acc.x += v[k].x;
                acc.y += v[k].y;
                acc.z += v[k].z;
                acc.w += v[k].w;
              }
            }
            reinterpret_cast<float4*>(wred)[g * F + f] = acc;
          }
          __syncthreads();
          if (tid < n4) {
            float s = wred[tid];
#pragma unroll 4
            for (int g2 = 1; g2 < Gr; ++g2) s += wred[g2 * n4 + tid];
            wsum[tid] = s;
          }
        } else if (!alone) {
          // all-reduce: group g sums partials g, g + Gr, ... in ascending order,
          // a word per thread; its rows go where the streamed columns' were
          if (streamed) __syncthreads();
          const int gs = min(Gr, active);
          int g = x_g, f = x_f;
#pragma unroll 1
          while (g < gs) {
            const float4 a = ur_gather(words + (size_t(it & 1) * G + g) * W + f, size_t(Gr) * W,
                                       (active - g + Gr - 1) / Gr, tag, flags);
            ok = ok && a.w != 0.0f;
            float* const xr = xrow + g * n4 + 3 * f;
            xr[0] = a.x;
            if (3 * f + 1 < n4) xr[1] = a.y;
            if (3 * f + 2 < n4) xr[2] = a.z;
            f += kUrThreads;
            while (f >= W) {
              f -= W;
              ++g;
            }
          }
          __syncthreads();
          if (tid < n4) {
            float s = xrow[tid];
#pragma unroll 4
            for (int g = 1; g < gs; ++g) s += xrow[g * n4 + tid];
            wsum[tid] = s;
          }
        }
        if (__syncthreads_or(!ok)) return;
        lap(3);
        iters = it + 1;
        // every warp finishes the step: w, its norm, the new u, the change, the
        // stop decision (the same values in every warp of every CTA) and, when
        // stopping, the sign (u . d_old >= 0)
        float4 wv[KF];
        float s2 = 0.0f;
#pragma unroll
        for (int k = 0; k < KF; ++k) {
          const int f = lane + 32 * k;
          const float4 acc = f < F ? wsum4[f] : make_float4(0.f, 0.f, 0.f, 0.f);
          wv[k] = acc;
          s2 = fmaf(acc.x, acc.x, fmaf(acc.y, acc.y, fmaf(acc.z, acc.z, fmaf(acc.w, acc.w, s2))));
        }
        const float nrm2 = warp_sum(s2);
        bool stop;
        if (!(nrm2 > 0.0f)) {
          stop = true;  // E == 0: keep the old atom direction
        } else {
          const float inv = 1.0f / sqrtf(nrm2);
          float dm = 0.0f;
#pragma unroll
          for (int k = 0; k < KF; ++k) {
            const float4 o = uo[k];
            float4 un;
            un.x = wv[k].x * inv;
            un.y = wv[k].y * inv;
            un.z = wv[k].z * inv;
            un.w = wv[k].w * inv;
            dm = fmaxf(dm, fmaxf(fmaxf(fabsf(un.x - o.x), fabsf(un.y - o.y)),
                                 fmaxf(fabsf(un.z - o.z), fabsf(un.w - o.w))));
            uo[k] = un;
          }
          // never NaN nor negative (fmaxf), so its bits order as it does
          dm = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(dm)));
          // stop when the change is below the tolerance, or when the observed
          // contraction rho = dm / dprev puts the remaining distance to the
          // limit, about dm rho / (1 - rho), below it
          stop = dm < kUrTol;
          if (!stop && it > 0 && dprev > 0.0f && dm < 1e-3f) {
            const float rho = dm / dprev;
            stop = rho < 0.5f && dm * rho < kUrTol * (1.0f - rho);
          }
          dprev = dm;
        }
        if (stop) {
          float sd = 0.0f;
#pragma unroll
          for (int k = 0; k < KF; ++k) {
            const int f = lane + 32 * k;
            if (f < F) {
              const float4 a = uo[k], d = dold4[f];
              sd = fmaf(a.x, d.x, fmaf(a.y, d.y, fmaf(a.z, d.z, fmaf(a.w, d.w, sd))));
            }
          }
          sd = warp_sum(sd);
          if (sd < 0.0f)
#pragma unroll
            for (int k = 0; k < KF; ++k) uo[k] = make_float4(-uo[k].x, -uo[k].y, -uo[k].z, -uo[k].w);
        }
        if (warp == 0)
#pragma unroll
          for (int k = 0; k < KF; ++k)
            if (lane + 32 * k < F) {
              const int f = lane + 32 * k;
              u4[f] = uo[k];
              ut[f] = uo[k].x;
              ut[ft + f] = uo[k].y;
              ut[2 * ft + f] = uo[k].z;
              ut[3 * ft + f] = uo[k].w;
            }
        __syncthreads();
        lap(4);
        if (stop) break;
      }
      if (b == 0) {
        for (int i = tid; i < n; i += kUrThreads) __stcg(D + int64_t(j) * n + i, u[i]);
        if (tid == 0) {
          atomicAdd(&stats->power_iters, (unsigned long long)iters);
          atomicAdd(&stats->atoms_updated, 1ull);
        }
      }

      // ---- coefficients x = u . e (0 beyond the cap) and residual e - x u ----
      for (int q0 = 0; q0 + warp * 8 < mres; q0 += kUrThreads / 4) {
        const int q = q0 + q_l;
        const float x = dot_u(q, q < mcr, false, 0.0f);
        if (q < mres && (lane & 3) == 0) {
          v_s[q] = q < mc ? x : 0.0f;
          __stcg(coef + (q0 == 0 ? c_en : __ldg(entries + first + q)), q < mc ? x : 0.0f);
        }
      }
      if (m > cap) {  // streamed columns: a warp per two columns
        float ur[NW];
#pragma unroll
        for (int k = 0; k < NW; ++k) {
          const int i = lane + 32 * k;
          ur[k] = (i < n) ? u[i] : 0.0f;
        }
        Pair next = stream_meta(cap + warp, m);
        for (int q = cap + warp; q < m; q += 2 * kUrWarps) {
          float e0[NW], e1[NW];
          const Pair p = next;
          const int ea = p.ea, eb = p.eb;
          stream_cols(p, e0, e1);
          next = stream_meta(q + 2 * kUrWarps, m);
          stream_form(p, e0, e1);
          float x0 = 0.0f, x1 = 0.0f;
#pragma unroll
          for (int k = 0; k < NW; ++k) {
            x0 = fmaf(ur[k], e0[k], x0);
            x1 = fmaf(ur[k], e1[k], x1);
          }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            x0 += __shfl_xor_sync(0xffffffffu, x0, o);
            x1 += __shfl_xor_sync(0xffffffffu, x1, o);
          }
          if (q >= mc) x0 = 0.0f;
          if (q + kUrWarps >= mc) x1 = 0.0f;
          float* ra = R + int64_t(ea / L) * n;
          if (last == nullptr || __ldg(last + ea / L) != j) {
#pragma unroll
            for (int k = 0; k < NW; ++k) {
              const int i = lane + 32 * k;
              if (i < n) __stcg(ra + i, fmaf(-x0, ur[k], e0[k]));
            }
          }
          if (lane == 0) __stcg(coef + ea, x0);
          if (eb >= 0) {
            float* rb = R + int64_t(eb / L) * n;
            if (last == nullptr || __ldg(last + eb / L) != j) {
#pragma unroll
              for (int k = 0; k < NW; ++k) {
                const int i = lane + 32 * k;
                if (i < n) __stcg(rb + i, fmaf(-x1, ur[k], e1[k]));
              }
            }
            if (lane == 0) __stcg(coef + eb, x1);
          }
        }
      }
      if (prefetch) {  // the next atom's meta and old atom
        meta_store(nm, slot ^ 1, jn, tid);
        if (tid < n4) dbuf[(slot ^ 1) * n4 + tid] = nd;
      }
      __syncthreads();
      if (prefetch && tid < n4) ut[(tid & 3) * ft + (tid >> 2)] = nd;
      if (tma) {  // rows of 16-byte aligned float4, (row, float4) pairs over the threads
        int q = s_q, f = s_f;
#pragma unroll 2
        while (q < mres) {
          const int p = row_s[q];
          if (p >= 0) {
            const float x = v_s[q];
            const float4 e = Es4[q * es4 + f], w = u4[f];
            float4 r;
            r.x = fmaf(-x, w.x, e.x);
            r.y = fmaf(-x, w.y, e.y);
            r.z = fmaf(-x, w.z, e.z);
            r.w = fmaf(-x, w.w, e.w);
            __stcg(reinterpret_cast<float4*>(R + int64_t(p) * n) + f, r);
          }
          q += d_q;
          f += d_f;
          if (f >= F) {
            f -= F;
            ++q;
          }
        }
      } else {
        for (int q = warp; q < mres; q += kUrWarps) {
          const int p = row_s[q];
          if (p < 0) continue;
          const float x = v_s[q];
          float* const row = R + int64_t(p) * n;
          for (int i = lane; i < n; i += 32) __stcg(row + i, fmaf(-x, u[i], Es[size_t(q) * es + i]));
        }
      }
      fence_proxy_async_smem();  // generic accesses of Es before the next bulk copies into it
      __syncthreads();
      // nobody else waits for a CTA alone on this atom and the next one
      if (tid == 0 && (active > 1 || nact > 1)) red_release_add(done_cnt + j, 1u);
      lap(5);
      if (prefetch) slot ^= 1;
      meta_atom = prefetch ? jn : -1;
    }
  }
  if (timer)
    for (int k = 0; k < 8; ++k) atomicAdd(&stats->phase_ns[k], s_ph[k]);
}

template <int NW>
static void* ur_fn() {
  return reinterpret_cast<void*>(update_res_kernel<NW>);
}

static void* pick_update_res(int n) {
  switch ((n + 31) / 32) {
    case 1: return ur_fn<1>();
    case 2: return ur_fn<2>();
    case 3: return ur_fn<3>();
    case 4: return ur_fn<4>();
    case 5: return ur_fn<5>();
    case 6: return ur_fn<6>();
    case 7: return ur_fn<7>();
    case 8: return ur_fn<8>();
    case 9: return ur_fn<9>();
    case 10: return ur_fn<10>();
    case 11: return ur_fn<11>();
    case 12: return ur_fn<12>();
    case 13: return ur_fn<13>();
    case 14: return ur_fn<14>();
    case 15: return ur_fn<15>();
    case 16: return ur_fn<16>();
    default: return nullptr;
  }
}

bool update_res_supported(int n) { return n >= 1 && n <= 512 && update_res_capacity(n) >= 16; }

int update_res_grid_size(int n, int num_sms) {
  void* fn = pick_update_res(n);
  const int cap = update_res_capacity(n);
  if (!fn || cap < 16) return 0;
  const size_t smem = update_res_smem_bytes(n, cap);
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess) return 0;
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kUrThreads, smem) != cudaSuccess) return 0;
  if (per_sm < 1) return 0;
  return num_sms;  // one CTA per SM: co-resident by construction
}

// Zeroed by the launch: the tagged partials (two per CTA, by parity of the power
// step) and two counters per atom; then the plain partials.
static size_t ur_zeroed_bytes(int n, int grid, int K) {
  return (size_t(2) * grid * ur_words(n) + (K + 1) / 2) * sizeof(uint4);
}

size_t update_res_scratch_bytes(int n, int grid, int K) {
  return ur_zeroed_bytes(n, grid, K) + size_t(2) * grid * ur_n4(n) * sizeof(float);
}

cudaError_t launch_residual(const float* Y, int64_t N, int n, const float* D, int K, int L, const int32_t* idx,
                            const float* coef, float* R, int* last, int num_sms, cudaStream_t s) {
  const int64_t want = (N + 7) / 8;
  const int blocks = int(want < int64_t(num_sms) * 16 ? want : int64_t(num_sms) * 16);
  const int vec4 = ((n & 3) == 0 && (reinterpret_cast<uintptr_t>(Y) & 15) == 0 &&
                    (reinterpret_cast<uintptr_t>(D) & 15) == 0 && (reinterpret_cast<uintptr_t>(R) & 15) == 0)
                       ? 1
                       : 0;
  residual_kernel<<<blocks > 0 ? blocks : 1, 256, 0, s>>>(Y, N, n, D, K, L, idx, coef, R, last, vec4, nullptr,
                                                          nullptr);
  return cudaGetLastError();
}

cudaError_t launch_residual_list(const float* Y, int64_t N, int n, const float* D, int K, int L, const int32_t* idx,
                                 const float* coef, float* R, int* last, const int64_t* list,
                                 const unsigned long long* count, int num_sms, cudaStream_t s) {
  if (!list || !count) return cudaErrorInvalidValue;
  const int vec4 = ((n & 3) == 0 && (reinterpret_cast<uintptr_t>(Y) & 15) == 0 &&
                    (reinterpret_cast<uintptr_t>(D) & 15) == 0 && (reinterpret_cast<uintptr_t>(R) & 15) == 0)
                       ? 1
                       : 0;
  residual_kernel<<<num_sms * 2, 256, 0, s>>>(Y, N, n, D, K, L, idx, coef, R, last, vec4, list, count);
  return cudaGetLastError();
}

cudaError_t launch_update_batch(const UpdBatch& batch, GridBarrier* flags, DevStats* stats, int timers, int grid,
                                cudaStream_t s) {
  if (batch.ngroups < 1 || batch.ngroups > kUpdMaxGroups || grid < 1) return cudaErrorInvalidValue;
  int nmax = 0;
  for (int i = 0; i < batch.ngroups; ++i) {
    const UpdGroup& g = batch.g[i];
    if (g.ctas < 1 || g.cta_begin < 0 || g.cta_begin + g.ctas > grid) return cudaErrorInvalidValue;
    if (g.cap < 16 || g.cap > update_res_capacity(g.n)) return cudaErrorInvalidValue;
    nmax = g.n > nmax ? g.n : nmax;
  }
  void* fn = pick_update_res(nmax);
  if (!fn) return cudaErrorInvalidValue;
  size_t smem = 0;
  for (int i = 0; i < batch.ngroups; ++i) {
    const size_t b = update_res_smem_bytes(batch.g[i].n, batch.g[i].cap);
    smem = b > smem ? b : smem;
  }
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  if (e != cudaSuccess) return e;
  for (int i = 0; i < batch.ngroups; ++i) {
    const UpdGroup& g = batch.g[i];
    // the counters, and the words: no tag of an earlier sweep may be left
    e = cudaMemsetAsync(g.gw, 0, ur_zeroed_bytes(g.n, g.ctas, g.K), s);
    if (e != cudaSuccess) return e;
  }
  UpdBatch b = batch;
  void* args[] = {(void*)&b, (void*)&flags, (void*)&stats, (void*)&timers};
  return cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kUrThreads), args, smem, s);
}

}  // namespace ksvd
