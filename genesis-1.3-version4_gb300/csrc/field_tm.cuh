// The fused field step with the first right-hand side's stencil term in tensor memory
// (deposition and ADI of one slice in one CTA, FieldSolverADI.cpp:9-122; mixed form).
// Included by kernels_mixed.cu.
//
// As in k_field_fused_f the slice's system is solved in shared memory, S [ng][st]:
//   S = S1 = (I + c Dy) u    every column cut into segments of rows, one thread each, u
//                            straight from global memory; S1 is kept in tensor memory
//   S = S1 + src             deposition
//   S = Thomas_x(S)          rows, segments
//   u = Thomas_y(2 S - S1)   columns: the segments of the first phase, so that each thread
//                            finds its own S1
// What bounded k_field_fused_f was the sum of its phases' latencies (one CTA an SM: the
// slice's bulk load, the deposition's reads, the reread of u from L2 for the second
// right-hand side, the bulk store) and the shared-memory wavefronts of the solves. Here a
// persistent CTA takes slice after slice and prefetches the next one's field and particles
// into L2 while it solves; S1 costs no shared-memory or L2 traffic (tensor memory holds 64
// words a thread at 1024 threads: 32 rows of a column); and a solve reads and writes each
// row once (solve_window), without a barrier inside. The segments are solved as if the
// field were zero outside them, with the settled coefficients (cbet and cwet reach their
// limits within W rows): (I - i c D) is then the same convolution everywhere, whose response
// fades by kappa = -c cbet per row on both sides, so
//   x_k = x0_k + kappa^{k-b+1} l + kappa^{e-k} r
// with l and r the neighbours' x0 next to the segment, or at the grid's edges, where the
// field is zero one row outside, minus kappa times its own first or last x0 (the mirror
// image). The terms are kept for W rows, kappa^W below 2^-32 (the host's segment_warmup;
// every segment is longer than W). The columns' rows next to a segment's ends get them as
// they are written to u. Rows have an odd stride st, so that the row solve, whose lanes walk
// different rows, finds different banks on even grids too.
// Measured (after 20 steps, k_field_fused_f at its best CTA size before): 4096 slices x 8192
// particles, 151^2 1000 -> 630 us (3.4 TB/s of the algorithmic bytes; the DRAM traffic, part of
// the particles still being in L2, is 44 % of the copy bandwidth); 700 x 8192, 151^2 197 ->
// 128 us; 2000 x 4096, 117^2 253 -> 193 us; 700 x 8192, 128^2 336 -> 106 us. Of a slice's 46 thousand cycles the deposition takes 12, the column solve
// 10, the row solve 7, the last pass 7, S1 5, the rows' carries 3.

// Sixteen words (eight complex values) of this thread's tensor memory.
#define G4_TM_W(v, j) "r"(__float_as_uint(v[j].x)), "r"(__float_as_uint(v[j].y))
__device__ __forceinline__ void tm_put8(uint32_t a, const float2 *v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16};" ::"r"(a),
      G4_TM_W(v, 0), G4_TM_W(v, 1), G4_TM_W(v, 2), G4_TM_W(v, 3), G4_TM_W(v, 4), G4_TM_W(v, 5), G4_TM_W(v, 6),
      G4_TM_W(v, 7)
      : "memory");
}
#undef G4_TM_W
__device__ __forceinline__ void tm_get8(uint32_t a, float2 *v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];\n"
      "tcgen05.wait::ld.sync.aligned;\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(a)
      : "memory");
#pragma unroll
  for (int j = 0; j < 8; j++) v[j] = make_float2(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
}

// v + w x for complex w
__device__ __forceinline__ float2 add_cmulf(float2 v, float2 w, float2 x) {
  return make_float2(fmaf(w.x, x.x, fmaf(-w.y, x.y, v.x)), fmaf(w.x, x.y, fmaf(w.y, x.x, v.y)));
}

constexpr int kTmLook = 16;   // the longest look-ahead of the solves
constexpr int kTmChunk = 8;   // rows a window of the solves loads and delivers at a time
// 85 registers a thread hold the windows (1024 threads, 64 registers, spilled)
constexpr int kTmMaxThreads = 768;
struct TmShape {
  int threads, nseg, words, cols;  // words of tensor memory a thread, columns a CTA allocates
};
// The shape for CTAs of `threads`: as many segments as the threads and the warm-up allow,
// up to 8 (threads 0: none fits).
inline TmShape tm_shape(int ng, int threads, int W) {
  threads = std::min(threads, kTmMaxThreads);
  TmShape t{threads, std::min(std::min(threads / ng, 8), ng / (W + 1)), 0, 0};
  if (W < 1 || W > kTmLook + 1 || t.nseg < 2) return TmShape{0, 0, 0, 0};
  const int len = (ng + t.nseg - 1) / t.nseg, per = (threads / 32 + 3) / 4;  // warps a lane quarter
  t.words = (len + 7) / 8 * 16;
  int c = 32;
  while (c < per * t.words) c *= 2;
  if (c > 512) return TmShape{0, 0, 0, 0};
  t.cols = c;
  return t;
}
inline size_t tm_smem_bytes(int ng, int W, int threads) {
  return (((size_t)W + 1) / 2 * 2 + ((size_t)ng * (ng | 1) + 1) / 2 * 2) * sizeof(float2) +
         (size_t)(threads / 32 + 1) * kFieldSums * sizeof(double);
}

// The solve of rows [b, e) of a line, zeros outside, in one pass over it: the forward values d
// of a window of CH + LA rows stay in registers, and the back substitution runs over the
// window from zero, LA rows ahead of the CH rows it delivers (LA + 1 >= W: the part left out
// is below kappa^W). So a row is read once and
// written once, where a pass down and one up move it four times: the solves are bound by
// shared-memory wavefronts and issue. load(r, v) gives the right-hand sides of CH rows from
// r, zeros for rows >= e (every thread of a warp calls it together), emit(r, x) takes the
// solution of row r < e.
template <int LA, class LD, class EM>
__device__ __forceinline__ void solve_window(int b, int e, int nchunk, float cs, float2 cb, float2 kap, LD load,
                                             EM emit) {
  constexpr int CH = kTmChunk;
  float2 d[CH + LA], last = make_float2(0.f, 0.f);
  auto forward = [&](int r, float2 *o) {
    load(r, o);
#pragma unroll
    for (int j = 0; j < CH; j++) {
      last = cmulf(sub_imulf(o[j], -cs, last), cb);
      o[j] = last;
    }
  };
#pragma unroll
  for (int p = 0; p < LA; p += CH) forward(b + p, d + p);
#pragma unroll 1
  for (int q = 0; q < nchunk; q++) {
    const int r0 = b + q * CH;
    forward(r0 + LA, d + LA);
    float2 x = d[CH + LA - 1];
#pragma unroll
    for (int j = CH + LA - 2; j >= 0; j--) {
      x = add_cmulf(d[j], kap, x);
      if (j < CH && r0 + j < e) emit(r0 + j, x);
    }
#pragma unroll
    for (int j = 0; j < LA; j++) d[j] = d[CH + j];
  }
}

// Adds the carries over the ends of rows [b, e) of a line
__device__ __forceinline__ void add_carries(float2 *L, const float2 *PW, int b, int e, int W, float2 lc, float2 rc) {
  for (int j = 0; j < W; j++) {
    L[b + j] = add_cmulf(L[b + j], PW[j], lc);
    L[e - 1 - j] = add_cmulf(L[e - 1 - j], PW[j], rc);
  }
}

// Prefetches [p, p + bytes) of an array into L2, rounded inwards to 16 bytes.
__device__ __forceinline__ void l2_prefetch(const void *p, size_t bytes) {
  const uintptr_t a = (reinterpret_cast<uintptr_t>(p) + 15) & ~(uintptr_t)15;
  const uintptr_t z = (reinterpret_cast<uintptr_t>(p) + bytes) & ~(uintptr_t)15;
  if (z > a)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"((uint32_t)(z - a)) : "memory");
}

// Sums of v[0..8) over a warp: lane 4 k holds the sum of v[k], as a pair hi + lo (each step
// halves the values a lane carries; the additions' errors go to lo).
__device__ __forceinline__ float2 add_pairs(float2 a, float2 b) {
  const float t = a.x + b.x, bp = t - a.x;
  return make_float2(t, a.y + b.y + ((a.x - (t - bp)) + (b.x - bp)));
}
__device__ __forceinline__ float2 shfl_xor2(float2 v, int o) {
  return make_float2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}
__device__ __forceinline__ float2 warp_sums8(float2 (&v)[8]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 16, n = 4; o >= 4; o >>= 1, n >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (j < n) {
        const float2 send = up ? v[j] : v[j + n], keep = up ? v[j + n] : v[j];
        v[j] = add_pairs(keep, shfl_xor2(send, o));
      }
  }
  float2 s = v[0];
  s = add_pairs(s, shfl_xor2(s, 2));
  return add_pairs(s, shfl_xor2(s, 1));
}

// S1 = (I + c Dy) u of rows [b, e) of a column: into S (rows of st) and, eight rows at a
// time, into this thread's tensor memory. u and S point at the band's first row; `above`: the
// grid goes on above row b; `below`: rows of the grid from the band's first on. Rows outside
// the grid are zeros, which gives the one-sided differences at its edges.
__device__ __forceinline__ void tm_stencil_cols(const float2 *u, float2 *S, uint32_t tm, int ng, int st, int line,
                                                bool act, int b, int e, int nq, bool above, int below, float cs) {
  const float2 zero = make_float2(0.f, 0.f);
  float2 prev = above ? u[(b - 1) * ng + line] : zero;
  float2 cur = act ? u[b * ng + line] : zero;
#pragma unroll 1
  for (int q = 0; q < nq; q++) {
    float2 v[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int r = b + 8 * q + j;
      v[j] = r < e && r + 1 < below ? u[(r + 1) * ng + line] : zero;
    }
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const float2 nx = v[j];
      v[j] = stencil(cs, cur, make_float2(nx.x - 2.f * cur.x + prev.x, nx.y - 2.f * cur.y + prev.y));
      prev = cur;
      cur = nx;
      const int r = b + 8 * q + j;
      if (r < e) S[r * st + line] = v[j];
    }
    __syncwarp();
    tm_put8(tm + 16 * q, v);
  }
}

// The column solve of the second right-hand side 2 u' - S1 in place, zeros outside [b, e).
template <int LA>
__device__ __forceinline__ void tm_solve_cols(float2 *L, uint32_t tm, int st, int b, int e, int nq, int nchunk,
                                              float cs, float2 cb, float2 kap) {
  const float2 zero = make_float2(0.f, 0.f);
  solve_window<LA>(
      b, e, nchunk, cs, cb, kap,
      [&](int r, float2 *v) {
        const int q = (r - b) >> 3;
        if (q < nq) {
          float2 s1[8];
#pragma unroll
          for (int j = 0; j < 8; j++) v[j] = r + j < e ? L[(r + j) * st] : zero;
          __syncwarp();
          tm_get8(tm + 16 * q, s1);
#pragma unroll
          for (int j = 0; j < 8; j++)
            v[j] = r + j < e ? make_float2(2.f * v[j].x - s1[j].x, 2.f * v[j].y - s1[j].y) : zero;
        } else {
#pragma unroll
          for (int j = 0; j < 8; j++) v[j] = zero;
        }
      },
      [&](int r, float2 x) { L[r * st] = x; });
}

// Writes rows [b, e) of a column with the carries lc and rc over its ends to u, and sums the
// field record's terms (global row of row 0: r0), compensated like k_diag_field_f's, so that a
// record formed in the step is the one formed after it: plain FP32 sums here and over the warp
// erred by 3e-8 to 7e-8 of the sums of a 151^2 field, these by 2e-9 (a step with its record:
// 300 slices of 255^2 270 -> 283 us, 4096 of 151^2 1332 -> 1357, one 23.3 -> 24.2).
template <bool REC>
__device__ __forceinline__ void tm_write_cols(float2 *u, const float2 *L, const float2 *PW, int ng, int st, int line,
                                              int b, int e, int W, float2 lc, float2 rc, int r0, float2 (&f)[8]) {
  const int lo = b + W, hi = e - W;  // [lo, hi): no carry
  const float shift = -0.5f * (float)(ng - 1);
  float dy = (float)(r0 + b) + shift;
  KahanF2 su, sw;  // the field itself; w and dy w
  KahanF s2;       // dy^2 w
  auto put = [&](int r, float2 x) {
    u[r * ng + line] = x;
    if constexpr (REC) {
      const float w = fmaf(x.x, x.x, x.y * x.y), t = dy * w;
      sw.add(make_float2(w, t));
      s2.add(dy * t);
      su.add(x);
      dy += 1.f;
    }
  };
  const int mid = min(lo, e);
#pragma unroll 4
  for (int r = b; r < mid; r++) {
    float2 x = add_cmulf(L[r * st], PW[r - b], lc);
    if (r >= hi) x = add_cmulf(x, PW[e - 1 - r], rc);
    put(r, x);
  }
#pragma unroll 4
  for (int r = mid; r < hi; r++) put(r, L[r * st]);
#pragma unroll 4
  for (int r = max(mid, hi); r < e; r++) put(r, add_cmulf(L[r * st], PW[e - 1 - r], rc));
  if constexpr (REC) {
    const float dx = (float)line + shift;
    auto times_dx = [&](float2 v) {
      const float h = dx * v.x;
      return make_float2(h, fmaf(dx, v.y, fmaf(dx, v.x, -h)));
    };
    f[0] = make_float2(sw.s.x, -sw.c.x);
    f[1] = times_dx(f[0]);
    f[2] = times_dx(f[1]);
    f[3] = make_float2(sw.s.y, -sw.c.y);
    f[4] = make_float2(s2.s, -s2.c);
    f[5] = make_float2(su.s.x, -su.c.x);
    f[6] = make_float2(su.s.y, -su.c.y);
    f[7] = make_float2(0.f, 0.f);
  }
}

// The CTA's totals of the threads' record terms: emit(q, pair) from the last warp, which
// folds the warps' pairs, four lanes a value, while the others go on. One barrier.
template <class EM>
__device__ __forceinline__ void tm_fold_record(float2 (&f)[8], float2 *red, EM emit) {
  const int tid = threadIdx.x, warp = tid >> 5;
  const float2 v = warp_sums8(f);
  if ((tid & 3) == 0 && (tid & 31) < 4 * kFieldSums) red[warp * kFieldSums + ((tid & 31) >> 2)] = v;
  __syncthreads();
  if (warp == (int)(blockDim.x >> 5) - 1) {
    const int k2 = (tid & 31) >> 2;
    float2 t = make_float2(0.f, 0.f);
    if (k2 < kFieldSums)
      for (int w = tid & 3; w < (int)(blockDim.x >> 5); w += 4) t = add_pairs(t, red[w * kFieldSums + k2]);
    t = add_pairs(t, shfl_xor2(t, 1));
    t = add_pairs(t, shfl_xor2(t, 2));
    if ((tid & 3) == 0 && k2 < kFieldSums) emit(k2, t);
  }
}

// REC: the field record of every slice (k_diag_field_f's sums) is formed too.
template <int LA, bool REC>
__global__ void __launch_bounds__(kTmMaxThreads, 1)
    k_field_tm_f(StepConstF sc, int k, PtrsF p, float2 *__restrict__ field, const float2 *__restrict__ coef,
                 const float2 *__restrict__ pows, int ns, int np, int ng, int deposit, int nseg, int W, int words,
                 int cols, double *dfield) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint32_t tm_base;
  const int tid = threadIdx.x, warp = tid >> 5, st = ng | 1;
  const FieldStepF &fs = sc.f[k];
  float2 *PW = reinterpret_cast<float2 *>(smem_raw);  // kappa^{j+1}
  float2 *S = PW + (W + 1) / 2 * 2;
  float2 *red = S + (ng * st + 1) / 2 * 2;  // [warp][kFieldSums]
  if (warp == 0) {
    __syncwarp();
    const uint32_t sadr = (uint32_t)__cvta_generic_to_shared(&tm_base);
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sadr), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  for (int t = tid; t < W; t += blockDim.x) PW[t] = pows[t];
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tm = tm_base + ((uint32_t)(warp & 3) << 21) + (uint32_t)((warp >> 2) * words);
  chain_next();
  chain_wait();

  // line (a column in the column phases, a row in the row solve) and segment of the thread
  const int line = tid % ng, seg = tid / ng;
  const bool act = seg < nseg;
  const int b = act ? seg * ng / nseg : 0, e = act ? (seg + 1) * ng / nseg : 0;
  const bool left = act && seg > 0, right = act && seg + 1 < nseg;
  const int nq = words >> 4;  // batches of eight rows
  const int nchunk = ((ng + nseg - 1) / nseg + kTmChunk - 1) / kTmChunk;
  const float cs = fs.cstep;
  const float2 cb = coef[2 * ng - 1], kap = PW[0], zero = make_float2(0.f, 0.f);
  // the part of a segment's solution that reaches it over its ends: its neighbour's at the
  // end, times kappa per row; at the grid's edges minus the mirror image of its own (the
  // field is zero one row outside)
  auto carry = [&](bool inner, float2 other, float2 own) { return inner ? other : cmulf(make_float2(-kap.x, -kap.y), own); };

#pragma unroll 1
  for (int is = blockIdx.x; is < ns; is += gridDim.x) {
    const int i = ring_slot(is, fs.first, ns);
    float2 *u = field + (size_t)i * ng * ng;
    // the first particles' loads in flight while S1 is formed (the vector path: full slices
    // of a multiple of 4 particles)
    const size_t base = (size_t)is * np;
    const bool vec = deposit && (np & 3) == 0 && !p.count;
    Quad quad{};
    if (vec && tid < (np >> 2)) quad = load_quad(p, base, tid);
    tm_stencil_cols(u, S, tm, ng, st, line, act, b, e, nq, left, ng, cs);
    __syncwarp();
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    __syncthreads();
    if (deposit) {  // S = S1 + src
      if (vec)
        deposit_quads(sc, fs, p, S, is, np, Grid(ng, st), quad);
      else
        deposit_smem(sc, fs, p, S, is, np, Grid(ng, st));
      __syncthreads();
    }
    // the next slice's field and particles on their way to L2 while this one is solved
    if (tid < 5 && is + (int)gridDim.x < ns) {
      const int nx = is + gridDim.x;
      const size_t o = (size_t)nx * np;
      const size_t n = p.count ? min(p.count[nx], np) : np;
      if (tid == 0) l2_prefetch(field + (size_t)ring_slot(nx, fs.first, ns) * ng * ng, (size_t)ng * ng * 8);
      if (deposit && tid == 1) l2_prefetch(p.x + o, n * 4);
      if (deposit && tid == 2) l2_prefetch(p.y + o, n * 4);
      if (deposit && tid == 3) l2_prefetch(p.dg + o, n * 4);
      if (deposit && tid == 4) l2_prefetch(p.theta + o, n * 8);
    }
    // rows: u', zero carries, then the neighbours'
    {
      float2 *L = S + line * st;
      solve_window<LA>(
          b, e, nchunk, cs, cb, kap,
          [&](int r, float2 *v) {
#pragma unroll
            for (int j = 0; j < kTmChunk; j++) v[j] = r + j < e ? L[r + j] : zero;
          },
          [&](int r, float2 x) { L[r] = x; });
      __syncthreads();
      float2 lc = zero, rc = zero;
      if (act) {
        lc = carry(left, left ? L[b - 1] : zero, L[b]);
        rc = carry(right, right ? L[e] : zero, L[e - 1]);
      }
      __syncthreads();
      if (act) add_carries(L, PW, b, e, W, lc, rc);
    }
    __syncthreads();
    // columns: the second right-hand side 2 u' - S1, solved, then written with the
    // neighbours' carries (writing the rows without carries from the solve itself: 631 against
    // 640 us for 4096 slices of 151^2, 257 against 250 us for 2000 of 117^2)
    float2 *L = S + line;
    tm_solve_cols<LA>(L, tm, st, b, e, nq, nchunk, cs, cb, kap);
    __syncthreads();
    float2 f[8];
    {
      float2 lc = zero, rc = zero;
      if (act) {
        lc = carry(left, left ? L[(b - 1) * st] : zero, L[b * st]);
        rc = carry(right, right ? L[e * st] : zero, L[(e - 1) * st]);
      }
      tm_write_cols<REC>(u, L, PW, ng, st, line, b, e, W, lc, rc, 0, f);
    }
    if constexpr (REC) {
      double *o = dfield + (size_t)i * (kFieldSums + 2);
      if (line == ng / 2 && b <= ng / 2 && ng / 2 < e) {  // the value on the axis
        const float2 v = u[(ng / 2) * ng + ng / 2];
        o[7] = v.x;
        o[8] = v.y;
      }
      tm_fold_record(f, red, [&](int q, float2 t) { o[q] = (double)t.x + (double)t.y; });
    } else {
      __syncthreads();
    }
  }
  __syncwarp();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tm_base), "r"(cols) : "memory");
}

// ---- the same step with a slice's rows split between the CTAs of a cluster ---------------
//
// For slices that do not fit one CTA's shared memory, and for windows of so few slices that
// one CTA a slice leaves most SMs idle. CTA q of CL holds rows [q ng / CL, (q + 1) ng / CL) of
// the slice, and the phases are those of k_field_tm_f on this band:
//  * the column segments end at the band's rows; a segment next to the band's edge finds the
//    neighbour's row there in its shared memory (one row of the band above and one of the
//    band below is all that crosses), and the rows next to the band's that S1 needs in
//    global memory, which nobody writes before every CTA has passed a cluster barrier;
//  * every CTA reads all the slice's particles and deposits into its own rows (adding to a
//    peer's shared memory instead took 2.8 times as long as one CTA's whole deposition; a
//    list of the particles with a row in the band, made first, gained nothing: what the
//    deposition of a band takes is the latency of its atomics, not the lanes left idle);
//  * rows are solved within the CTA, in more segments the fewer rows it has.
// One slice a cluster: the hardware hands out the next, whose field and particles are
// prefetched into L2. Two CTAs of clusters never share an SM (kClusterMinSmem): the second
// would wait for tensor memory while its peers wait for it, and the first's peers likewise.
// Measured against k_field_band_f and k_field_tm_f: at field_cluster (kernels_mixed.cu). Of a band's
// 63 thousand cycles (255^2, CL 3) S1 takes 13, the deposition 5 to 19 (the middle band holds the
// beam), the columns 11, the rows 10, the last pass 7; of the 32 of 151^2 with CL 4 the deposition
// up to 10, S1, rows and columns 4 to 6 each.
constexpr size_t kClusterMinSmem = 116u * 1024u;
constexpr int kMaxCluster = 8;
struct ClShape {
  int cl, threads, nseg, words, cols;
  size_t smem;
};
// The shape for clusters of cl CTAs (cl 0: it does not fit). Every segment is longer than W.
inline ClShape cl_shape(int ng, int W, int cl) {
  const int nmin = ng / cl, nmax = (ng + cl - 1) / cl;
  const ClShape none{0, 0, 0, 0, 0, 0};
  if (W < 1 || W > kTmLook + 1 || nmin < W + 1 || ng > kTmMaxThreads) return none;
  ClShape t{cl, 0, std::max(1, std::min(std::min(kTmMaxThreads / ng, 8), nmin / (W + 1))), 0, 32, 0};
  // as many threads as the tensor memory has words for
  for (int need = 0;; t.nseg--) {
    if (t.nseg < 1) return none;
    const int len = (nmax + t.nseg - 1) / t.nseg, least = (ng * t.nseg + 31) / 32 * 32;
    t.words = (len + 7) / 8 * 16;
    t.threads = kTmMaxThreads;
    auto fits = [&] { return (need = (t.threads / 32 + 3) / 4 * t.words) <= 512; };
    while (!fits() && t.threads > least) t.threads -= 32;
    if (t.threads < least || need > 512) continue;
    while (t.cols < need) t.cols *= 2;
    break;
  }
  t.smem = (((size_t)W + 1) / 2 * 2 + ((size_t)nmax * (ng | 1) + 1) / 2 * 2) * sizeof(float2) +
           (size_t)(t.threads / 32 + 1 + kMaxCluster) * kFieldSums * sizeof(double);
  if (t.smem > 227u * 1024u - 16) return none;
  t.smem = std::max(t.smem, kClusterMinSmem);
  return t;
}

template <int LA, bool REC>
__global__ void __launch_bounds__(kTmMaxThreads, 1)
    k_field_cl_f(StepConstF sc, int k, PtrsF p, float2 *__restrict__ field, const float2 *__restrict__ coef,
                 const float2 *__restrict__ pows, int ns, int np, int ng, int deposit, int nseg, int W, int words,
                 int cols, int ahead, double *dfield) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint32_t tm_base;
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int CL = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int tid = threadIdx.x, warp = tid >> 5, st = ng | 1;
  const FieldStepF &fs = sc.f[k];
  const int r0 = rank * ng / CL, nrow = (rank + 1) * ng / CL - r0, nmax = (ng + CL - 1) / CL;
  float2 *PW = reinterpret_cast<float2 *>(smem_raw);  // kappa^{j+1}
  float2 *S = PW + (W + 1) / 2 * 2;
  float2 *red = S + (nmax * st + 1) / 2 * 2;  // [warp][kFieldSums]
  float2 *parts = red + (size_t)(blockDim.x / 32 + 1) * kFieldSums;  // [CTA][kFieldSums], used in CTA 0
  if (warp == 0) {
    __syncwarp();
    const uint32_t sadr = (uint32_t)__cvta_generic_to_shared(&tm_base);
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sadr), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  for (int t = tid; t < W; t += blockDim.x) PW[t] = pows[t];
  const int is = blockIdx.x / CL, i = ring_slot(is, fs.first, ns);
  float2 *u = field + (size_t)i * ng * ng + (size_t)r0 * ng;  // the band
  const size_t base = (size_t)is * np;
  const bool vec = deposit && (np & 3) == 0 && !p.count;
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tm = tm_base + ((uint32_t)(warp & 3) << 21) + (uint32_t)((warp >> 2) * words);
  chain_next();
  chain_wait();
  // the first particles' loads in flight while S1 is formed
  Quad quad{};
  if (vec && tid < (np >> 2)) quad = load_quad(p, base, tid);

  // column and segment of the thread
  const int line = tid % ng, seg = tid / ng;
  const bool act = seg < nseg;
  const int b = act ? seg * nrow / nseg : 0, e = act ? (seg + 1) * nrow / nseg : 0;
  const bool left = act && r0 + b > 0, right = act && r0 + e < ng;
  const int nq = words >> 4;  // batches of eight rows
  const float cs = fs.cstep;
  const float2 cb = coef[2 * ng - 1], kap = PW[0], zero = make_float2(0.f, 0.f);
  auto carry = [&](bool inner, float2 other, float2 own) { return inner ? other : cmulf(make_float2(-kap.x, -kap.y), own); };

  const bool cols_on = __any_sync(0xffffffffu, act);  // warps without a column have nothing to issue
  if (cols_on) {
    tm_stencil_cols(u, S, tm, ng, st, line, act, b, e, nq, left, ng - r0, cs);
    __syncwarp();
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  }
  __syncthreads();
  if (deposit) {
    const Band g(ng, st, r0, nrow);
    if (vec)
      deposit_quads(sc, fs, p, S, is, np, g, quad);
    else
      deposit_smem(sc, fs, p, S, is, np, g);
    __syncthreads();
  }
  // a later slice's field and particles on their way to L2
  if (rank == 0 && tid < 5 && is + ahead < ns) {
    const int nx = is + ahead;
    const size_t o = (size_t)nx * np;
    const size_t n = p.count ? min(p.count[nx], np) : np;
    if (tid == 0) l2_prefetch(field + (size_t)ring_slot(nx, fs.first, ns) * ng * ng, (size_t)ng * ng * 8);
    if (deposit && tid == 1) l2_prefetch(p.x + o, n * 4);
    if (deposit && tid == 2) l2_prefetch(p.y + o, n * 4);
    if (deposit && tid == 3) l2_prefetch(p.dg + o, n * 4);
    if (deposit && tid == 4) l2_prefetch(p.theta + o, n * 8);
  }
  {  // the band's rows
    const int nsr = min((int)blockDim.x / nrow, ng / (W + 1));
    const int row = tid % nrow, sr = tid / nrow;
    const bool on = sr < nsr;
    const int rb = on ? sr * ng / nsr : 0, re = on ? (sr + 1) * ng / nsr : 0;
    float2 *L = S + row * st;
    if (__any_sync(0xffffffffu, on)) solve_window<LA>(
        rb, re, ((ng + nsr - 1) / nsr + kTmChunk - 1) / kTmChunk, cs, cb, kap,
        [&](int r, float2 *v) {
#pragma unroll
          for (int j = 0; j < kTmChunk; j++) v[j] = r + j < re ? L[r + j] : zero;
        },
        [&](int r, float2 x) { L[r] = x; });
    __syncthreads();
    float2 lc = zero, rc = zero;
    if (on) {
      const bool hl = sr > 0, hr = sr + 1 < nsr;
      lc = carry(hl, hl ? L[rb - 1] : zero, L[rb]);
      rc = carry(hr, hr ? L[re] : zero, L[re - 1]);
    }
    __syncthreads();
    if (on) add_carries(L, PW, rb, re, W, lc, rc);
  }
  __syncthreads();
  float2 *L = S + line;
  if (cols_on) tm_solve_cols<LA>(L, tm, st, b, e, nq, ((nmax + nseg - 1) / nseg + kTmChunk - 1) / kTmChunk, cs, cb, kap);
  __syncwarp();
  cl.sync();  // the neighbours' edge rows are solved, and nobody reads u any more
  float2 f[8];
  {
    float2 lc = zero, rc = zero;
    if (act) {
      float2 above = zero, below = zero;
      if (left) {
        const int hi = (rank - 1) * ng / CL;  // first row of the band above
        above = b > 0 ? L[(b - 1) * st] : cl.map_shared_rank(S, rank - 1)[(r0 - 1 - hi) * st + line];
      }
      if (right) below = e < nrow ? L[e * st] : cl.map_shared_rank(S, rank + 1)[line];
      lc = carry(left, above, L[b * st]);
      rc = carry(right, below, L[(e - 1) * st]);
    }
    // the peers' rows are read: the last barrier, which keeps a CTA's shared memory until then, does
    // not wait for the field's writes (with the record it also brings the parts to CTA 0, below)
    if constexpr (!REC) {
      __syncwarp();  // the carries above and the rows below part a warp's lanes
      asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    }
    tm_write_cols<REC>(u, L, PW, ng, st, line, b, e, W, lc, rc, r0, f);
  }
  if constexpr (REC) {
    double *o = dfield + (size_t)i * (kFieldSums + 2);
    const int mid = ng / 2 - r0;
    if (line == ng / 2 && b <= mid && mid < e) {  // the value on the axis
      const float2 v = u[mid * ng + line];
      o[7] = v.x;
      o[8] = v.y;
    }
    float2 *to = cl.map_shared_rank(parts, 0) + rank * kFieldSums;
    tm_fold_record(f, red, [&](int q, float2 t) { to[q] = t; });
  }
  __syncwarp();
  if constexpr (!REC) {
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  } else {
    cl.sync();
    if (rank == 0 && tid < kFieldSums) {
      float2 t = parts[tid];
      for (int q = 1; q < CL; q++) t = add_pairs(t, parts[q * kFieldSums + tid]);
      dfield[(size_t)i * (kFieldSums + 2) + tid] = (double)t.x + (double)t.y;
    }
  }
  __syncwarp();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tm_base), "r"(cols) : "memory");
}
