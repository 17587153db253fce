// FP64 ADI half steps on tiles of whole lines in shared memory (FieldSolverADI::ADI,
// src/Core/FieldSolverADI.cpp:60-122). Included by kernels_plain.cu after its complex
// helpers.
//
//   k_adi_rows  one CTA per (slice, band of L rows): S1 = u + i c Dy u, then S1 + src
//               solved along the rows into tmp; S1 replaces src;
//   k_adi_cols  one CTA per (slice, band of L columns): the second right-hand side,
//               solved along the columns into the field.
//
// The second right-hand side (src + u') + i c Dx u' is 2 u' - S1, because u' solves
// (I - i c Dx) u' = S1 + src: two FP64 instructions a cell instead of eight (the stencil
// and the source's addition), and u' and S1 are read once each.
namespace adi64 {

// The coefficients of one solve in shared memory: cbet and cwet settle to a constant
// after the first elements (their distance from it falls by kappa^2 per element), so the
// first nco entries and that constant serve a whole line; with nco = ng (no segments)
// they are the reference's tables. pw[j] = kappa^{j+1}, lw[j] = kappa^{j+1} / (1 - kappa^2).
struct Lines {
  C2 *cbet, *cwet, *pw, *lw;
  C2 *edge_d, *edge_x;  // [nseg][nline]
  C2 *T;
};

// Shared memory of a CTA: the tables, the segments' carries, the tile.
inline size_t lines_bytes(int nline, int stride, int nseg, int nco, int W) {
  return sizeof(double2) * (2 * (size_t)nco + 2 * (size_t)W + 2 * (size_t)nseg * nline + (size_t)stride);
}
__device__ __forceinline__ Lines lines_setup(unsigned char *smem, int nline, int nseg, int nco, int W, int ng,
                                             const Coef &cf) {
  Lines s;
  s.cbet = reinterpret_cast<C2 *>(smem);
  s.cwet = s.cbet + nco;
  s.pw = s.cwet + nco;
  s.lw = s.pw + W;
  s.edge_d = s.lw + W;
  s.edge_x = s.edge_d + nseg * nline;
  s.T = s.edge_x + nseg * nline;
  for (int t = threadIdx.x; t < nco; t += blockDim.x) {
    s.cbet[t] = ld(cf.cbet + t);
    s.cwet[t] = ld(cf.cwet + min(t + 1, ng - 1));  // cwet[t + 1], the back substitution's
  }
  for (int t = threadIdx.x; t < W; t += blockDim.x) {
    s.pw[t] = ld(cf.pw + t);
    s.lw[t] = ld(cf.pw + kSegPow + t);
  }
  return s;
}

__device__ __forceinline__ bool finite(C2 v) {
  return (__double2hiint(v.x) & 0x7ff00000) != 0x7ff00000 && (__double2hiint(v.y) & 0x7ff00000) != 0x7ff00000;
}

// Solves (I - i c D) x = r in place on the nline lines of the tile (element k of line l
// at T[l * lstride + k * estride]), nseg threads per line. The Thomas recurrences
// (tridagx / tridagy, FieldSolverADI.cpp:94-122)
//   d_k = (r_k - c_k d_{k-1}) cbet_k,   x_k = d_k - cwet_{k+1} x_{k+1}
// are linear in their carries, and a carry fades by kappa = -c cbet = -cwet per element:
// each segment [b, e) of at least W elements (kappa^W below 2^-62: the host's
// segment_warmup) runs both from zero carries, giving x0, and then
//   x_k = x0_k + D kappa^{k-b+1} / (1 - kappa^2) + kappa^{e-k} x_e
// with D the last d of the segment before (its own zero start is forgotten there) and x_e
// the first x of the segment after. Only the W elements next to a segment's ends need the
// terms; the CTA's threads share them out. With nseg = 1 the sweeps are the reference's.
// A value that is not finite runs through a whole line in the reference's sweeps, and so it
// does here (`bad`, by the barrier that is there anyway).
// Why segments: the FP64 pipe takes 64 cycles for a warp's instruction, so one thread per
// line is a chain of 10 ng of them, and a window of few slices leaves most SMs idle.
// Every thread calls it, after a barrier; a barrier has passed when it returns.
__device__ __forceinline__ void solve_lines(const Lines &s, int nline, int lstride, int estride, int ng, int nseg,
                                            int nco, int W, double c) {
  const int tid = threadIdx.x;
  const int line = tid % nline, seg = tid / nline;
  const int b = seg * ng / nseg, e = (seg + 1) * ng / nseg;
  bool bad = false;
  if (seg < nseg) {
    C2 *L = s.T + (size_t)line * lstride;
    // one loop for all segments (the tables' last entry is their constant): lanes of
    // different segments stay together, and a warp's FP64 instruction costs the same for
    // one lane as for 32
    C2 d = {0, 0};
    for (int k = b; k < e; k++) {
      d = cmul_fma(add_imul(L[k * estride], c, d), s.cbet[min(k, nco - 1)]);
      L[k * estride] = d;
    }
    s.edge_d[seg * nline + line] = d;
    // x_{e-1} = d_{e-1}, what the forward sweep ended with
    C2 x = d;
    for (int k = e - 2; k >= b; k--) {
      x = sub_cmul(L[k * estride], s.cwet[min(k, nco - 1)], x);
      L[k * estride] = x;
    }
    s.edge_x[seg * nline + line] = x;
    bad = !finite(x);
  }
  if (__syncthreads_or(bad)) {
    if (seg < nseg) {
      bad = false;
      for (int q = 0; q < nseg; q++) bad = bad || !finite(s.edge_x[q * nline + line]);
      const double nan = __longlong_as_double(0x7ff8000000000000LL);
      if (bad)
        for (int k = b; k < e; k++) s.T[(size_t)line * lstride + k * estride] = C2{nan, nan};
    }
    __syncthreads();
  }
  if (nseg == 1) return;
  const int ntask = (nseg - 1) * W * nline;
  for (int t = tid; t < ntask; t += blockDim.x) {
    const int l = t % nline, q = t / nline, j = q % W, g = q / W + 1;  // segment g's left end
    C2 *p = s.T + (size_t)l * lstride + (g * ng / nseg + j) * estride;
    const C2 a = s.lw[j], v = sub_cmul(*p, C2{-a.x, -a.y}, s.edge_d[(g - 1) * nline + l]);
    *p = v;
    if (j == 0) s.edge_x[g * nline + l] = v;
  }
  __syncthreads();
  for (int t = tid; t < ntask; t += blockDim.x) {
    const int l = t % nline, q = t / nline, j = q % W, g = q / W;  // segment g's right end
    C2 *p = s.T + (size_t)l * lstride + ((g + 1) * ng / nseg - 1 - j) * estride;
    const C2 a = s.pw[j];
    *p = sub_cmul(*p, C2{-a.x, -a.y}, s.edge_x[(g + 1) * nline + l]);
  }
  __syncthreads();
}

// Tile T [L][ng | 1]: an odd row stride, so that the lanes of a warp, which walk L rows
// at once, read 16-byte elements of different banks.
template <int L>
__global__ void k_adi_rows(const double2 *field, double2 *src, double2 *tmp,
                           Coef cf, double c, int ns, int ng, int first, int nband, int nseg, int nco, int W,
                           int has_src) {
  extern __shared__ __align__(16) unsigned char adi_smem[];
  const int st1 = ng | 1;
  const Lines ln = lines_setup(adi_smem, L, nseg, nco, W, ng, cf);  // tables: no kernel writes them
  chain_wait();
  C2 *T = ln.T;
  const int ii = blockIdx.x / nband, r0 = (blockIdx.x - ii * nband) * L, nr = min(L, ng - r0);
  const size_t ncell = (size_t)ng * ng;
  const double2 *u = field + (size_t)((ii + first) % ns) * ncell + (size_t)r0 * ng;
  double2 *s = src + (size_t)ii * ncell + (size_t)r0 * ng;
  double2 *w = tmp + (size_t)ii * ncell + (size_t)r0 * ng;
  for (int k = threadIdx.x; k < ng; k += blockDim.x) {
    C2 uu[L + 2], sv[L];
#pragma unroll
    for (int r = 0; r < L + 2; r++)  // uu[r]: u of row r0 + r - 1
      uu[r] = (r0 + r >= 1 && r0 + r - 1 < ng && r < nr + 2) ? ld(u + (long long)(r - 1) * ng + k) : C2{0, 0};
#pragma unroll
    for (int r = 0; r < L; r++) sv[r] = (has_src && r < nr) ? ld(s + (size_t)r * ng + k) : C2{0, 0};
#pragma unroll
    for (int r = 0; r < L; r++) {
      C2 v = {0, 0};
      if (r < nr) {
        // the rows outside the grid are zeros: (next - 2 u) + prev is then the reference's
        // one-sided difference, bit for bit
        v = add_imul(uu[r + 1], c, cadd(sub2(uu[r + 2], uu[r + 1]), uu[r]));
        st(s + (size_t)r * ng + k, v);
      }
      T[r * st1 + k] = cadd(v, sv[r]);
    }
  }
  __syncthreads();
  solve_lines(ln, L, st1, 1, ng, nseg, nco, W, c);
  for (int k = threadIdx.x; k < ng; k += blockDim.x)
#pragma unroll
    for (int r = 0; r < L; r++)
      if (r < nr) st(w + (size_t)r * ng + k, T[r * st1 + k]);
}

// Tile T [ng][L].
template <int L>
__global__ void k_adi_cols(double2 *field, const double2 *s1, const double2 *tmp, Coef cf, double c, int ns, int ng, int first, int nband,
                           int nseg, int nco, int W) {
  extern __shared__ __align__(16) unsigned char adi_smem[];
  const Lines ln = lines_setup(adi_smem, L, nseg, nco, W, ng, cf);  // tables: no kernel writes them
  const int ii = blockIdx.x / nband, c0 = (blockIdx.x - ii * nband) * L, nc = min(L, ng - c0);
  chain_wait();
  C2 *T = ln.T;
  const size_t ncell = (size_t)ng * ng;
  double2 *u = field + (size_t)((ii + first) % ns) * ncell + c0;
  const double2 *a = s1 + (size_t)ii * ncell + c0;
  const double2 *w = tmp + (size_t)ii * ncell + c0;
  const int line = threadIdx.x % L, row0 = threadIdx.x / L, dr = blockDim.x / L;
#pragma unroll 4
  for (int r = row0; r < ng; r += dr) {
    C2 v = {0, 0};
    if (line < nc) {
      const C2 wv = ld(w + (size_t)r * ng + line), av = ld(a + (size_t)r * ng + line);
      v = C2{fma(2., wv.x, -av.x), fma(2., wv.y, -av.y)};
    }
    T[r * L + line] = v;
  }
  __syncthreads();
  solve_lines(ln, L, 1, L, ng, nseg, nco, W, c);
  if (line < nc)
#pragma unroll 4
    for (int r = row0; r < ng; r += dr) st(u + (size_t)r * ng + line, T[r * L + line]);
}

}  // namespace adi64
