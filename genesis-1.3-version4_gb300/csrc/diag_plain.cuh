// Per-slice diagnostic sums of the FP64 form (DiagBeam::getValues and
// DiagField::getValues, src/Core/Diagnostic.cpp:415-456, 754-776), finished on the host.
// Included by kernels_plain.cu.
//
// One launch forms a whole record: CTAs of `chunk` particles of a slice, then CTAs of
// `rows` rows of a field slice. A slice's CTAs leave their partial sums in `part`, and the
// last of them to finish (a ticket per slice, no waiting) folds the partials, always in
// the same order.
//
// What bounds it is the FP64 pipe (64 cycles a warp's instruction), so instructions are
// spent only where the sums need them: e^{i theta} is the phasor the push left for the
// particle instead of a sincos of 24 instructions, higher harmonics its powers; minima and
// maxima compare the bit patterns on the integer pipe; the row moments' factors come from
// a table. 14 instructions a particle (one harmonic) and 7 a cell. Measured, with the
// host-link copy of the record: 1 slice x 8192, 255^2 530 -> 12 us a step; 320 x 8192,
// 151^2 850 -> 250 us.
namespace diag64 {

struct Args {
  Ptrs p;
  const double2 *ph1;  // e^{i theta} of every particle while *p.phasor_ok, null: none
  int ns, np, nharm, ng;
  double gref;  // gammaref: the record's gamma sums are about it
  int nbc, chunk;  // CTAs and particles of a CTA per beam slice
  int nfc, rows;   // CTAs and rows of a CTA per field slice
  double *rec;     // the record: beam [ns][beam_diag_width], fields [nfield][ns][kFieldSums + 2]
  double *part;
  unsigned *count;  // [ns] beam, [nfield][ns] fields; zero between launches
};

// NH harmonics at most: 12 + 2 NH sums, then 5 minima and 5 maxima
template <int NH>
constexpr int kSlots = kBeamSums + 2 * NH + kBeamMinMax;

// A double as a signed integer of the same order (its own inverse)
__device__ __forceinline__ long long order_key(long long b) { return b ^ ((b >> 63) & 0x7fffffffffffffffLL); }
__device__ __forceinline__ bool is_nan(long long b) {
  return (b & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL;
}
// fmin / fmax of the running extrema with v: a NaN changes nothing
__device__ __forceinline__ void extend(long long &mn, long long &mx, double v) {
  const long long b = __double_as_longlong(v);
  if (is_nan(b)) return;
  const long long k = order_key(b);
  mn = min(mn, k);
  mx = max(mx, k);
}

// Folds every thread's v[NV] (the first nsum are doubles to add, the next nmin keys to
// minimise, the rest keys to maximise) into out[NV]. red: NV x blockDim. Four threads a
// value, each over a quarter of the CTA; their reads start at different places so that
// they lie in different banks.
template <int NV>
__device__ __forceinline__ void fold(const long long (&v)[NV], int nsum, int nmin, long long *red, long long *out) {
  const int tid = threadIdx.x, nt = blockDim.x, n4 = nt >> 2;
#pragma unroll
  for (int k = 0; k < NV; k++) red[k * nt + tid] = v[k];
  __syncthreads();
  for (int t0 = 0; t0 < NV * 4; t0 += nt) {
    const int t = t0 + tid, k = min(t >> 2, NV - 1), q = t & 3;
    const long long *r = red + k * nt + q * n4;
    int i = (k + 8 * q) % n4;
    long long a = r[i];
    if (k < nsum) {
      // four partial sums: shorter chains of roundings and of latencies (n4 is a multiple of 8)
      double s[4];
      auto next = [&] {
        const double v = __longlong_as_double(r[i]);
        i = i + 1 < n4 ? i + 1 : 0;
        return v;
      };
#pragma unroll
      for (int w = 0; w < 4; w++) s[w] = next();
      for (int j = 4; j < n4; j += 4)
#pragma unroll
        for (int w = 0; w < 4; w++) s[w] += next();
      a = __double_as_longlong((s[0] + s[1]) + (s[2] + s[3]));
    } else {
      const bool lo = k < nsum + nmin;
      for (int j = 1; j < n4; j++) {
        i = i + 1 < n4 ? i + 1 : 0;
        a = lo ? min(a, r[i]) : max(a, r[i]);
      }
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      const long long b = __shfl_xor_sync(0xffffffffu, a, o);
      if (k < nsum)
        a = __double_as_longlong(__longlong_as_double(a) + __longlong_as_double(b));
      else
        a = k < nsum + nmin ? min(a, b) : max(a, b);
    }
    if (q == 0 && t < NV * 4) out[k] = a;
  }
  __syncthreads();
}

// The slice's value out[NV] from every CTA's v: folds the CTA, then (n CTAs a slice) the
// CTAs' partials part[NV][n] in the last CTA. False for the CTAs that are not the last.
template <int NV>
__device__ __forceinline__ bool fold_slice(long long (&v)[NV], int nsum, int nmin, const long long (&neutral)[NV],
                                           long long *red, long long *out, long long *part, unsigned *count, int n,
                                           int c) {
  fold<NV>(v, nsum, nmin, red, out);
  if (n == 1) return true;
  __shared__ bool last;
  if (threadIdx.x < NV) part[(size_t)threadIdx.x * n + c] = out[threadIdx.x];
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(count, 1u) == (unsigned)n - 1;
    if (last) *count = 0;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
#pragma unroll
  for (int k = 0; k < NV; k++) v[k] = neutral[k];
  for (int i = threadIdx.x; i < n; i += blockDim.x)
#pragma unroll
    for (int k = 0; k < NV; k++) {
      const long long b = __ldcg(part + (size_t)k * n + i);
      if (k < nsum)
        v[k] = __double_as_longlong(__longlong_as_double(v[k]) + __longlong_as_double(b));
      else
        v[k] = k < nsum + nmin ? min(v[k], b) : max(v[k], b);
    }
  fold<NV>(v, nsum, nmin, red, out);
  return true;
}

template <int NH>
__device__ __forceinline__ void beam_chunk(const Args &a, int is, int c, long long *red, long long *out) {
  constexpr int NS = kBeamSums + 2 * NH, NV = kSlots<NH>;
  const Ptrs &p = a.p;
  const size_t base = (size_t)is * a.np;
  const int n = slice_np(p, is, a.np), i0 = c * a.chunk, i1 = min(n, i0 + a.chunk);
  const bool cached = a.ph1 && *p.phasor_ok;
  double s[NS] = {0};
  // the reference's starting extrema (Diagnostic.cpp:424-438)
  long long mn[5], mx[5];
#pragma unroll
  for (int k = 0; k < 5; k++) {
    mn[k] = order_key(__double_as_longlong(k < 4 ? 1e5 : 1e7));
    mx[k] = order_key(__double_as_longlong(k < 4 ? -1e5 : 1.));
  }
  long long v[NV], neutral[NV];
#pragma unroll
  for (int k = 0; k < NV; k++) neutral[k] = k < NS ? 0 : k < NS + 5 ? mn[k - NS] : mx[k - NS - 5];
  for (int ip = i0 + (int)threadIdx.x; ip < i1; ip += blockDim.x) {
    const size_t o = base + ip;
    const double x = p.x[o], y = p.y[o], g = p.gamma[o], px = p.px[o], py = p.py[o];
    C2 z;
    if (cached) {
      z = ld(a.ph1 + o);
    } else {
      double sn, cs;
      sincos(p.theta[o], &sn, &cs);
      z = C2{cs, sn};
    }
    // gamma about gammaref: the difference is exact, and the spread does not cancel
    const double dg = g - a.gref;
    s[0] += dg;
    s[1] = fma(dg, dg, s[1]);
    s[2] += x;
    s[3] = fma(x, x, s[3]);
    s[4] += y;
    s[5] = fma(y, y, s[5]);
    s[6] += px;
    s[7] = fma(px, px, s[7]);
    s[8] += py;
    s[9] = fma(py, py, s[9]);
    s[10] = fma(x, px, s[10]);
    s[11] = fma(y, py, s[11]);
    extend(mn[0], mx[0], x);
    extend(mn[1], mx[1], px);
    extend(mn[2], mx[2], y);
    extend(mn[3], mx[3], py);
    extend(mn[4], mx[4], g);
    C2 zh = z;
#pragma unroll
    for (int h = 0; h < NH; h++) {
      if (h >= a.nharm) break;
      if (h > 0) zh = cmul_fma(zh, z);
      s[kBeamSums + 2 * h] += zh.x;
      s[kBeamSums + 2 * h + 1] += zh.y;
    }
  }
#pragma unroll
  for (int k = 0; k < NV; k++)
    v[k] = k < NS ? __double_as_longlong(s[k]) : k < NS + 5 ? mn[k - NS] : mx[k - NS - 5];
  if (!fold_slice<NV>(v, NS, 5, neutral, red, out, reinterpret_cast<long long *>(a.part) + (size_t)is * a.nbc * NV,
                      a.count + is, a.nbc, c))
    return;
  double *o = a.rec + (size_t)is * beam_diag_width(a.nharm);
  const int t = threadIdx.x;
  if (t < kBeamSums) o[t] = __longlong_as_double(out[t]);
  if (t < 2 * a.nharm) o[kBeamSums + kBeamMinMax + t] = __longlong_as_double(out[kBeamSums + t]);
  if (t < 10) o[kBeamSums + t] = __longlong_as_double(order_key(out[NS + 5 * (t & 1) + (t >> 1)]));
}

template <int NV>
__device__ __forceinline__ void field_rows(const Args &a, int k, int i, int c, long long *red, long long *out,
                                           double *part) {
  static_assert(NV == kFieldSums, "");
  const int ng = a.ng, r0 = c * a.rows, nr = min(a.rows, ng - r0), tid = threadIdx.x;
  const double shift = -0.5 * (double)(ng - 1);
  const double2 *f = a.p.field[k] + (size_t)i * ng * ng;
  double2 *dy = reinterpret_cast<double2 *>(red);  // the rows' dy, dy^2 (before the fold uses red)
  for (int r = tid; r < nr; r += blockDim.x) {
    const double d = (double)(r0 + r) + shift;
    dy[r] = make_double2(d, d * d);
  }
  __syncthreads();
  double s[NV] = {0};
  for (int col = tid; col < ng; col += blockDim.x) {
    double s2[2] = {0, 0};
    auto row = [&](int r, double2 u, double &sw) {
      const double2 d = dy[r];
      const double w = fma(u.x, u.x, u.y * u.y);
      sw += w;
      s[3] = fma(d.x, w, s[3]);
      s[4] = fma(d.y, w, s[4]);
      s[5] += u.x;
      s[6] += u.y;
    };
    for (int r4 = 0; r4 < nr; r4 += 4) {  // four rows' loads together
      double2 u[4];
#pragma unroll
      for (int q = 0; q < 4; q++) u[q] = f[(size_t)(r0 + min(r4 + q, nr - 1)) * ng + col];
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (r4 + q < nr) row(r4 + q, u[q], s2[q & 1]);
    }
    const double sw = s2[0] + s2[1];
    const double dx = (double)col + shift, t = dx * sw;
    s[0] += sw;
    s[1] += t;
    s[2] = fma(dx, t, s[2]);
  }
  __syncthreads();
  long long v[NV];
  const long long neutral[NV] = {0};
#pragma unroll
  for (int q = 0; q < NV; q++) v[q] = __double_as_longlong(s[q]);
  double *o = a.rec + (size_t)a.ns * beam_diag_width(a.nharm) + ((size_t)k * a.ns + i) * (kFieldSums + 2);
  // the value on the axis, from the CTA that holds it
  if (tid == 0 && ng / 2 >= r0 && ng / 2 < r0 + nr) {
    const double2 u = f[(size_t)(ng / 2) * ng + ng / 2];
    o[7] = u.x;
    o[8] = u.y;
  }
  if (!fold_slice<NV>(v, NV, 0, neutral, red, out, reinterpret_cast<long long *>(part) + ((size_t)k * a.ns + i) * a.nfc * NV,
                      a.count + a.ns + (size_t)k * a.ns + i, a.nfc, c))
    return;
  if (tid < NV) o[tid] = __longlong_as_double(out[tid]);
}

// Shared memory: kSlots<NH> x (blockDim + 1) doubles, the last column the folded values.
template <int NH>
__global__ void __launch_bounds__(256) k_diag(Args a) {
  extern __shared__ __align__(16) unsigned char diag_smem[];
  long long *red = reinterpret_cast<long long *>(diag_smem), *out = red + kSlots<NH> * blockDim.x;
  unsigned b = blockIdx.x;
  const unsigned nb = (unsigned)a.ns * a.nbc;
  if (b < nb) {
    beam_chunk<NH>(a, b / a.nbc, b % a.nbc, red, out);
    return;
  }
  b -= nb;
  const unsigned per = (unsigned)a.ns * a.nfc;
  field_rows<kFieldSums>(a, b / per, b % per / a.nfc, b % a.nfc, red, out, a.part + (size_t)nb * kSlots<NH>);
}

}  // namespace diag64
