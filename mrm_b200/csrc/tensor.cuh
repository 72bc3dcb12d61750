// tensor.cuh -- FP64 magnetostatic tensor and its spectrum, once per run.
//
// Device restatement of volume_averaged_n / plane_to_plane
// (src/tensor_element.f90:13-102, :219-261) and calculate_tensor
// (src/tensor.f90:82-216): every in-plane offset that wraps onto a slot and all
// its periodic images, from corner values that the slots of a tile share
// (tensor_real_kernel).  The FP64 real tensor is then transformed in FP64
// (demag.f90:259-267 does this once per run) and packed: each of the 9
// components of a layer pair has a purely real (xx, yy, zz, xy, yx) or purely
// imaginary (xz, zx, yz, zy) spectrum, even or odd in ky, so one real number
// per (kx, 0 <= ky <= py/2) is kept.
#pragma once
#include "common.cuh"
#include "dd.cuh"
#include "fft.cuh"

namespace mrm {

struct PairGeom {
  double dz_s, dz_o;  // source / observation layer thickness
  double rz;          // centre-to-centre z offset, source - observation
  double rz_sul, f_sul;    // SUL image term (f_sul = 0: none), tensor.f90:162-171
  double rz_head, f_head;  // head image term, tensor.f90:172-181
  double norm;        // 1/(dx dy dz_o px py), tensor.f90:183
};

// One corner combination of volume_averaged_n (tensor_element.f90:39-72) in
// double-double: the corner offsets (x, y, z), d = |(x, y, z)|, the three
// arctangents and six logarithms that g1 and g2 (:78-100) share, and the
// six distinct elements.  g1(x,y,z,d) and g2(z,x,y,d) are the reference's
// closed forms with their max(1e-300, .) guards and Fortran sign(); the
// arctangent arguments y z / sign(max(1e-300, |x| d), x) and their
// permutations are A_x, A_y, A_z.
struct TensCorner {
  dd t00, t11, t22, t12, t02, t01;  // g1(x,y,z), g1(y,z,x), g1(z,x,y), g2(x,y,z), g2(y,z,x), g2(z,x,y)
};

__device__ __forceinline__ dd tens_den(dd v, dd d) {
  // sign(max(1e-300, |v| d), v)
  const dd a = dd_max_d(dd_mul(dd_abs(v), d), 1.0e-300);
  return signbit(v.hi) ? dd_neg(a) : a;
}
__device__ __forceinline__ dd tens_log(dd v) { return dd_log(dd_max_d(v, 1.0e-300)); }

__device__ __noinline__ TensCorner tens_corner(dd x, dd y, dd z) {
  const dd x2 = dd_mul(x, x), y2 = dd_mul(y, y), z2 = dd_mul(z, z);
  const dd d = dd_sqrt(dd_add(dd_add(x2, y2), z2));
  const dd xyz = dd_mul(dd_mul(x, y), z);
  const dd ax = dd_atan(dd_div(dd_mul(y, z), tens_den(x, d)));
  const dd ay = dd_atan(dd_div(dd_mul(z, x), tens_den(y, d)));
  const dd az = dd_atan(dd_div(dd_mul(x, y), tens_den(z, d)));
  const dd lmx = tens_log(dd_sub(d, x)), lmy = tens_log(dd_sub(d, y)), lmz = tens_log(dd_sub(d, z));
  const dd lpx = tens_log(dd_add(d, x)), lpy = tens_log(dd_add(d, y)), lpz = tens_log(dd_add(d, z));
  const dd sixth = dd_recip_int(6), third = dd_recip_int(3);
  auto half = [](dd v) { return dd_ldexp(v, -1); };
  TensCorner c;
  // g1(x, y, z, d)
  c.t00 = dd_add(dd_add(dd_mul(xyz, ax), half(dd_mul(dd_mul(y, dd_sub(z2, x2)), lmy))),
                 dd_add(half(dd_mul(dd_mul(z, dd_sub(y2, x2)), lmz)),
                        dd_mul(dd_mul(dd_sub(dd_add(y2, z2), dd_ldexp(x2, 1)), d), sixth)));
  // g1(y, z, x, d)
  c.t11 = dd_add(dd_add(dd_mul(xyz, ay), half(dd_mul(dd_mul(z, dd_sub(x2, y2)), lmz))),
                 dd_add(half(dd_mul(dd_mul(x, dd_sub(z2, y2)), lmx)),
                        dd_mul(dd_mul(dd_sub(dd_add(z2, x2), dd_ldexp(y2, 1)), d), sixth)));
  // g1(z, x, y, d)
  c.t22 = dd_add(dd_add(dd_mul(xyz, az), half(dd_mul(dd_mul(x, dd_sub(y2, z2)), lmx))),
                 dd_add(half(dd_mul(dd_mul(y, dd_sub(x2, z2)), lmy)),
                        dd_mul(dd_mul(dd_sub(dd_add(x2, y2), dd_ldexp(z2, 1)), d), sixth)));
  // g2(x, y, z, d): -x y z log(d+x) + z (z^2 - 3x^2) log(d+y)/6 + y (y^2 - 3x^2) log(d+z)/6
  //   + y^2 x A_y / 2 + z^2 x A_z / 2 + x^3 A_x / 6 + y z d / 3
  c.t12 = dd_add(dd_add(dd_neg(dd_mul(xyz, lpx)),
                        dd_mul(dd_add(dd_mul(dd_mul(z, dd_sub(z2, dd_mul_d(x2, 3.0))), lpy),
                                      dd_mul(dd_mul(y, dd_sub(y2, dd_mul_d(x2, 3.0))), lpz)),
                               sixth)),
                 dd_add(dd_add(half(dd_mul(dd_mul(y2, x), ay)), half(dd_mul(dd_mul(z2, x), az))),
                        dd_add(dd_mul(dd_mul(dd_mul(x2, x), ax), sixth), dd_mul(dd_mul(dd_mul(y, z), d), third))));
  // g2(y, z, x, d)
  c.t02 = dd_add(dd_add(dd_neg(dd_mul(xyz, lpy)),
                        dd_mul(dd_add(dd_mul(dd_mul(x, dd_sub(x2, dd_mul_d(y2, 3.0))), lpz),
                                      dd_mul(dd_mul(z, dd_sub(z2, dd_mul_d(y2, 3.0))), lpx)),
                               sixth)),
                 dd_add(dd_add(half(dd_mul(dd_mul(z2, y), az)), half(dd_mul(dd_mul(x2, y), ax))),
                        dd_add(dd_mul(dd_mul(dd_mul(y2, y), ay), sixth), dd_mul(dd_mul(dd_mul(z, x), d), third))));
  // g2(z, x, y, d)
  c.t01 = dd_add(dd_add(dd_neg(dd_mul(xyz, lpz)),
                        dd_mul(dd_add(dd_mul(dd_mul(y, dd_sub(y2, dd_mul_d(z2, 3.0))), lpx),
                                      dd_mul(dd_mul(x, dd_sub(x2, dd_mul_d(z2, 3.0))), lpy)),
                               sixth)),
                 dd_add(dd_add(half(dd_mul(dd_mul(x2, z), ax)), half(dd_mul(dd_mul(y2, z), ay))),
                        dd_add(dd_mul(dd_mul(dd_mul(z2, z), az), sixth), dd_mul(dd_mul(dd_mul(x, y), d), third))));
  return c;
}

// volume_averaged_n (tensor_element.f90:13-102) sums the corner values over 64
// sign combinations.  The source and the observation cell have the same extent
// along x, so the x offsets of a slot's corners are the lattice points a dx,
// a = -i - 1, -i, -i + 1 for the source offset i, with weights -1, 2, -1: a
// second difference, whose points adjacent slots share.  Along y (the
// reference's quirk dyo = xo, :31) the four offsets -j dy + (+-xo +- ys)/2 form
// the same lattice when dx == dy; otherwise every slot row has four y values of
// its own.  Along z there are four heights (three for equal thicknesses).
// A block evaluates the corner values of a tile of slots once, in shared
// memory, and takes the differences: (T + 2)^2 / T^2 evaluations per slot and
// height instead of 64 / 4 (T = 8: 1.6 against 16).  The element is even or
// odd in each of i and j, so only slots with f <= n/2 are evaluated.
// Bound by the double-double arithmetic of the corner values (six logarithms
// and three arctangents each).  T = 8: the 300 values of a tile and three
// heights are two rounds of a 256-thread block, which is what a small grid's
// few tiles wait for; T = 16 saves a fifth of the evaluations and doubles the rounds.
// Measured with the calls' copies and allocation: build_tensor and a field
// evaluation on 512 x 512 slots 1.7 to 2.4 ms (64 evaluations per slot: 30.5),
// off_field on 1024 x 256 slots and two layers 2.7 to 3.5 ms (50.1).
constexpr int kTensTile = 8, kTensBlock = 256, kTensItems = kTensTile * kTensTile * 6;
MRM_HD constexpr int tens_rows(bool lattice_y) { return lattice_y ? kTensTile + 2 : 4 * kTensTile; }
MRM_HD constexpr size_t tens_smem(bool lattice_y) {
  return (size_t)6 * sizeof(dd) * tens_rows(lattice_y) * (kTensTile + 2) * 4;
}

// Corner offset q of the four (+-o/2) - (+-s/2) around the centre c, in the
// reference's order of operations: q = 0, 1 the two of weight +1 (equal signs),
// q = 2, 3 those of weight -1.
__device__ __forceinline__ dd tens_offset(dd c, double o, double s, int q) {
  const double po = (q & 1) ? 0.5 : -0.5, ps = (q == 0 || q == 3) ? -0.5 : 0.5;
  return dd_add_d(dd_add_d(c, po * o), -(ps * s));
}

// calculate_tensor (tensor.f90:82-216) with plane_to_plane
// (tensor_element.f90:233-257): n2d[((pair*9 + c)*py + fj)*px + fi], c = 3*b + a
// holds t(a,b) (Fortran n2d layout).  Slot f of n holds every offset i with
// (n - i) mod n == f: i = -f (f <= n/2) with its periodic images -nimg..nimg;
// the slot half way round holds -n/2 with images <= 0 and +n/2 with images
// >= 0, the mirror image of the former, so its element is twice the first
// set's (even components) or zero (odd ones).  Slot n - f mirrors slot f.
// grid: (tiles of slots 0..px/2 x 0..py/2, pairs).
__global__ void __launch_bounds__(kTensBlock) tensor_real_kernel(double* __restrict__ n2d,
                                                                 const PairGeom* __restrict__ pg, int px, int py,
                                                                 double dx, double dy, int nimg) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  dd* F = reinterpret_cast<dd*>(smem_raw);  // [component][height][row][column]
  constexpr int T = kTensTile, C = T + 2;
  const bool lat = dx == dy;
  const int rows = tens_rows(lat), ntx = (px / 2 + T) / T;
  const int fi0 = (int)(blockIdx.x % ntx) * T, fj0 = (int)(blockIdx.x / ntx) * T, pair = blockIdx.y;
  const PairGeom g = pg[pair];
  const bool eqz = g.dz_s == g.dz_o;
  const int nz = eqz ? 3 : 4, plane = rows * C, cstride = plane * nz;
  constexpr int Q = (kTensItems + kTensBlock - 1) / kTensBlock;
  // the element as the rows a = 0, 1 and the row a = 2 of the tensor have it
  // (an image term carries -f and +f there)
  dd lo[Q], hi[Q];
  for (int q = 0; q < Q; ++q) lo[q] = hi[q] = dd_from(0.0);
  for (int src = 0; src < 3; ++src) {
    const double f = src == 0 ? 1.0 : src == 1 ? g.f_sul : g.f_head;
    if (f == 0.0) continue;
    const double rz = src == 0 ? g.rz : src == 1 ? g.rz_sul : g.rz_head;
    dd acc[Q];
    for (int q = 0; q < Q; ++q) acc[q] = dd_from(0.0);
    for (int iy = -nimg; iy <= nimg; ++iy)
      for (int ix = -nimg; ix <= nimg; ++ix) {
        __syncthreads();
#pragma unroll 1
        for (int it = threadIdx.x; it < cstride; it += kTensBlock) {
          const int h = it / plane, rc = it - h * plane, r = rc / C, c = rc - r * C;
          const int a = fi0 + c - 1, b = lat ? fj0 + r - 1 : fj0 + (r >> 2);
          if (a > px / 2 + 1 || b > py / 2 + (lat ? 1 : 0)) continue;  // past the last slot: not read
          const dd x = two_prod((double)(a - ix * px), dx);
          const dd yc = two_prod((double)(b - iy * py), dy);
          const dd y = lat ? yc : tens_offset(yc, dx, dy, r & 3);
          // heights: 0 the two of weight +1 (one for equal thicknesses), then those of weight -1
          const dd z = tens_offset(dd_from(-rz), g.dz_o, g.dz_s, eqz && h ? h + 1 : h);
          TensCorner k;
          if (x.hi == 0.0 && y.hi == 0.0 && z.hi == 0.0)  // d = 0
            k.t00 = k.t11 = k.t22 = k.t12 = k.t02 = k.t01 = dd_from(0.0);
          else
            k = tens_corner(x, y, z);
          F[it] = k.t00;
          F[cstride + it] = k.t11;
          F[2 * cstride + it] = k.t22;
          F[3 * cstride + it] = k.t12;
          F[4 * cstride + it] = k.t02;
          F[5 * cstride + it] = k.t01;
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          const int w = threadIdx.x + q * kTensBlock;
          if (w >= kTensItems) continue;
          const int si = w % T, sj = (w / T) % T, comp = w / (T * T);
          const int fi = fi0 + si, fj = fj0 + sj;
          if (fi > px / 2 || fj > py / 2) continue;
          if ((fi == px / 2 && ix > 0) || (fj == py / 2 && iy > 0)) continue;
          dd n = dd_from(0.0);
          for (int h = 0; h < nz; ++h) {
            const dd* P = F + comp * cstride + h * plane + si;
            auto diff_x = [&](int r) {
              const dd* p = P + r * C;
              return dd_sub(dd_ldexp(p[1], 1), dd_add(p[0], p[2]));
            };
            const dd v = lat ? dd_sub(dd_ldexp(diff_x(sj + 1), 1), dd_add(diff_x(sj), diff_x(sj + 2)))
                             : dd_sub(dd_add(diff_x(4 * sj), diff_x(4 * sj + 1)),
                                      dd_add(diff_x(4 * sj + 2), diff_x(4 * sj + 3)));
            const bool plus = eqz ? h == 0 : h < 2;
            n = plus ? dd_add(n, eqz ? dd_ldexp(v, 1) : v) : dd_sub(n, v);
          }
          acc[q] = dd_add(acc[q], n);
        }
      }
    for (int q = 0; q < Q; ++q) {
      lo[q] = dd_add(lo[q], src == 0 ? acc[q] : dd_mul_d(acc[q], -f));
      hi[q] = dd_add(hi[q], src == 0 ? acc[q] : dd_mul_d(acc[q], f));
    }
  }
  for (int q = 0; q < Q; ++q) {
    const int w = threadIdx.x + q * kTensBlock;
    if (w >= kTensItems) continue;
    const int si = w % T, sj = (w / T) % T, comp = w / (T * T);
    const int fi = fi0 + si, fj = fj0 + sj;
    if (fi > px / 2 || fj > py / 2) continue;
    // components 00, 11, 22, 12, 02, 01
    const bool oddx = comp >= 4, oddy = comp == 3 || comp == 5;
    const int ca = comp < 3 ? comp : comp == 3 ? 1 : 0, cb = comp < 3 ? comp : comp == 5 ? 1 : 2;
    double s = g.norm;
    if (fi == px / 2) s *= oddx ? 0.0 : 2.0;
    if (fj == py / 2) s *= oddy ? 0.0 : 2.0;
    // (a, b) = (ca, cb), and its transpose
    const double v = dd_mul_d(ca == 2 ? hi[q] : lo[q], s).hi, vt = dd_mul_d(cb == 2 ? hi[q] : lo[q], s).hi;
    for (int my = 0; my < 2; ++my) {
      if (my && (fj == 0 || fj == py / 2)) continue;
      for (int mx = 0; mx < 2; ++mx) {
        if (mx && (fi == 0 || fi == px / 2)) continue;
        const double sign = ((mx && oddx) != (my && oddy)) ? -1.0 : 1.0;
        const long long at = (long long)(my ? py - fj : fj) * px + (mx ? px - fi : fi);
        double* dst = n2d + (long long)pair * 9 * py * px + at;
        dst[(long long)(3 * cb + ca) * py * px] = sign * v;
        if (ca != cb) dst[(long long)(3 * ca + cb) * py * px] = sign * vt;
      }
    }
  }
}

// FP64 r2c along x of `planes` real planes [p][py][px] -> [p][py][px/2+1]
__global__ void __launch_bounds__(256) r2c_rows_f64(const double* __restrict__ in,
                                                    Cx<double>* __restrict__ out, int lgpx,
                                                    int py, const Cx<double>* __restrict__ tw) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lgM = lgpx - 1, M = 1 << lgM, ph = M + 1, px = 2 * M;
  const long long row = blockIdx.x;  // p*py + j
  const int cs = pad_stride(M);
  Cx<double>* A = reinterpret_cast<Cx<double>*>(smem_raw);
  Cx<double>* B = A + cs;
  const double* src = in + row * px;
  for (int k = threadIdx.x; k < M; k += blockDim.x) A[k] = Cx<double>{src[2 * k], src[2 * k + 1]};
  __syncthreads();
  Cx<double>* Y = block_fft<double, -1>(A, B, lgM, 1, cs, tw, kTwLog);
  for (int k = threadIdx.x; k < ph; k += blockDim.x) {
    const Cx<double> yk = Y[k & (M - 1)], ymk = cconj(Y[(M - k) & (M - 1)]);
    const Cx<double> e = cscale(cadd(yk, ymk), 0.5), o = cscale(csub(yk, ymk), 0.5);
    const Cx<double> wo = cmul(twiddle(tw, k & (px - 1), lgpx), o);
    out[row * ph + k] = csub(e, cmul_i(wo, 1.0));
  }
}

// FP64 complex FFT along y of [p][py][ph], in place; one block per (p, column)
__global__ void __launch_bounds__(256) c2c_cols_f64(Cx<double>* __restrict__ data, int lgpy, int ph,
                                                    const Cx<double>* __restrict__ tw) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int py = 1 << lgpy;
  const long long p = blockIdx.x / ph;
  const int k = blockIdx.x - (int)(p * ph);
  const int cs = pad_stride(py);
  Cx<double>* A = reinterpret_cast<Cx<double>*>(smem_raw);
  Cx<double>* B = A + cs;
  Cx<double>* base = data + p * (long long)py * ph + k;
  for (int j = threadIdx.x; j < py; j += blockDim.x) A[j] = base[(long long)j * ph];
  __syncthreads();
  Cx<double>* Y = block_fft<double, -1>(A, B, lgpy, 1, cs, tw, kTwLog);
  for (int j = threadIdx.x; j < py; j += blockDim.x) base[(long long)j * ph] = Y[j];
}

// inverse FP64 complex FFT along y of [p][py][ph], in place (unnormalised)
__global__ void __launch_bounds__(256) c2c_cols_f64_inv(Cx<double>* __restrict__ data, int lgpy, int ph,
                                                        const Cx<double>* __restrict__ tw) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int py = 1 << lgpy;
  const long long p = blockIdx.x / ph;
  const int k = blockIdx.x - (int)(p * ph);
  const int cs = pad_stride(py);
  Cx<double>* A = reinterpret_cast<Cx<double>*>(smem_raw);
  Cx<double>* B = A + cs;
  Cx<double>* base = data + p * (long long)py * ph + k;
  for (int j = threadIdx.x; j < py; j += blockDim.x) A[j] = base[(long long)j * ph];
  __syncthreads();
  Cx<double>* Y = block_fft<double, +1>(A, B, lgpy, 1, cs, tw, kTwLog);
  for (int j = threadIdx.x; j < py; j += blockDim.x) base[(long long)j * ph] = Y[j];
}

// FP64 c2r along x (FFTW's unnormalised c2r): rows [p][py][px/2+1] -> real
// [p][py][px] through the half-length complex transform (imaginary parts of
// the k = 0 and k = px/2 bins ignored)
__global__ void __launch_bounds__(256) c2r_rows_f64(const Cx<double>* __restrict__ in, double* __restrict__ out,
                                                    int lgpx, const Cx<double>* __restrict__ tw) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lgM = lgpx - 1, M = 1 << lgM, ph = M + 1, px = 2 * M;
  const long long row = blockIdx.x;  // p*py + j
  const int cs = pad_stride(M);
  Cx<double>* A = reinterpret_cast<Cx<double>*>(smem_raw);
  Cx<double>* B = A + cs;
  const Cx<double>* X = in + row * ph;
  for (int k = threadIdx.x; k < M; k += blockDim.x) {
    Cx<double> a = X[k], b = X[M - k];
    if (k == 0) {
      a.y = 0.0;
      b.y = 0.0;
    }
    const Cx<double> e = cadd(a, cconj(b)), o = csub(a, cconj(b));
    const Cx<double> w = cconj(twiddle(tw, k, lgpx));  // e^{+2 pi i k / px}
    A[k] = cadd(e, cmul_i(cmul(o, w), 1.0));
  }
  __syncthreads();
  Cx<double>* Z = block_fft<double, +1>(A, B, lgM, 1, cs, tw, kTwLog);
  double* dst = out + row * px;
  for (int n = threadIdx.x; n < M; n += blockDim.x) {
    dst[2 * n] = Z[n].x;
    dst[2 * n + 1] = Z[n].y;
  }
}

// block-wide max of two non-negative doubles, one atomicMax per block
__device__ __forceinline__ void block_max2(double a, double b, unsigned long long* ga,
                                           unsigned long long* gb) {
  __shared__ double sa[32], sb[32];
  for (int o = 16; o > 0; o >>= 1) {
    a = fmax(a, __shfl_xor_sync(0xffffffffu, a, o));
    b = fmax(b, __shfl_xor_sync(0xffffffffu, b, o));
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) { sa[warp] = a; sb[warp] = b; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x + 31) / 32; ++w) { a = fmax(a, sa[w]); b = fmax(b, sb[w]); }
    atomicMax(ga, (unsigned long long)__double_as_longlong(a));
    atomicMax(gb, (unsigned long long)__double_as_longlong(b));
  }
}

// parity-violating part of one spectral value (and its ky mirror) and the kept part
__device__ __forceinline__ void parity_parts(const Cx<double>* S, int c, int kyh, int k, int py, int ph,
                                             double* keep, double* disc) {
  const Cx<double> v = S[(long long)kyh * ph + k];
  const bool imag = (kImagMask >> c) & 1;
  const bool odd = (kOddMask >> c) & 1;
  *keep = imag ? v.y : v.x;
  double d = imag ? fabs(v.x) : fabs(v.y);
  if (kyh > 0 && kyh < py - kyh) {
    const Cx<double> u = S[(long long)(py - kyh) * ph + k];
    const double um = imag ? u.y : u.x;
    d = fmax(d, fabs(um - (odd ? -*keep : *keep)));
  }
  *disc = d;
}

// spectrum [pair][9][py][ph] (FP64) -> tens[k][pair][c][kyh] (R, rows of pyhs
// reals): one real per component and 0 <= ky <= py/2 (FP32 runs); tracks the
// dropped residue.
template <typename R>
__global__ void pack_tensor_kernel(const Cx<double>* __restrict__ spec, R* __restrict__ tens,
                                   int npair, int py, int ph, int pyhs, unsigned long long* resid,
                                   unsigned long long* kept) {
  const int pyh = py / 2 + 1;
  const long long total = (long long)ph * npair * 9 * pyh;
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  double keep = 0.0, disc = 0.0;
  if (gid < total) {
    const int kyh = (int)(gid % pyh);
    long long r = gid / pyh;
    const int c = (int)(r % 9);
    r /= 9;
    const int pair = (int)(r % npair);
    const int k = (int)(r / npair);
    parity_parts(spec + ((long long)pair * 9 + c) * py * ph, c, kyh, k, py, ph, &keep, &disc);
    tens[(gid / pyh) * pyhs + kyh] = (R)keep;
  }
  block_max2(disc, fabs(keep), resid, kept);
}

// spectrum [pair][9][py][ph] (FP64) -> the register column kernel's tensor
// (colreg.cuh): floats [column pair][pair of layers][6][j < 4][t < py/8][h < 2][column],
// components xx, yy, zz, xy, xz, yz (yx, zx, zy taken as xy, xz, yz) at
// position 8t + 2j + h of the column transform's digit-reversed order (element
// p holds k_y = ip_freq(p)), the sign of the odd components for k_y > py/2
// folded in, zero for the partner of a last odd column.  mx: wrong-parity
// residue, kept part, largest difference between a component and its transpose.
__global__ void pack_tensor_creg_kernel(const Cx<double>* __restrict__ spec, float* __restrict__ tens, int npair,
                                        int lgpy, int ph, unsigned long long* mx) {
  const int py = 1 << lgpy;
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long per = (long long)npair * 6 * 2 * py;
  double keep = 0.0, disc = 0.0, asym = 0.0;
  if (gid < (ph + 1) / 2 * per) {
    const int col = (int)(gid & 1), h = (int)(gid >> 1) & 1;
    const int t = (int)(gid >> 2) & (py / 8 - 1), j = (int)(gid >> (lgpy - 1)) & 3;
    const int r = (int)((gid % per) >> (lgpy + 1)), c6 = r % 6, pair = r / 6;
    const int k = 2 * (int)(gid / per) + col;
    const int ky = ip_freq(8 * t + 2 * j + h, lgpy);
    const bool upper = ky > py / 2;
    const int kyh = upper ? py - ky : ky;
    constexpr int kComp[6] = {0, 4, 8, 1, 2, 5};   // xx yy zz xy xz yz
    constexpr int kTrans[6] = {0, 4, 8, 3, 6, 7};  // their transposes
    const int c = kComp[c6], ct = kTrans[c6];
    if (k < ph) {
      const Cx<double>* S = spec + (long long)pair * 9 * py * ph;
      parity_parts(S + (long long)c * py * ph, c, kyh, k, py, ph, &keep, &disc);
      if (ct != c) {
        double kt, dt;
        parity_parts(S + (long long)ct * py * ph, ct, kyh, k, py, ph, &kt, &dt);
        disc = fmax(disc, dt);
        asym = fabs(kt - keep);
      }
    }
    const bool odd = (kOddMask >> c) & 1;
    tens[gid] = (float)((odd && upper) ? -keep : keep);
  }
  block_max2(disc, fabs(keep), mx, mx + 1);
  __syncthreads();
  block_max2(asym, 0.0, mx + 2, mx + 1);
}

// spectrum [pair][9][py][ph] -> tens[k][pair][c][p] complex (FP64 runs), position
// p of the column transform's digit-reversed order holding k_y = ip_freq(p), so
// the product reads consecutive values
__global__ void pack_tensor_full_kernel(const Cx<double>* __restrict__ spec, Cx<double>* __restrict__ tens,
                                        int npair, int lgpy, int ph, unsigned long long* resid,
                                        unsigned long long* kept) {
  const int py = 1 << lgpy;
  const long long total = (long long)ph * npair * 9 * py;
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  double keep = 0.0, disc = 0.0;
  if (gid < total) {
    const int ky = ip_freq((int)(gid % py), lgpy);
    long long r = gid / py;
    const int c = (int)(r % 9);
    r /= 9;
    const int pair = (int)(r % npair);
    const int k = (int)(r / npair);
    const Cx<double>* S = spec + ((long long)pair * 9 + c) * py * ph;
    tens[gid] = S[(long long)ky * ph + k];
    if (ky <= py / 2) parity_parts(S, c, ky, k, py, ph, &keep, &disc);
  }
  block_max2(disc, fabs(keep), resid, kept);
}

}  // namespace mrm
