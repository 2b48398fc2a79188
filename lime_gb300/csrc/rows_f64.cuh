// Row lists of a Lindblad generator for the FP64 propagators.
//
// GB300 issues a warp-wide FP64 instruction every 64 clocks on each of an
// SM's four partitions, and 1.68 FP64 lanes per clock and SM when all four
// are busy (measured with independent fma chains of 1 to 16 warps): one DFMA
// takes the time of some sixty other instructions, and its result is there
// when the next one can issue.  An FP64 kernel is therefore as fast as its
// DFMA count allows, and shared-memory traffic, index arithmetic and branches
// are nearly free beside it.  The generators this library meets are rarely
// full: a nearest-neighbour chain has two off-diagonal entries a row, a
// relaxation operator |j><k| one entry in all, and a real symmetric H leaves
// the off-diagonal of Heff real (half the DFMA).  So the right-hand side is
// evaluated element by element over lists of the nonzero entries,
//     f_pq = c_pq rho_pq - i (sum_k h_pk rho_kq - sum_k conj(h_qk) rho_pk)
//            + sum_k (L_k rho L_k^dag)_pq,
//     c_pq = -i (h_pp - conj(h_qq)) + M_pq,
// for p <= q only (rho and f are Hermitian), and one real component at a
// time: the n^2 real numbers of a Hermitian matrix are the work items, item
// (i, j) being Re rho_ij for i <= j and Im rho_ji for i > j, which leaves no
// half-empty warp for the real diagonal.  With own the item's component and
// oth the other one, times +1 (Re) or -1 (Im),
//     f = c.x own_pq - c.y oth_pq + sum_k h_pk.x oth_kq - sum_k h_qk.x oth_pk
//         + sum_k h_pk.y own_kq + sum_k h_qk.y own_pk.
// A full complex H costs the 4 n^3 DFMA of the product Heff rho, with no
// padding to a tile.
#pragma once

#include "common.cuh"

namespace lime {
namespace f64 {

// Off-diagonal entries of an n x n matrix in `width` columns, entry e of row
// i at [e * n + i].
//   sparse: ent = {Re h, the column's offsets as two words (k ld2, 2 k)},
//           hy = Im h (complex rows only); shorter rows end in zeros at the
//           row's own column
//   dense:  full rows, entry e is column e + (e >= i); ent holds Re h as
//           doubles (real) or h as double2
// d: the diagonal.
struct Rows {
  const double2* ent;
  const double* hy;
  const double2* d;
  int n, width;
  bool dense, real;
};

// Largest dimension that takes sparse rows; a larger matrix uses full rows
// in global memory and the spare last row of their array for its diagonal.
constexpr int kRowsSmemMax = 4096;

template <bool kCg>
__device__ __forceinline__ double2 ldz(const double2* p) {
  if (kCg) return __ldcg(p);
  return *p;
}
template <bool kCg>
__device__ __forceinline__ double ldd(const double* p) {
  if (kCg) return __ldcg(p);
  return *p;
}

// One work item: element (p, q) of the upper triangle, im: its imaginary part.
struct Item {
  int p, q;
  bool im;
};
__device__ __forceinline__ Item item_of(int i, int j) {
  return i <= j ? Item{i, j, false} : Item{j, i, true};
}

// c_pq of the header comment
__device__ __forceinline__ double2 diag_coef(double2 hp, double2 hq, double2 m) {
  return make_double2(hp.y + hq.y + m.x, hq.x - hp.x + m.y);
}

// x with its sign flipped where `mask` (0 or the sign bit) says so; an
// integer operation, the FP64 pipe is the bound
__device__ __forceinline__ double flip(double x, int mask) {
  return __hiloint2double(__double2hiint(x) ^ mask, __double2loint(x));
}

// f of kN items without the jump terms of the operators.  x: the n x n state
// as doubles, ld2 doubles a row.  The entry loop is outside, so the loads of
// the items overlap.
template <int kN, bool kCg, class Idx>
__device__ __forceinline__ void rhs_items(const Rows& R, const double2 (&c)[kN], const double* x, Idx ld2,
                                          const Item (&it)[kN], double (&f)[kN]) {
  const int n = R.n, W = R.width;
  const auto oth = [&](int u) { return it[u].im ? 0 : 1; };
  const auto sgn = [&](int u) { return it[u].im ? (int)0x80000000 : 0; };
#pragma unroll
  for (int u = 0; u < kN; ++u) {
    const double* xq = x + (Idx)it[u].p * ld2 + 2 * it[u].q;
    f[u] = fma(-c[u].y, flip(ldd<kCg>(xq + oth(u)), sgn(u)), c[u].x * ldd<kCg>(xq + (1 - oth(u))));
  }
  if (R.dense) {
    // entry e: columns e + (e >= p) and e + (e >= q); h rho and rho h^dag in
    // sums of their own (one chain of both has 1.4 times the rounding error)
    double g[kN];
#pragma unroll
    for (int u = 0; u < kN; ++u) g[u] = 0.0;
    if (R.real) {
      const double* h = reinterpret_cast<const double*>(R.ent);
#pragma unroll(kN == 1 ? 4 : 2)
      for (int e = 0; e < W; ++e) {
        const double* he = h + (Idx)e * n;
#pragma unroll
        for (int u = 0; u < kN; ++u) {
          const int p = it[u].p, q = it[u].q;
          f[u] = fma(he[p], flip(ldd<kCg>(x + (Idx)(e + (e >= p)) * ld2 + 2 * q + oth(u)), sgn(u)), f[u]);
          g[u] = fma(-he[q], flip(ldd<kCg>(x + (Idx)p * ld2 + 2 * (e + (e >= q)) + oth(u)), sgn(u)), g[u]);
        }
      }
    } else {
#pragma unroll(kN == 1 ? 4 : 1)
      for (int e = 0; e < W; ++e) {
        const double2* he = R.ent + (Idx)e * n;
#pragma unroll
        for (int u = 0; u < kN; ++u) {
          const int p = it[u].p, q = it[u].q;
          const double2 a = he[p], b = he[q];
          const double2 r = ldz<kCg>(reinterpret_cast<const double2*>(x + (Idx)(e + (e >= p)) * ld2 + 2 * q));
          const double2 z = ldz<kCg>(reinterpret_cast<const double2*>(x + (Idx)p * ld2 + 2 * (e + (e >= q))));
          f[u] = fma(a.x, flip(it[u].im ? r.x : r.y, sgn(u)), f[u]);
          f[u] = fma(a.y, it[u].im ? r.y : r.x, f[u]);
          g[u] = fma(-b.x, flip(it[u].im ? z.x : z.y, sgn(u)), g[u]);
          g[u] = fma(b.y, it[u].im ? z.y : z.x, g[u]);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < kN; ++u) f[u] += g[u];
  } else if (R.real) {
#pragma unroll(kN == 1 ? 2 : 1)
    for (int e = 0; e < W; ++e) {
      const double2* ee = R.ent + e * n;
#pragma unroll
      for (int u = 0; u < kN; ++u) {
        const double2 a = ee[it[u].p], b = ee[it[u].q];
        f[u] = fma(a.x, flip(ldd<kCg>(x + __double2loint(a.y) + 2 * it[u].q + oth(u)), sgn(u)), f[u]);
        f[u] = fma(-b.x, flip(ldd<kCg>(x + (Idx)it[u].p * ld2 + __double2hiint(b.y) + oth(u)), sgn(u)), f[u]);
      }
    }
  } else {
#pragma unroll 1
    for (int e = 0; e < W; ++e) {
      const double2* ee = R.ent + e * n;
      const double* ye = R.hy + e * n;
#pragma unroll
      for (int u = 0; u < kN; ++u) {
        const double2 a = ee[it[u].p], b = ee[it[u].q];
        const double2 r = ldz<kCg>(reinterpret_cast<const double2*>(x + __double2loint(a.y) + 2 * it[u].q));
        const double2 z =
            ldz<kCg>(reinterpret_cast<const double2*>(x + (Idx)it[u].p * ld2 + __double2hiint(b.y)));
        f[u] = fma(a.x, flip(it[u].im ? r.x : r.y, sgn(u)), f[u]);
        f[u] = fma(ye[it[u].p], it[u].im ? r.y : r.x, f[u]);
        f[u] = fma(-b.x, flip(it[u].im ? z.x : z.y, sgn(u)), f[u]);
        f[u] = fma(ye[it[u].q], it[u].im ? z.y : z.x, f[u]);
      }
    }
  }
}

// Builds the rows of the matrix entry(i, c) with pattern nz(i, c) and
// im(i, c) (nonzero imaginary part); the whole CTA calls it, it ends
// synchronised.  v_s: vcap double2 of shared memory for the entries; v_g: n * n
// double2 of global memory, used by full rows that do not fit.  Rows become
// full when one has more than n / 2 entries or the lists do not fit v_s.
struct RowsBuild {
  int max_cnt, imag;
};

template <class Entry>
__device__ __forceinline__ void fill_row(const Rows& R, const Entry& entry, int i, int e, int c, int ld2, bool pad) {
  double2* ent = const_cast<double2*>(R.ent);
  const double2 h = pad ? cz() : entry(i, c);
  const int64_t at = (int64_t)e * R.n + i;
  if (R.dense) {
    if (R.real) reinterpret_cast<double*>(ent)[at] = h.x;
    else ent[at] = h;
  } else {
    ent[at] = make_double2(h.x, __hiloint2double(2 * c, c * ld2));
    if (!R.real) const_cast<double*>(R.hy)[at] = h.y;
  }
}

template <class Entry, class Nz, class Im>
__device__ Rows build_rows(const Entry& entry, const Nz& nz, const Im& im, int n, int ld2, double2* v_s, int vcap,
                           double2* v_g, double2* d_s, RowsBuild* S) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nw = blockDim.x >> 5;
  const bool small = n <= kRowsSmemMax;
  if (t == 0) S->max_cnt = S->imag = 0;
  __syncthreads();
  for (int i = warp; i < n; i += nw) {
    int k = 0;
    bool any = false;
    for (int c0 = 0; c0 < n; c0 += 32) {
      const int c = c0 + lane;
      const bool on = c < n && c != i && nz(i, c);
      any |= on && im(i, c);
      k += __popc(__ballot_sync(0xffffffffu, on));
    }
    any = __any_sync(0xffffffffu, any);
    if (lane == 0) {
      atomicMax(&S->max_cnt, k);
      if (any) atomicOr(&S->imag, 1);
    }
  }
  __syncthreads();
  const int mx = S->max_cnt;
  Rows R;
  R.n = n;
  R.real = S->imag == 0;
  // words of 8 bytes: 2 a sparse entry, 3 a complex one
  R.dense = !small || 2 * mx > n || (int64_t)mx * n * (R.real ? 2 : 3) > 2 * (int64_t)vcap;
  R.width = R.dense ? n - 1 : mx;
  const int64_t words = (int64_t)(n - 1) * n * (R.real ? 1 : 2);
  R.ent = (!R.dense || (small && words <= 2 * (int64_t)vcap)) ? v_s : v_g;
  R.hy = reinterpret_cast<const double*>(R.ent + (int64_t)mx * n);
  double2* d = small ? d_s : v_g + (int64_t)(n - 1) * n;
  R.d = d;
  for (int i = warp; i < n; i += nw) {
    int k = 0;
    for (int c0 = 0; c0 < n; c0 += 32) {
      const int c = c0 + lane;
      const bool on = c < n && c != i && (R.dense || nz(i, c));
      const unsigned b = __ballot_sync(0xffffffffu, on);
      if (on) fill_row(R, entry, i, k + __popc(b & ((1u << lane) - 1u)), c, ld2, false);
      k += __popc(b);
    }
    if (!R.dense)
      for (int e = k + lane; e < mx; e += 32) fill_row(R, entry, i, e, i, ld2, true);
    if (lane == 0) d[i] = entry(i, i);
  }
  __syncthreads();
  return R;
}

// The values of existing rows again (a driven generator); same CTA.
template <class Entry>
__device__ void refill_rows(const Rows& R, const Entry& entry, int ld2) {
  const int n = R.n;
  double2* d = const_cast<double2*>(R.d);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    for (int e = 0; e < R.width; ++e) {
      const int c = R.dense ? e + (e >= i) : __double2hiint(R.ent[(int64_t)e * n + i].y) / 2;
      fill_row(R, entry, i, e, c, ld2, !R.dense && c == i);
    }
    d[i] = entry(i, i);
  }
}

}  // namespace f64
}  // namespace lime
