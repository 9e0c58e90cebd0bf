// bc_offset.h -- the angular offsets of the non-reflecting edges: which cells
// they reach.  Plain C++, for the boundary kernel and for tests on the host.
#pragma once

#ifdef __CUDACC__
#define BC_HD __host__ __device__ __forceinline__
#else
#define BC_HD inline
#endif

// The sector that an offset leads to from sector j, with the reference's one
// wrap (Kernels.cu:676-702): inside the ring while |off| <= nsec, else a cell
// counted from the ring's start that lies in another ring.
BC_HD int bc_wrap(int j, int off, int nsec) {
  int jp = j + off;
  if (jp >= nsec) jp -= nsec;
  if (jp < 0) jp += nsec;
  return jp;
}

// How a call's offsets (of the inner and the outer edge, in sectors, before
// their truncation to int) can be applied.
enum BcReach {
  kBcInRing,    // every target in its ring
  kBcInRows,    // targets in other rings, all inside the (nrad + 1) * nsec cells
  kBcOutside,   // some target outside the fields
  kBcNotFinite  // no offset at all: a NaN in the sound speed of an edge ring
};
BC_HD BcReach bc_reach(double a, double a2, int nrad, int nsec) {
  if (!(a == a) || !(a2 == a2)) return kBcNotFinite;
  const double far = 1.0e9;  // within int, sums with a sector too; infinite offsets end here
  if (!(a > -far && a < far && a2 > -far && a2 < far)) return kBcOutside;
  const long long n = nsec, in = (int)a, out = -(long long)(int)a2;  // out: what is added to j
  if (in >= -n && in <= n && out >= -n && out <= n) return kBcInRing;
  const long long cells = (nrad + 1LL) * n, ring = (nrad - 2LL) * n;
  // the cells first .. last that sectors 0 .. nsec-1 lead to, from the ring's start
  const long long in0 = in > n ? in - n : in < -n ? in + n : 0, in1 = in > n || in < -n ? in0 + n - 1 : n - 1;
  const long long out0 = out > n ? out - n : out < -n ? out + n : 0,
                  out1 = out > n || out < -n ? out0 + n - 1 : n - 1;
  return in0 >= 0 && in1 < cells && ring + out0 >= 0 && ring + out1 < cells ? kBcInRows : kBcOutside;
}
