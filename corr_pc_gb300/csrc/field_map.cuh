// field_map.cuh -- which of the 13 output fields each corel accumulates in the
// block histograms of the pair kernels.
#pragma once

#include "cpc_device.cuh"

namespace cpc {

// Per corel: the main fields m(k), k < FM, the jackknife fields j(g), g < FJ, and
// jm(g), the main slot holding jackknife field g (m(jm(g)) == j(g)).  FA, a(i):
// the main slots whose terms differ between the two orders of a pair whose
// galaxies carry the same data in either role (twin jobs); the others are the
// same in both orders.  Twin jobs run the corels with FA = 0 and shape_shape.
struct NoAsym {
  static constexpr int FA = 0;
  __host__ __device__ static constexpr int a(int) { return -1; }
};
template <int C> struct FieldMap;
template <> struct FieldMap<COREL_DD> : NoAsym {
  static constexpr int FM = 1, FJ = 1;
  __host__ __device__ static constexpr int m(int) { return 0; }
  __host__ __device__ static constexpr int j(int) { return 0; }
  __host__ __device__ static constexpr int jm(int) { return 0; }
};
template <> struct FieldMap<COREL_SD> : NoAsym {
  static constexpr int FM = 7, FJ = 4;
  __host__ __device__ static constexpr int m(int k) {
    return k == 0 ? 0 : k == 1 ? 1 : k == 2 ? 2 : k == 3 ? 3 : k == 4 ? 4 : k == 5 ? 11 : 12;
  }
  __host__ __device__ static constexpr int j(int k) { return k == 0 ? 0 : k == 1 ? 1 : k == 2 ? 3 : 11; }
  __host__ __device__ static constexpr int jm(int g) { return g == 0 ? 0 : g == 1 ? 1 : g == 2 ? 3 : 5; }
};
template <> struct FieldMap<COREL_SS> {
  static constexpr int FM = 11, FJ = 6;
  __host__ __device__ static constexpr int m(int k) { return k < 2 ? k : k == 2 ? 2 : k + 2; }
  __host__ __device__ static constexpr int j(int k) { return k == 0 ? 0 : 2 * k - 1 + (k >= 2 ? 2 : 0); }
  __host__ __device__ static constexpr int jm(int g) { return g == 0 ? 0 : 2 * g - 1; }
  // estimator 0: e+ of the shape holder (data[1]) and its square, the phi term
  // (data[6]) and its square: fields 1, 2, 11, 12
  static constexpr int FA = 4;
  __host__ __device__ static constexpr int a(int i) { return i == 0 ? 1 : i == 1 ? 2 : i == 2 ? 9 : 10; }
};
template <> struct FieldMap<COREL_SSA> : NoAsym {
  static constexpr int FM = 13, FJ = 7;
  __host__ __device__ static constexpr int m(int k) { return k; }
  __host__ __device__ static constexpr int j(int k) { return k == 0 ? 0 : 2 * k - 1; }
  __host__ __device__ static constexpr int jm(int g) { return g == 0 ? 0 : 2 * g - 1; }
};
// density_convergence: wt, data[1].val
template <> struct FieldMap<COREL_DK> : NoAsym {
  static constexpr int FM = 2, FJ = 2;
  __host__ __device__ static constexpr int m(int k) { return k; }
  __host__ __device__ static constexpr int j(int k) { return k; }
  __host__ __device__ static constexpr int jm(int g) { return g; }
};
// shape_convergence: wt, data[1].val, data[3].val, data[5].val
template <> struct FieldMap<COREL_SK> : NoAsym {
  static constexpr int FM = 4, FJ = 4;
  __host__ __device__ static constexpr int m(int k) { return k == 0 ? 0 : k == 1 ? 1 : k == 2 ? 5 : 9; }
  __host__ __device__ static constexpr int j(int k) { return k == 0 ? 0 : k == 1 ? 1 : k == 2 ? 5 : 9; }
  __host__ __device__ static constexpr int jm(int g) { return g; }
};
// ED: wt, data[6].val, data[6].err (regions: wt, data[6].val)
template <> struct FieldMap<COREL_ED> : NoAsym {
  static constexpr int FM = 3, FJ = 2;
  __host__ __device__ static constexpr int m(int k) { return k == 0 ? 0 : k == 1 ? 11 : 12; }
  __host__ __device__ static constexpr int j(int k) { return k == 0 ? 0 : 11; }
  __host__ __device__ static constexpr int jm(int g) { return g; }
};

template <class FM, int G = 0>
constexpr bool jm_consistent() {
  if constexpr (G >= FM::FJ) {
    return true;
  } else {
    return FM::m(FM::jm(G)) == FM::j(G) && jm_consistent<FM, G + 1>();
  }
}
// position of main slot k among the order-dependent slots a(i), or -1
template <class FM>
__host__ __device__ constexpr int asym_pos(int k) {
  for (int i = 0; i < FM::FA; i++)
    if (FM::a(i) == k) return i;
  return -1;
}
static_assert(FieldMap<COREL_SS>::m(FieldMap<COREL_SS>::a(0)) == 1 &&
                  FieldMap<COREL_SS>::m(FieldMap<COREL_SS>::a(1)) == 2 &&
                  FieldMap<COREL_SS>::m(FieldMap<COREL_SS>::a(2)) == 11 &&
                  FieldMap<COREL_SS>::m(FieldMap<COREL_SS>::a(3)) == 12,
              "order-dependent shape_shape fields");
static_assert(jm_consistent<FieldMap<COREL_DD>>() && jm_consistent<FieldMap<COREL_SD>>() &&
                  jm_consistent<FieldMap<COREL_SS>>() && jm_consistent<FieldMap<COREL_SSA>>() &&
                  jm_consistent<FieldMap<COREL_DK>>() && jm_consistent<FieldMap<COREL_SK>>() &&
                  jm_consistent<FieldMap<COREL_ED>>(),
              "jackknife fields must map onto main slots");

}  // namespace cpc
