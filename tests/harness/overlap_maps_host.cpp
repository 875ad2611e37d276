// Host build of the operand aliasing test (mref_overlap) for operands with
// class maps of their own, for its CPU test.
#include <math.h>

#include "../../skkr_budapest_gb300/csrc/common.cuh"

// operands base + off (elements of one allocation), common strides sk / sc and
// ld, a class map each; mref_overlap for nk x nc items of `cols` columns
extern "C" int overlap_maps_eval(long long offa, const int *mapa, long long offb, const int *mapb, long long sk,
                                 long long sc, int ld, int nk, int nc, int cols) {
  static zd pool[1];
  return mref_overlap(mref_map(pool + offa, sk, sc, ld, mapa, nc), mref_map(pool + offb, sk, sc, ld, mapb, nc), nk,
                      nc, cols)
             ? 1
             : 0;
}

// operands of rows_a and rows_b rows, identity maps
extern "C" int overlap_rows_eval(long long offa, int rows_a, long long offb, int rows_b, long long sk, long long sc,
                                 int ld, int nk, int nc, int cols) {
  static zd pool[1];
  return mref_overlap(mref(pool + offa, sk, sc, ld), mref(pool + offb, sk, sc, ld), nk, nc, cols, rows_a, rows_b) ? 1
                                                                                                                 : 0;
}
