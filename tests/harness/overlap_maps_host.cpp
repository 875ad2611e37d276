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
