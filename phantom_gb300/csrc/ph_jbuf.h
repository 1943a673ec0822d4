// Size rule of the j-side buffer of the symmetric pair passes (host code).
#pragma once
#include <algorithm>
#include <cstdint>

namespace ph {

// The passes store value v of trial row t at v stride + t (v < nj, t < rows)
// with the stride of the allocation, so what has to fit is nj strides, not nj
// times the rows of the call: the adjoint's 10 values follow the force's 7 in the
// buffer that the force's lists sized, and lists may shrink between calls.
struct JbufPlan {
  int64_t stride, doubles;
  bool keep;  // the held buffer serves the call as it is
};

inline JbufPlan jbuf_plan(int64_t held_stride, int64_t held_doubles, int64_t rows, int nj) {
  if (rows == 0 || (rows <= held_stride && nj * held_stride <= held_doubles)) return {held_stride, held_doubles, true};
  // room for 25 % more trial entries than this build has; a stride that serves
  // the rows is kept
  const int64_t stride = rows <= held_stride ? held_stride : rows + rows / 4 + 1024;
  return {stride, nj * stride, false};
}

}  // namespace ph
