// The rule that says which K and V tensors the four-row TMA gather can address (host code without CUDA, so that a test can
// compile it alone).
#pragma once

#include <stdint.h>

namespace lvar {

// A [B, H, L, D] view as a 2-D tensor of rows: key l of (b, h) is row b * rb + h * rh + l, from column h * ch on.  Not ok where
// batches are not whole rows apart, or heads neither whole rows apart nor side by side in a row.
struct RowsView {
  bool ok;
  int rb, rh, ch;
  int64_t rows, width;
};
inline RowsView rows_view(int B, int H, int L, int D, int64_t sb, int64_t sh, int64_t sl) {
  RowsView r = {};
  if (sl < D || (B > 1 && sb % sl != 0)) return r;
  const int64_t rb = B > 1 ? sb / sl : 0;
  int64_t rh = 0, ch = 0;
  if (H > 1) {
    if (sh % sl == 0) rh = sh / sl;
    else if ((H - 1) * sh + D <= sl) ch = sh;
    else return r;
  }
  r.rows = (B - 1) * rb + (H - 1) * rh + L;
  r.width = (H - 1) * ch + D;
  if (r.rows > 0x7fffffff || r.width > 0x7fffffff || sl * 2 >= (1ll << 40)) return r;
  r.rb = (int)rb;
  r.rh = (int)rh;
  r.ch = (int)ch;
  r.ok = true;
  return r;
}

}  // namespace lvar
