// The order of a dof column's records in a gather layout. A first transposed apply
// builds such a layout (C48 x 70 W2: 41 k columns of one or two records), where
// std::stable_sort allocated scratch memory for each column.
#pragma once

#include <algorithm>
#include <vector>

namespace lfx {

// stable, by less: few records by insertion
template <class R, class Less>
void stable_order(std::vector<R>& v, Less less) {
  if (v.size() > 32) {
    std::stable_sort(v.begin(), v.end(), less);
    return;
  }
  for (size_t i = 1; i < v.size(); ++i) {
    const R x = v[i];
    size_t j = i;
    for (; j > 0 && less(x, v[j - 1]); --j) v[j] = v[j - 1];
    v[j] = x;
  }
}

}  // namespace lfx
