// Where one (batch, head) of a mixed-attention call finds its tensors.
#pragma once
#include "saf_internal.h"

namespace saf {

struct HeadIdx {
  int b, h, state, hq, hk, hv, hp;
};

__device__ __forceinline__ HeadIdx head_index(const SafMixedAttnArgs& a, int bh) {
  HeadIdx x;
  x.b = bh / a.H;
  x.h = bh % a.H;
  x.state = a.force_state >= 0 ? a.force_state : a.frozen[x.h];
  x.hq = a.hidx ? a.hidx[x.h] : x.h;
  if (a.HKV > 0) {
    x.hk = x.hv = a.kvidx ? a.kvidx[x.h] : 0;
  } else {
    x.hk = x.hq;
    x.hv = x.h;
  }
  x.hp = a.pidx ? a.pidx[x.h] : x.h;
  return x;
}

}  // namespace saf
