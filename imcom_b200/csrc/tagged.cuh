// tagged.cuh -- values exchanged between CTAs of one cooperative grid as
// 16-byte {value, tag} records: a record is written and read as one 128-bit
// access, so a reader polls the data itself and needs no fence, flag or
// barrier.  A poll that does not succeed within a limit reports an error.
#pragma once

#include <cuda_runtime.h>

namespace imcom {

__device__ __forceinline__ void st_tagged(ulonglong2* p, double v, unsigned tag) {
  asm volatile(
      "{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}\n" ::"l"(p),
      "l"(__double_as_longlong(v)), "l"((unsigned long long)tag)
      : "memory");
}

__device__ __forceinline__ ulonglong2 ld_tagged(const ulonglong2* p) {
  ulonglong2 r;
  asm volatile(
      "{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}\n"
      : "=l"(r.x), "=l"(r.y)
      : "l"(p)
      : "memory");
  return r;
}

// Bounds a poll loop: false once `limit` rounds have passed or another thread
// of the grid has failed (the error word is then set).
__device__ __forceinline__ bool poll_again(int& it, long long limit, int* err) {
  if ((++it & 31) != 0) return true;
  if (it <= limit && !*(volatile int*)err) return true;
  atomicExch(err, 1);
  return false;
}

// Polls N records at once: p(u) the u-th record, on(u) whether it is wanted
// (else its value is 0).  False if they did not all come.
template <int N, class P, class On>
__device__ __forceinline__ bool poll_records(P p, On on, unsigned tag, double (&out)[N],
                                             long long limit, int* err) {
  unsigned miss = 0;
#pragma unroll
  for (int u = 0; u < N; ++u) {
    out[u] = 0.0;
    if (on(u)) miss |= 1u << u;
  }
  for (int it = 0; miss;) {
    ulonglong2 t[N];
#pragma unroll
    for (int u = 0; u < N; ++u)
      if (miss & (1u << u)) t[u] = ld_tagged(p(u));
#pragma unroll
    for (int u = 0; u < N; ++u)
      if ((miss & (1u << u)) && (unsigned)t[u].y == tag) {
        out[u] = __longlong_as_double((long long)t[u].x);
        miss &= ~(1u << u);
      }
    if (miss && !poll_again(it, limit, err)) return false;
  }
  return true;
}

}  // namespace imcom
