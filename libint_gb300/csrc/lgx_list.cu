// Classification of explicit quartet lists on the GPU: from the caller's
// quartets and offsets to work items grouped by (class, precision, contraction
// depth), the order in which the class launches read them.
//
// What bounds it: one read of the list (24 bytes a quartet) and one write of
// the items (24 bytes); on the host the same took 5.5 ms for 692,076 and 13 ms
// for 1.1 million quartets, as long as their integrals (whole calls: 11.9 ->
// 4.2 ms and 19.3 -> 3.1 ms).  Within a class the
// items are ordered deepest contraction first: the lanes of a warp then run
// equally many primitive quartets, and the longest chains start first.
#include "lgx_kernels.cuh"

namespace lgx {

namespace {

// Canonical quartet (the rule of canonicalize, lgx_api.cu; engine.impl.h:
// 1181-1211), its class key and the values of its sets.
__device__ __forceinline__ bool list_item(const ListArgs& a, long long i, QuartetItem& it,
                                          int& key, long long& nv, long long& nq) {
  const int4 q4 = a.q[i];
  const int s[4] = {q4.x, q4.y, q4.z, q4.w};
  int l[4], np[4];
  nv = a.nsets;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (s[k] < 0 || s[k] >= a.b.nshell) return false;
    l[k] = a.b.l[s[k]];
    np[k] = a.b.nprim[s[k]];
    nv *= a.b.pure[s[k]] ? 2 * l[k] + 1 : ncart_of(l[k]);
  }
  const bool stb = l[0] < l[1], stk = l[2] < l[3], sbk = l[0] + l[1] > l[2] + l[3];
  // canonical bra = caller's bra, or ket when the pairs are exchanged
  const int b0 = sbk ? 2 : 0, k0 = sbk ? 0 : 2;
  const bool tb = sbk ? stk : stb, tk = sbk ? stb : stk;
  const int c0 = tb ? s[b0 + 1] : s[b0], c1 = tb ? s[b0] : s[b0 + 1];
  const int c2 = tk ? s[k0 + 1] : s[k0], c3 = tk ? s[k0] : s[k0 + 1];
  const int l0 = tb ? l[b0 + 1] : l[b0], l1 = tb ? l[b0] : l[b0 + 1];
  const int l2 = tk ? l[k0 + 1] : l[k0], l3 = tk ? l[k0] : l[k0 + 1];
  const bool bsw = c0 < c1, ksw = c2 < c3;  // stored pairs have s1 >= s2
  const long long bh = max(c0, c1), bl = min(c0, c1), kh = max(c2, c3), kl = min(c2, c3);
  it.bra_pair = int(bh * (bh + 1) / 2 + bl);
  it.ket_pair = int(kh * (kh + 1) / 2 + kl);
  it.flags = (bsw ? 1 : 0) | (ksw ? 2 : 0) | ((sbk ? 1 : 0) | (stb ? 2 : 0) | (stk ? 4 : 0)) << 2;
  it.pad = int(i);
  it.out = a.off ? a.off[i] : i;
  const int ci = a.tab[((l0 * kListLK + l1) * kListLK + l2) * kListLK + l3];
  nq = (long long)(np[0] * np[1]) * (np[2] * np[3]);
  int fp32 = 0;
  if (a.kpair) fp32 = a.kpair[it.bra_pair] * a.kpair[it.ket_pair] < a.mixed ? 1 : 0;
  const int depth = 63 - __clzll(nq);  // nq in [2^depth, 2^(depth + 1))
  key = (ci * 2 + fp32) * kListDepth + (kListDepth - 1 - min(depth, kListDepth - 1));
  return true;
}

// Counts per key, primitive quartets per (class, precision), the end of the
// furthest set, and whether a shell index is out of range.
__global__ void __launch_bounds__(256) list_count_kernel(ListArgs a) {
  extern __shared__ unsigned s_hist[];
  for (int k = threadIdx.x; k < a.nkeys; k += blockDim.x) s_hist[k] = 0;
  __syncthreads();
  unsigned long long need = 0;
  bool bad = false;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < a.n;
       i += (long long)gridDim.x * blockDim.x) {
    QuartetItem it;
    int key;
    long long nv, nq;
    if (!list_item(a, i, it, key, nv, nq)) {
      bad = true;
      continue;
    }
    a.keys[i] = (unsigned short)key;
    atomicAdd(&s_hist[key], 1u);
    // lanes with the same class add once
    const unsigned act = __activemask();
    const int cls = key / kListDepth;
    const unsigned same = __match_any_sync(act, cls);
    const unsigned sum = __reduce_add_sync(same, unsigned(nq));
    if ((threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(a.nqsum + cls, (unsigned long long)sum);
    const unsigned long long end = (unsigned long long)(it.out + nv);
    need = end > need ? end : need;
  }
  if (need) atomicMax(a.stat, need);
  if (bad) atomicExch(a.stat + 1, 1ull);
  __syncthreads();
  for (int k = threadIdx.x; k < a.nkeys; k += blockDim.x)
    if (s_hist[k]) atomicAdd(a.hist + k, s_hist[k]);
}

// Items to their places: the lanes of a warp that share a key reserve a run of
// that key's range (cursor) together.
__global__ void __launch_bounds__(256) list_scatter_kernel(ListArgs a) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  QuartetItem it;
  int key;
  long long nv, nq;
  if (!list_item(a, i, it, key, nv, nq)) return;
  key = a.keys[i];
  const int lane = threadIdx.x & 31;
  const unsigned same = __match_any_sync(__activemask(), key);
  const int lead = __ffs(same) - 1;
  unsigned at = 0;
  if (lane == lead) at = atomicAdd(a.hist + key, (unsigned)__popc(same));
  at = __shfl_sync(same, at, lead) + __popc(same & ((1u << lane) - 1u));
  a.items[at] = it;
}

}  // namespace

cudaError_t launch_list_count(const ListArgs& a, int nsm, cudaStream_t st) {
  const int block = 256;
  const long long need = (a.n + block - 1) / block;
  const int grid = int(need < 4LL * nsm ? need : 4LL * nsm);
  list_count_kernel<<<grid, block, size_t(a.nkeys) * sizeof(unsigned), st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_list_scatter(const ListArgs& a, cudaStream_t st) {
  const int block = 256;
  list_scatter_kernel<<<(unsigned)((a.n + block - 1) / block), block, 0, st>>>(a);
  return cudaGetLastError();
}

}  // namespace lgx
