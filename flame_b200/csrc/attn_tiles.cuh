// The work list of the attention kernels: 128-row tiles of packed documents, built once per batch (fb_attn_tile_list): one
// int32 array of 3 nseq + 2,
//
//   int32 [nseq + 1]  prefix sum of the tiles of the documents, in their order (VarlenMeta.tile_offsets; no kernel reads it)
//   int32 [nseq + 1]  the same over the documents by falling length
//   int32 [nseq]      those documents
//
// CTAs take long documents first, inside a document the tiles with the longest walk first, and the heads of a tile side by side:
// the last CTAs to start are the shortest, and a document's keys and values stay in L2 while its tiles are worked on.  With
// a grid of tiles x heads in the order of the rows the last head's long walks started last: an SM of the head-dim-64 forward
// was idle 9 % of the time at 32,768 tokens, of the stick-breaking forward 20 % at 8,192.  Attention layer at 65,536 tokens 4.40 ->
// 4.33 ms under the power cap, stick-breaking layer at 32,768 4.30 -> 4.20 ms.
#pragma once

// largest i in [0, n) with offs[i] <= x
__device__ __forceinline__ int upper_doc(const int* __restrict__ offs, int n, int x) {
  int lo = 0, hi = n;
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (offs[mid] <= x) lo = mid; else hi = mid;
  }
  return lo;
}

// This CTA's head, document and tile of it, of a grid of heads x tiles; `late`: tiles at the document's end walk longest.
__device__ __forceinline__ bool attn_tile(const int* __restrict__ list, int nseq, int heads, bool late, int& head, int& doc, int& tile) {
  const int* sorted = list + nseq + 1;
  const int rank = (int)(blockIdx.x / (unsigned)heads);
  head = (int)(blockIdx.x % (unsigned)heads);
  if (rank >= sorted[nseq]) return false;
  const int i = upper_doc(sorted, nseq + 1, rank);
  doc = sorted[nseq + 1 + i];
  tile = late ? sorted[i + 1] - 1 - rank : rank - sorted[i];
  return true;
}
