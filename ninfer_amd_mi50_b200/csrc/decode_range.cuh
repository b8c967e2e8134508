// The key range of one decode row, shared by the kernels of attention_decode.cu and
// attention_decode_stream.cu so that they agree on which blocks of 128 keys a row has.
#pragma once

namespace nf {

// Row at position `pos` with `window` (0: none) and a workspace of `nsplit` blocks of `block`
// keys: sets lo..pos to the keys the row reads.  A position that needs a block beyond the
// workspace is cut to the workspace's last key (and lo to at most that), so that every block in
// [lo / block, pos / block] exists and holds a key; returns true when it had to cut.
__device__ __forceinline__ bool decode_key_range(int& pos, int& lo, int window, int nsplit, int block) {
  lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
  const int most = nsplit * block - 1;
  if (pos <= most) return false;
  pos = most;
  if (lo > pos) lo = pos;
  return true;
}

// The keys of a row with a window that keeps the request's first `keep_first` keys visible: those below `kept`, and
// lo..pos.  Its blocks, in ascending order: the `before` that hold kept keys and lie before the window's first, and the window's.
struct KeptRange {
  int lo, kept, before, first, blocks;
  __device__ __forceinline__ int block(int i) const { return i < before ? i : first + i - before; }
};
__device__ __forceinline__ KeptRange kept_key_range(int pos, int window, int keep_first, int block) {
  KeptRange r;
  r.lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
  r.kept = min(keep_first, r.lo);
  r.first = r.lo / block;
  r.before = min(r.first, (r.kept + block - 1) / block);
  r.blocks = r.before + pos / block - r.first + 1;
  return r;
}

}  // namespace nf
