// Host-side steps of a tick that the interpreter is slow at (no device code): Python lists into int32 staging memory.
//
// A decode tick hands over its sequences as dicts with lists of block ids, some thousands of ids in all; numpy converts forty to
// fifty a microsecond, which for one 2 000-block list or 32 short ones is as long as three projections of the tick.  Reading
// the objects directly takes 4 to 5 ns each and one call a tick: 1 x 2 047 blocks 44 us before, 8 here; 8 x 260 blocks 41 us,
// 8; 32 x 76 blocks 59 us, 12.  It needs the interpreter (loaded with ctypes.PyDLL); without Python's headers at build time the
// entry points are left out and the callers keep to numpy.  No counterpart in the reference, whose tick fills its inputs in
// Python (src/tilerl/decode_graph.py:112).
#include <stdint.h>
#include <string.h>

#include "common.cuh"

#if defined(__has_include)
#if __has_include(<Python.h>)
#define PY_SSIZE_T_CLEAN
#include <Python.h>

namespace {

// A plain integer in [lo, hi); false for anything else.
bool plain_int(PyObject* o, long lo, long hi, long* v) {
  if (o == nullptr || !PyLong_CheckExact(o)) return false;
  int over = 0;
  *v = PyLong_AsLongAndOverflow(o, &over);
  return over == 0 && *v >= lo && *v < hi;
}

}  // namespace

// The integers of a list or tuple -> dst[0 .. n).  Returns n, or -1 when `seq` is neither, holds anything but plain integers,
// or one outside [lo, hi); -2 when it is longer than `cap`.  Nothing is raised; dst may be partly written.
TRL_API long trl_list_i32(PyObject* seq, void* dst, long cap, long lo, long hi) {
  const bool list = PyList_CheckExact(seq);
  if (!list && !PyTuple_CheckExact(seq)) return -1;
  const Py_ssize_t n = list ? PyList_GET_SIZE(seq) : PyTuple_GET_SIZE(seq);
  if (n > cap) return -2;
  int32_t* d = static_cast<int32_t*>(dst);
  for (Py_ssize_t i = 0; i < n; ++i) {
    long v;
    if (!plain_int(list ? PyList_GET_ITEM(seq, i) : PyTuple_GET_ITEM(seq, i), lo, hi, &v)) return -1;
    d[i] = (int32_t)v;
  }
  return (long)n;
}

// Inputs of a captured decode tick: `seqs` a list of dicts {tokens: [id], start, blocks, slot}, `dst` the bucket's block
// [ids b][positions b][KV rows b][KV lengths b][state slots b][block table b x max_blocks], padding zero.  Returns the number of
// sequences, -1 when anything is not of that plain form or does not fit (the caller then goes the general way, which also
// raises what there is to raise).
TRL_API long trl_fill_decode(PyObject* seqs, void* dst, long b, long max_blocks, long kv_block) {
  if (!PyList_CheckExact(seqs) || PyList_GET_SIZE(seqs) > b) return -1;
  const long n = (long)PyList_GET_SIZE(seqs), top = 1L << 31;
  int32_t* a = static_cast<int32_t*>(dst);
  memset(a, 0, sizeof(int32_t) * (size_t)(5 * b + b * max_blocks));
  for (long r = 0; r < n; ++r) {
    PyObject* s = PyList_GET_ITEM(seqs, r);
    if (!PyDict_CheckExact(s)) return -1;
    PyObject* toks = PyDict_GetItemString(s, "tokens");
    PyObject* blocks = PyDict_GetItemString(s, "blocks");
    long tok, pos, slot;
    if (toks == nullptr || blocks == nullptr || !PyList_CheckExact(toks) || PyList_GET_SIZE(toks) != 1) return -1;
    if (!plain_int(PyList_GET_ITEM(toks, 0), 0, top, &tok) || !plain_int(PyDict_GetItemString(s, "start"), 0, top - 1, &pos) ||
        !plain_int(PyDict_GetItemString(s, "slot"), 0, top, &slot))
      return -1;
    int32_t* row = a + 5 * b + r * max_blocks;
    const long nb = trl_list_i32(blocks, row, max_blocks, 0, top / kv_block);
    if (nb < 0 || pos / kv_block >= nb) return -1;
    a[r] = (int32_t)tok, a[b + r] = (int32_t)pos;
    a[2 * b + r] = (int32_t)(row[pos / kv_block] * kv_block + pos % kv_block);
    a[3 * b + r] = (int32_t)(pos + 1), a[4 * b + r] = (int32_t)slot;
  }
  return n;
}
#endif
#endif
