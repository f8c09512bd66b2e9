// TVMBackendPackedCFunc entry points: decode and validate the packed arguments the way the
// host stub generated by the reference does (src/tir/transforms/make_packed_api.cc:244-305,
// src/tir/transforms/arg_binder.cc:172-282), then call the plain-pointer launchers.
#include <cmath>
#include <vector>

#include "common.h"

namespace {

using sptir::fail;

struct Packed {
  const char* fn;
  TVMValue* v;
  int* tc;
  int n;
  int device_id = -1;

  bool is_tensor(int i) const {
    return i < n && (tc[i] == kTVMDLTensorHandle || tc[i] == kTVMNDArrayHandle ||
                     tc[i] == kTVMOpaqueHandle);
  }

  // A flat, compact, 1-D device tensor of the given element type.
  int tensor(int i, const char* name, uint8_t code, uint8_t bits, void** data, int64_t* len) {
    if (i >= n) return fail("%s: missing argument %d (%s)", fn, i, name);
    if (!is_tensor(i)) {
      if (tc[i] == kTVMNullptr) return fail("%s: argument %s is a null handle", fn, name);
      return fail("%s: Expect arg[%d] (%s) to be pointer, got type code %d", fn, i, name, tc[i]);
    }
    const DLTensor* t = static_cast<const DLTensor*>(v[i].v_handle);
    if (t == nullptr) return fail("%s: argument %s is a null DLTensor", fn, name);
    if (t->ndim != 1)
      return fail("%s: %s.ndim is expected to equal 1 (flat buffer), got %d", fn, name, t->ndim);
    if (t->dtype.code != code || t->dtype.bits != bits || t->dtype.lanes != 1)
      return fail("%s: %s.dtype is expected to be %s%d, got code=%d bits=%d lanes=%d", fn, name,
                  code == kDLFloat ? "float" : (code == kDLInt ? "int" : "uint"), bits,
                  t->dtype.code, t->dtype.bits, t->dtype.lanes);
    if (t->strides != nullptr && t->shape[0] > 1 && t->strides[0] != 1)
      return fail("%s: %s.strides: expected to be compact array", fn, name);
    if (t->byte_offset != 0)
      return fail("%s: %s.byte_offset is expected to be 0, got %llu", fn, name,
                  static_cast<unsigned long long>(t->byte_offset));
    if (t->shape[0] < 0) return fail("%s: %s has negative extent", fn, name);
    if (t->device.device_type != kDLCUDA)
      return fail("%s: %s.device_type is expected to be CUDA (2), got %d; this library has no "
                  "CPU path", fn, name, t->device.device_type);
    if (device_id < 0) device_id = t->device.device_id;
    if (t->device.device_id != device_id)
      return fail("%s: %s.device_id is expected to equal %d, got %d", fn, name, device_id,
                  t->device.device_id);
    if (t->data == nullptr && t->shape[0] > 0)
      return fail("%s: %s has a null data pointer", fn, name);
    *data = t->data;
    *len = t->shape[0];
    return 0;
  }

  int integer(int i, const char* name, int64_t* out) {
    if (i >= n) return fail("%s: missing argument %d (%s)", fn, i, name);
    if (tc[i] != kTVMArgInt)
      return fail("%s: Expect arg[%d] (%s) to be int, got type code %d", fn, i, name, tc[i]);
    *out = v[i].v_int64;
    return 0;
  }
};

int check_len(const char* fn, const char* name, int64_t got, int64_t want) {
  if (got != want)
    return fail("%s: Argument %s.shape[0] has an unsatisfied constraint: %lld == %lld", fn, name,
                static_cast<long long>(got), static_cast<long long>(want));
  return 0;
}

int fits_i32(const char* fn, const char* name, int64_t x) {
  if (x < 0 || x > INT32_MAX) return fail("%s: %s = %lld does not fit int32", fn, name, (long long)x);
  return 0;
}

#define TRY(expr)            \
  do {                       \
    if ((expr) != 0) return -1; \
  } while (0)

void set_void_return(TVMValue* ret, int* ret_tc) {
  if (ret) ret->v_int64 = 0;
  if (ret_tc) *ret_tc = kTVMNullptr;
}

}  // namespace

extern "C" {

int sparsetir_csrmm(SPARSETIR_PACKED_ARGS) {
  (void)resource_handle;
  Packed p{"sparsetir_csrmm", args, type_codes, num_args};
  if (num_args != 5 && num_args != 9)
    return fail("sparsetir_csrmm: num_args should be 5 or 9, got %d", num_args);
  void *a = nullptr, *b = nullptr, *c = nullptr, *indptr = nullptr, *indices = nullptr;
  int64_t la = 0, lb = 0, lc = 0, lp = 0, li = 0;
  TRY(p.tensor(0, "a", kDLFloat, 32, &a, &la));
  TRY(p.tensor(1, "b", kDLFloat, 32, &b, &lb));
  TRY(p.tensor(2, "c", kDLFloat, 32, &c, &lc));
  TRY(p.tensor(3, "indptr", kDLInt, 32, &indptr, &lp));
  TRY(p.tensor(4, "indices", kDLInt, 32, &indices, &li));
  int64_t m = 0, n = 0, feat = 0, nnz = 0;
  if (num_args == 9) {
    TRY(p.integer(5, "m", &m));
    TRY(p.integer(6, "n", &n));
    TRY(p.integer(7, "feat_size", &feat));
    TRY(p.integer(8, "nnz", &nnz));
  } else {
    m = lp - 1;
    nnz = la;
    if (m < 1) return fail("sparsetir_csrmm: cannot infer feat_size with m = %lld", (long long)m);
    if (lc % m != 0) return fail("sparsetir_csrmm: len(c) is not a multiple of m");
    feat = lc / m;
    if (feat == 0 || lb % feat != 0)
      return fail("sparsetir_csrmm: len(b) is not a multiple of feat_size");
    n = lb / feat;
  }
  TRY(fits_i32(p.fn, "m", m)); TRY(fits_i32(p.fn, "n", n));
  TRY(fits_i32(p.fn, "feat_size", feat)); TRY(fits_i32(p.fn, "nnz", nnz));
  TRY(check_len(p.fn, "a", la, nnz));
  TRY(check_len(p.fn, "b", lb, n * feat));
  TRY(check_len(p.fn, "c", lc, m * feat));
  TRY(check_len(p.fn, "indptr", lp, m + 1));
  TRY(check_len(p.fn, "indices", li, nnz));
  set_void_return(out_ret_value, out_ret_tcode);
  return sparsetir_csrmm_raw(static_cast<const float*>(a), static_cast<const float*>(b),
                             static_cast<float*>(c), static_cast<const int32_t*>(indptr),
                             static_cast<const int32_t*>(indices), (int)m, (int)n, (int)feat,
                             (int)nnz, p.device_id, sptir::stream_for(p.device_id));
}

// sparsetir_hyb_spmm and, with `with_peers`, sparsetir_hyb_spmm_peers (feat_size and flags are
// then followed by one integer per peer: the address of that peer's copy of c).
static int hyb_packed(const char* fn, bool with_peers, SPARSETIR_PACKED_ARGS) {
  (void)resource_handle;
  Packed p{fn, args, type_codes, num_args};
  int nt = 0;
  while (p.is_tensor(nt)) ++nt;
  int ns = num_args - nt;
  if (nt < 2 || (nt - 2) % 3 != 0)
    return fail("%s: expected (b, c, {w, rows, cols} x K, feat_size[, flags]%s); "
                "got %d tensor arguments", fn, with_peers ? ", peer_c..." : "", nt);
  std::vector<void*> peer_c;
  if (with_peers) {
    if (ns < 3 || ns > 2 + SPARSETIR_MAX_PEERS)
      return fail("%s: expected feat_size, flags and 1 to %d peer addresses after the tensors, got %d "
                  "scalar arguments", fn, SPARSETIR_MAX_PEERS, ns);
    for (int k = 2; k < ns; ++k) {
      int64_t addr = 0;
      TRY(p.integer(nt + k, "peer_c", &addr));
      peer_c.push_back(reinterpret_cast<void*>(static_cast<intptr_t>(addr)));
    }
    ns = 2;
  }
  if (ns < 1 || ns > 2)
    return fail("sparsetir_hyb_spmm: expected feat_size [and flags] after the tensors, got %d "
                "scalar arguments", ns);
  int K = (nt - 2) / 3;
  if (K > SPARSETIR_HYB_MAX_BUCKETS)
    return fail("sparsetir_hyb_spmm: %d buckets exceed the maximum of %d", K,
                SPARSETIR_HYB_MAX_BUCKETS);
  void *b = nullptr, *c = nullptr;
  int64_t lb = 0, lc = 0, feat = 0, flags = 0;
  TRY(p.tensor(0, "b", kDLFloat, 32, &b, &lb));
  TRY(p.tensor(1, "c", kDLFloat, 32, &c, &lc));
  TRY(p.integer(nt, "feat_size", &feat));
  if (ns == 2) TRY(p.integer(nt + 1, "flags", &flags));
  if (feat <= 0) return fail("sparsetir_hyb_spmm: feat_size must be positive");
  if (lb % feat != 0 || lc % feat != 0)
    return fail("sparsetir_hyb_spmm: len(b) and len(c) must be multiples of feat_size");
  TRY(fits_i32(p.fn, "feat_size", feat));
  TRY(fits_i32(p.fn, "m", lc / feat)); TRY(fits_i32(p.fn, "n", lb / feat));
  std::vector<SparsetirEllBucket> bk(K);
  for (int q = 0; q < K; ++q) {
    void *w = nullptr, *rows = nullptr, *cols = nullptr;
    int64_t lw = 0, lr = 0, lcol = 0;
    TRY(p.tensor(2 + 3 * q, "w", kDLFloat, 32, &w, &lw));
    TRY(p.tensor(3 + 3 * q, "rows", kDLInt, 32, &rows, &lr));
    TRY(p.tensor(4 + 3 * q, "cols", kDLInt, 32, &cols, &lcol));
    TRY(check_len(p.fn, "w", lw, lcol));
    int64_t width = 0;
    if (lr > 0) {
      if (lcol % lr != 0 || lcol == 0)
        return fail("sparsetir_hyb_spmm: bucket %d: len(cols) = %lld is not a positive multiple "
                    "of len(rows) = %lld", q, (long long)lcol, (long long)lr);
      width = lcol / lr;
    } else if (lcol != 0) {
      return fail("sparsetir_hyb_spmm: bucket %d has columns but no rows", q);
    }
    TRY(fits_i32(p.fn, "nrows", lr)); TRY(fits_i32(p.fn, "width", width));
    bk[q] = SparsetirEllBucket{static_cast<const float*>(w), static_cast<const int32_t*>(rows),
                               static_cast<const int32_t*>(cols), (int32_t)lr, (int32_t)width};
  }
  set_void_return(out_ret_value, out_ret_tcode);
  if (with_peers)
    return sparsetir_hyb_spmm_peers_raw(static_cast<const float*>(b), static_cast<float*>(c), bk.data(), K,
                                        (int)(lc / feat), (int)(lb / feat), (int)feat, (int)flags,
                                        (int)peer_c.size(), peer_c.data(), p.device_id,
                                        sptir::stream_for(p.device_id));
  return sparsetir_hyb_spmm_raw(static_cast<const float*>(b), static_cast<float*>(c), bk.data(), K,
                                (int)(lc / feat), (int)(lb / feat), (int)feat, (int)flags,
                                p.device_id, sptir::stream_for(p.device_id));
}

int sparsetir_hyb_spmm(SPARSETIR_PACKED_ARGS) {
  return hyb_packed("sparsetir_hyb_spmm", false, args, type_codes, num_args, out_ret_value, out_ret_tcode,
                    resource_handle);
}

int sparsetir_hyb_spmm_peers(SPARSETIR_PACKED_ARGS) {
  return hyb_packed("sparsetir_hyb_spmm_peers", true, args, type_codes, num_args, out_ret_value,
                    out_ret_tcode, resource_handle);
}

int sparsetir_sddmm(SPARSETIR_PACKED_ARGS) {
  (void)resource_handle;
  Packed p{"sparsetir_sddmm", args, type_codes, num_args};
  if (num_args != 5 && num_args != 6 && num_args != 9 && num_args != 10)
    return fail("sparsetir_sddmm: num_args should be 5, 6, 9 or 10, got %d", num_args);
  void *a = nullptr, *b = nullptr, *c = nullptr, *indptr = nullptr, *indices = nullptr;
  void* scale = nullptr;
  int64_t la = 0, lb = 0, lc = 0, lp = 0, li = 0, ls = 0;
  TRY(p.tensor(0, "a", kDLFloat, 32, &a, &la));
  TRY(p.tensor(1, "b", kDLFloat, 32, &b, &lb));
  TRY(p.tensor(2, "c", kDLFloat, 32, &c, &lc));
  TRY(p.tensor(3, "indptr", kDLInt, 32, &indptr, &lp));
  TRY(p.tensor(4, "indices", kDLInt, 32, &indices, &li));
  bool scalars = num_args >= 9;
  bool has_scale = (num_args == 6 || num_args == 10);
  int64_t m = 0, n = 0, feat = 0, nnz = 0;
  if (scalars) {
    TRY(p.integer(5, "m", &m));
    TRY(p.integer(6, "n", &n));
    TRY(p.integer(7, "feat_size", &feat));
    TRY(p.integer(8, "nnz", &nnz));
  } else {
    m = lp - 1;
    nnz = lc;
    if (m < 1) return fail("sparsetir_sddmm: cannot infer feat_size with m = %lld", (long long)m);
    if (la % m != 0) return fail("sparsetir_sddmm: len(a) is not a multiple of m");
    feat = la / m;
    if (feat == 0 || lb % feat != 0)
      return fail("sparsetir_sddmm: len(b) is not a multiple of feat_size");
    n = lb / feat;
  }
  if (has_scale) TRY(p.tensor(num_args - 1, "scale", kDLFloat, 32, &scale, &ls));
  TRY(fits_i32(p.fn, "m", m)); TRY(fits_i32(p.fn, "n", n));
  TRY(fits_i32(p.fn, "feat_size", feat)); TRY(fits_i32(p.fn, "nnz", nnz));
  TRY(check_len(p.fn, "a", la, m * feat));
  TRY(check_len(p.fn, "b", lb, n * feat));
  TRY(check_len(p.fn, "c", lc, nnz));
  TRY(check_len(p.fn, "indptr", lp, m + 1));
  TRY(check_len(p.fn, "indices", li, nnz));
  if (has_scale) TRY(check_len(p.fn, "scale", ls, nnz));
  set_void_return(out_ret_value, out_ret_tcode);
  return sparsetir_sddmm_raw(static_cast<const float*>(a), static_cast<const float*>(b),
                             static_cast<float*>(c), static_cast<const int32_t*>(indptr),
                             static_cast<const int32_t*>(indices),
                             static_cast<const float*>(scale), (int)m, (int)n, (int)feat, (int)nnz,
                             p.device_id, sptir::stream_for(p.device_id));
}

int sparsetir_sddmm_peers(SPARSETIR_PACKED_ARGS) {
  (void)resource_handle;
  Packed p{"sparsetir_sddmm_peers", args, type_codes, num_args};
  const bool has_scale = num_args > 6 && p.is_tensor(num_args - 1);
  const int np = num_args - 5 - (has_scale ? 1 : 0);
  if (np < 1 || np > SPARSETIR_MAX_PEERS)
    return fail("sparsetir_sddmm_peers: expected (a, b, c, indptr, indices, 1 to %d peer addresses[, scale]), "
                "got %d arguments", SPARSETIR_MAX_PEERS, num_args);
  void *a = nullptr, *b = nullptr, *c = nullptr, *indptr = nullptr, *indices = nullptr;
  void* scale = nullptr;
  int64_t la = 0, lb = 0, lc = 0, lp = 0, li = 0, ls = 0;
  TRY(p.tensor(0, "a", kDLFloat, 32, &a, &la));
  TRY(p.tensor(1, "b", kDLFloat, 32, &b, &lb));
  TRY(p.tensor(2, "c", kDLFloat, 32, &c, &lc));
  TRY(p.tensor(3, "indptr", kDLInt, 32, &indptr, &lp));
  TRY(p.tensor(4, "indices", kDLInt, 32, &indices, &li));
  std::vector<void*> peer_c;
  for (int k = 0; k < np; ++k) {
    int64_t addr = 0;
    TRY(p.integer(5 + k, "peer_c", &addr));
    peer_c.push_back(reinterpret_cast<void*>(static_cast<intptr_t>(addr)));
  }
  if (has_scale) TRY(p.tensor(num_args - 1, "scale", kDLFloat, 32, &scale, &ls));
  const int64_t m = lp - 1, nnz = lc;
  if (m < 1) return fail("sparsetir_sddmm_peers: cannot infer feat_size with m = %lld", (long long)m);
  if (la % m != 0) return fail("sparsetir_sddmm_peers: len(a) is not a multiple of m");
  const int64_t feat = la / m;
  if (feat == 0 || lb % feat != 0)
    return fail("sparsetir_sddmm_peers: len(b) is not a multiple of feat_size");
  const int64_t n = lb / feat;
  TRY(fits_i32(p.fn, "m", m)); TRY(fits_i32(p.fn, "n", n));
  TRY(fits_i32(p.fn, "feat_size", feat)); TRY(fits_i32(p.fn, "nnz", nnz));
  TRY(check_len(p.fn, "indices", li, nnz));
  if (has_scale) TRY(check_len(p.fn, "scale", ls, nnz));
  set_void_return(out_ret_value, out_ret_tcode);
  return sparsetir_sddmm_peers_raw(static_cast<const float*>(a), static_cast<const float*>(b),
                                   static_cast<float*>(c), static_cast<const int32_t*>(indptr),
                                   static_cast<const int32_t*>(indices), static_cast<const float*>(scale),
                                   (int)m, (int)n, (int)feat, (int)nnz, (int)peer_c.size(), peer_c.data(),
                                   p.device_id, sptir::stream_for(p.device_id));
}

int sparsetir_sddmm_edge_to_row(SPARSETIR_PACKED_ARGS) {
  (void)resource_handle;
  Packed p{"sparsetir_sddmm_edge_to_row", args, type_codes, num_args};
  if (num_args != 2)
    return fail("sparsetir_sddmm_edge_to_row: num_args should be 2, got %d", num_args);
  void *indptr = nullptr, *mid = nullptr;
  int64_t lp = 0, lm = 0;
  TRY(p.tensor(0, "indptr", kDLInt, 32, &indptr, &lp));
  TRY(p.tensor(1, "mid", kDLInt, 32, &mid, &lm));
  if (lp < 1) return fail("sparsetir_sddmm_edge_to_row: indptr must have at least one element");
  TRY(fits_i32(p.fn, "m", lp - 1)); TRY(fits_i32(p.fn, "nnz", lm));
  set_void_return(out_ret_value, out_ret_tcode);
  return sparsetir_sddmm_edge_to_row_raw(static_cast<const int32_t*>(indptr),
                                         static_cast<int32_t*>(mid), (int)(lp - 1), (int)lm,
                                         p.device_id, sptir::stream_for(p.device_id));
}

int sparsetir_bsrmm(SPARSETIR_PACKED_ARGS) {
  (void)resource_handle;
  Packed p{"sparsetir_bsrmm", args, type_codes, num_args};
  if (num_args != 10) return fail("sparsetir_bsrmm: num_args should be 10, got %d", num_args);
  void *a = nullptr, *b = nullptr, *c = nullptr, *indptr = nullptr, *indices = nullptr;
  int64_t la = 0, lb = 0, lc = 0, lp = 0, li = 0, nb = 0, mb = 0, nnzb = 0, blk = 0, feat = 0;
  TRY(p.tensor(0, "a", kDLFloat, 16, &a, &la));
  TRY(p.tensor(1, "b", kDLFloat, 16, &b, &lb));
  TRY(p.tensor(2, "c", kDLFloat, 32, &c, &lc));
  TRY(p.tensor(3, "indptr", kDLInt, 32, &indptr, &lp));
  TRY(p.tensor(4, "indices", kDLInt, 32, &indices, &li));
  TRY(p.integer(5, "nb", &nb));
  TRY(p.integer(6, "mb", &mb));
  TRY(p.integer(7, "nnzb", &nnzb));
  TRY(p.integer(8, "blk", &blk));
  TRY(p.integer(9, "feat_size", &feat));
  TRY(fits_i32(p.fn, "nb", nb)); TRY(fits_i32(p.fn, "mb", mb)); TRY(fits_i32(p.fn, "nnzb", nnzb));
  TRY(fits_i32(p.fn, "blk", blk)); TRY(fits_i32(p.fn, "feat_size", feat));
  TRY(check_len(p.fn, "a", la, nnzb * blk * blk));
  TRY(check_len(p.fn, "b", lb, mb * blk * feat));
  TRY(check_len(p.fn, "c", lc, nb * blk * feat));
  TRY(check_len(p.fn, "indptr", lp, nb + 1));
  TRY(check_len(p.fn, "indices", li, nnzb));
  set_void_return(out_ret_value, out_ret_tcode);
  return sparsetir_bsrmm_raw(a, b, static_cast<float*>(c), static_cast<const int32_t*>(indptr),
                             static_cast<const int32_t*>(indices), (int)nb, (int)mb, (int)nnzb,
                             (int)blk, (int)feat, p.device_id, sptir::stream_for(p.device_id));
}

int sparsetir_rgms(SPARSETIR_PACKED_ARGS) {
  (void)resource_handle;
  Packed p{"sparsetir_rgms", args, type_codes, num_args};
  if (num_args != 8 && num_args != 14)
    return fail("sparsetir_rgms: num_args should be 8 or 14, got %d", num_args);
  void *a = nullptr, *w = nullptr, *x = nullptr, *y = nullptr, *ip_i = nullptr, *ix_i = nullptr, *ip_j = nullptr, *ix_j = nullptr;
  int64_t la = 0, lw = 0, lx = 0, ly = 0, lpi = 0, lii = 0, lpj = 0, lij = 0;
  TRY(p.tensor(0, "a", kDLFloat, 32, &a, &la));
  TRY(p.tensor(1, "w", kDLFloat, 32, &w, &lw));
  TRY(p.tensor(2, "x", kDLFloat, 32, &x, &lx));
  TRY(p.tensor(3, "y", kDLFloat, 32, &y, &ly));
  TRY(p.tensor(4, "indptr_i", kDLInt, 32, &ip_i, &lpi));
  TRY(p.tensor(5, "indices_i", kDLInt, 32, &ix_i, &lii));
  TRY(p.tensor(6, "indptr_j", kDLInt, 32, &ip_j, &lpj));
  TRY(p.tensor(7, "indices_j", kDLInt, 32, &ix_j, &lij));
  int64_t m = 0, n = 0, R = 0, feat = 0, nnz_i = 0, nnz_j = 0;
  if (num_args == 14) {
    TRY(p.integer(8, "m", &m));
    TRY(p.integer(9, "n", &n));
    TRY(p.integer(10, "num_rels", &R));
    TRY(p.integer(11, "feat_size", &feat));
    TRY(p.integer(12, "nnz_i", &nnz_i));
    TRY(p.integer(13, "nnz_j", &nnz_j));
  } else {
    R = lpi - 1;
    nnz_i = lii;
    nnz_j = lij;
    if (R < 1) return fail("sparsetir_rgms: cannot infer feat_size with num_rels = %lld", (long long)R);
    feat = (int64_t)std::llround(std::sqrt((double)(lw / R)));
    if (feat <= 0 || feat * feat * R != lw)
      return fail("sparsetir_rgms: len(w) = %lld is not num_rels * feat_size^2", (long long)lw);
    if (lx % feat != 0 || ly % feat != 0)
      return fail("sparsetir_rgms: len(x) and len(y) must be multiples of feat_size");
    m = ly / feat;
    n = lx / feat;
  }
  TRY(fits_i32(p.fn, "m", m)); TRY(fits_i32(p.fn, "n", n)); TRY(fits_i32(p.fn, "num_rels", R));
  TRY(fits_i32(p.fn, "feat_size", feat)); TRY(fits_i32(p.fn, "nnz_i", nnz_i));
  TRY(fits_i32(p.fn, "nnz_j", nnz_j));
  TRY(check_len(p.fn, "a", la, nnz_j));
  TRY(check_len(p.fn, "w", lw, R * feat * feat));
  TRY(check_len(p.fn, "x", lx, n * feat));
  TRY(check_len(p.fn, "y", ly, m * feat));
  TRY(check_len(p.fn, "indptr_i", lpi, R + 1));
  TRY(check_len(p.fn, "indices_i", lii, nnz_i));
  TRY(check_len(p.fn, "indptr_j", lpj, nnz_i + 1));
  TRY(check_len(p.fn, "indices_j", lij, nnz_j));
  set_void_return(out_ret_value, out_ret_tcode);
  return sparsetir_rgms_raw(static_cast<const float*>(a), static_cast<const float*>(w),
                            static_cast<const float*>(x), static_cast<float*>(y),
                            static_cast<const int32_t*>(ip_i), static_cast<const int32_t*>(ix_i),
                            static_cast<const int32_t*>(ip_j), static_cast<const int32_t*>(ix_j),
                            (int)m, (int)n, (int)R, (int)feat, (int)nnz_i, (int)nnz_j, p.device_id,
                            sptir::stream_for(p.device_id));
}

int sparsetir_rgms_ell3d(SPARSETIR_PACKED_ARGS) {
  (void)resource_handle;
  Packed p{"sparsetir_rgms_ell3d", args, type_codes, num_args};
  int nt = 0;
  while (p.is_tensor(nt)) ++nt;
  if (num_args - nt != 1 || nt < 3 || (nt - 3) % 4 != 0)
    return fail("sparsetir_rgms_ell3d: expected (w, x, y, {a, rows, cols} x K, {mid} x K, feat_size); "
                "got %d tensor and %d scalar arguments", nt, num_args - nt);
  const int K = (nt - 3) / 4;
  void *w = nullptr, *x = nullptr, *y = nullptr;
  int64_t lw = 0, lx = 0, ly = 0, feat = 0;
  TRY(p.tensor(0, "w", kDLFloat, 32, &w, &lw));
  TRY(p.tensor(1, "x", kDLFloat, 32, &x, &lx));
  TRY(p.tensor(2, "y", kDLFloat, 32, &y, &ly));
  TRY(p.integer(nt, "feat_size", &feat));
  if (feat <= 0) return fail("sparsetir_rgms_ell3d: feat_size must be positive");
  if (lw % (feat * feat) != 0 || lx % feat != 0 || ly % feat != 0)
    return fail("sparsetir_rgms_ell3d: len(w), len(x), len(y) must be multiples of feat_size^2, "
                "feat_size, feat_size");
  TRY(fits_i32(p.fn, "feat_size", feat));
  TRY(fits_i32(p.fn, "m", ly / feat)); TRY(fits_i32(p.fn, "n", lx / feat));
  TRY(fits_i32(p.fn, "num_rels", lw / (feat * feat)));
  std::vector<SparsetirEll3dBucket> bk(K);
  for (int q = 0; q < K; ++q) {
    void *a = nullptr, *rows = nullptr, *cols = nullptr, *mid = nullptr;
    int64_t la = 0, lr = 0, lc = 0, lm = 0;
    TRY(p.tensor(3 + 3 * q, "a", kDLFloat, 32, &a, &la));
    TRY(p.tensor(4 + 3 * q, "rows", kDLInt, 32, &rows, &lr));
    TRY(p.tensor(5 + 3 * q, "cols", kDLInt, 32, &cols, &lc));
    TRY(p.tensor(3 + 3 * K + q, "mid", kDLInt, 32, &mid, &lm));
    TRY(check_len(p.fn, "a", la, lc));
    int64_t rpg = 0, cpr = 0;
    if (lm > 0) {
      if (lr == 0 || lr % lm != 0 || lc == 0 || lc % lr != 0)
        return fail("sparsetir_rgms_ell3d: bucket %d: len(mid) = %lld, len(rows) = %lld, len(cols) = %lld "
                    "do not describe groups x rows x columns", q, (long long)lm, (long long)lr, (long long)lc);
      rpg = lr / lm;
      cpr = lc / lr;
    } else if (lr != 0 || lc != 0) {
      return fail("sparsetir_rgms_ell3d: bucket %d has rows or columns but no groups", q);
    }
    TRY(fits_i32(p.fn, "groups", lm)); TRY(fits_i32(p.fn, "rows", lr)); TRY(fits_i32(p.fn, "slots", lc));
    bk[q] = SparsetirEll3dBucket{static_cast<const float*>(a), static_cast<const int32_t*>(rows),
                                 static_cast<const int32_t*>(cols), static_cast<const int32_t*>(mid),
                                 (int32_t)lm, (int32_t)rpg, (int32_t)cpr};
  }
  set_void_return(out_ret_value, out_ret_tcode);
  return sparsetir_rgms_ell3d_raw(static_cast<const float*>(w), static_cast<const float*>(x),
                                  static_cast<float*>(y), bk.data(), K, (int)(ly / feat), (int)(lx / feat),
                                  (int)(lw / (feat * feat)), (int)feat, p.device_id,
                                  sptir::stream_for(p.device_id));
}

int sparsetir_rgms_ell3d_f16(SPARSETIR_PACKED_ARGS) {
  (void)resource_handle;
  Packed p{"sparsetir_rgms_ell3d_f16", args, type_codes, num_args};
  int nt = 0;
  while (p.is_tensor(nt)) ++nt;
  if (num_args - nt != 2 || nt < 3 || (nt - 3) % 4 != 0)
    return fail("sparsetir_rgms_ell3d_f16: expected (w, x, y, {a, rows, cols} x K, {mid} x K, feat_in, "
                "feat_out); got %d tensor and %d scalar arguments", nt, num_args - nt);
  const int K = (nt - 3) / 4;
  void *w = nullptr, *x = nullptr, *y = nullptr;
  int64_t lw = 0, lx = 0, ly = 0, fin = 0, fout = 0;
  TRY(p.tensor(0, "w", kDLFloat, 16, &w, &lw));
  TRY(p.tensor(1, "x", kDLFloat, 16, &x, &lx));
  // the reference builds the function for a float16 or a float32 result
  int y_is_f16 = 1;
  if (args[2].v_handle != nullptr && static_cast<const DLTensor*>(args[2].v_handle)->dtype.bits == 32)
    y_is_f16 = 0;
  TRY(p.tensor(2, "y", kDLFloat, y_is_f16 ? 16 : 32, &y, &ly));
  TRY(p.integer(nt, "feat_in", &fin));
  TRY(p.integer(nt + 1, "feat_out", &fout));
  if (fin <= 0 || fout <= 0) return fail("sparsetir_rgms_ell3d_f16: feat_in and feat_out must be positive");
  if (lw % (fin * fout) != 0 || lx % fin != 0 || ly % fout != 0)
    return fail("sparsetir_rgms_ell3d_f16: len(w), len(x), len(y) must be multiples of feat_in*feat_out, "
                "feat_in, feat_out");
  TRY(fits_i32(p.fn, "feat_in", fin)); TRY(fits_i32(p.fn, "feat_out", fout));
  TRY(fits_i32(p.fn, "m", ly / fout)); TRY(fits_i32(p.fn, "n", lx / fin));
  TRY(fits_i32(p.fn, "num_rels", lw / (fin * fout)));
  std::vector<SparsetirEll3dBucketH> bk(K);
  for (int q = 0; q < K; ++q) {
    void *a = nullptr, *rows = nullptr, *cols = nullptr, *mid = nullptr;
    int64_t la = 0, lr = 0, lc = 0, lm = 0;
    TRY(p.tensor(3 + 3 * q, "a", kDLFloat, 16, &a, &la));
    TRY(p.tensor(4 + 3 * q, "rows", kDLInt, 32, &rows, &lr));
    TRY(p.tensor(5 + 3 * q, "cols", kDLInt, 32, &cols, &lc));
    TRY(p.tensor(3 + 3 * K + q, "mid", kDLInt, 32, &mid, &lm));
    TRY(check_len(p.fn, "a", la, lc));
    int64_t rpg = 0, cpr = 0;
    if (lm > 0) {
      if (lr == 0 || lr % lm != 0 || lc == 0 || lc % lr != 0)
        return fail("sparsetir_rgms_ell3d_f16: bucket %d: len(mid) = %lld, len(rows) = %lld, len(cols) = %lld "
                    "do not describe groups x rows x columns", q, (long long)lm, (long long)lr, (long long)lc);
      rpg = lr / lm;
      cpr = lc / lr;
    } else if (lr != 0 || lc != 0) {
      return fail("sparsetir_rgms_ell3d_f16: bucket %d has rows or columns but no groups", q);
    }
    TRY(fits_i32(p.fn, "groups", lm)); TRY(fits_i32(p.fn, "rows", lr)); TRY(fits_i32(p.fn, "slots", lc));
    bk[q] = SparsetirEll3dBucketH{a, static_cast<const int32_t*>(rows), static_cast<const int32_t*>(cols),
                                  static_cast<const int32_t*>(mid), (int32_t)lm, (int32_t)rpg, (int32_t)cpr};
  }
  set_void_return(out_ret_value, out_ret_tcode);
  return sparsetir_rgms_ell3d_f16_raw(w, x, y, y_is_f16, bk.data(), K, (int)(ly / fout), (int)(lx / fin),
                                      (int)(lw / (fin * fout)), (int)fin, (int)fout, p.device_id,
                                      sptir::stream_for(p.device_id));
}

int sparsetir_sparse_conv_f16(SPARSETIR_PACKED_ARGS) {
  (void)resource_handle;
  Packed p{"sparsetir_sparse_conv_f16", args, type_codes, num_args};
  if (num_args != 9) return fail("sparsetir_sparse_conv_f16: num_args should be 9, got %d", num_args);
  void *w = nullptr, *x = nullptr, *y = nullptr, *map = nullptr;
  int64_t lw = 0, lx = 0, ly = 0, lmap = 0, m = 0, rels = 0, fin = 0, fout = 0, add = 0;
  TRY(p.tensor(0, "w", kDLFloat, 16, &w, &lw));
  TRY(p.tensor(1, "x", kDLFloat, 16, &x, &lx));
  int y_is_f16 = 1;
  if (p.is_tensor(2) && args[2].v_handle != nullptr && static_cast<const DLTensor*>(args[2].v_handle)->dtype.bits == 32)
    y_is_f16 = 0;
  TRY(p.tensor(2, "y", kDLFloat, y_is_f16 ? 16 : 32, &y, &ly));
  TRY(p.tensor(3, "map", kDLInt, 32, &map, &lmap));
  TRY(p.integer(4, "m", &m));
  TRY(p.integer(5, "num_rels", &rels));
  TRY(p.integer(6, "feat_in", &fin));
  TRY(p.integer(7, "feat_out", &fout));
  TRY(p.integer(8, "add", &add));
  TRY(fits_i32(p.fn, "m", m)); TRY(fits_i32(p.fn, "num_rels", rels));
  TRY(fits_i32(p.fn, "feat_in", fin)); TRY(fits_i32(p.fn, "feat_out", fout));
  if (fin == 0 || fout == 0) return fail("sparsetir_sparse_conv_f16: feat_in and feat_out must be positive");
  if (lx % fin != 0) return fail("sparsetir_sparse_conv_f16: len(x) is not a multiple of feat_in");
  TRY(fits_i32(p.fn, "n", lx / fin));
  TRY(check_len(p.fn, "w", lw, rels * fin * fout));
  TRY(check_len(p.fn, "y", ly, m * fout));
  TRY(check_len(p.fn, "map", lmap, (m + 127) / 128 * rels * 128));
  set_void_return(out_ret_value, out_ret_tcode);
  return sparsetir_sparse_conv_f16_raw(w, x, y, y_is_f16, static_cast<const int32_t*>(map), (int)m, (int)(lx / fin),
                                       (int)rels, (int)fin, (int)fout, add != 0, p.device_id,
                                       sptir::stream_for(p.device_id));
}

int sparsetir_tcspmm(SPARSETIR_PACKED_ARGS) {
  (void)resource_handle;
  Packed p{"sparsetir_tcspmm", args, type_codes, num_args};
  if (num_args != 11) return fail("sparsetir_tcspmm: num_args should be 11, got %d", num_args);
  void *a = nullptr, *b = nullptr, *c = nullptr, *indptr = nullptr, *indices = nullptr;
  int64_t la = 0, lb = 0, lc = 0, lp = 0, li = 0, mb = 0, nb = 0, nnzb = 0, feat = 0, t = 0, g = 0;
  TRY(p.tensor(0, "a", kDLFloat, 16, &a, &la));
  TRY(p.tensor(1, "b", kDLFloat, 16, &b, &lb));
  // the reference's output buffer is float16; float32 (the accumulator's precision) is taken too
  int c_is_f16 = 1;
  if (num_args > 2 && p.is_tensor(2) && args[2].v_handle != nullptr &&
      static_cast<const DLTensor*>(args[2].v_handle)->dtype.bits == 32)
    c_is_f16 = 0;
  TRY(p.tensor(2, "c", kDLFloat, c_is_f16 ? 16 : 32, &c, &lc));
  TRY(p.tensor(3, "indptr", kDLInt, 32, &indptr, &lp));
  TRY(p.tensor(4, "indices", kDLInt, 32, &indices, &li));
  TRY(p.integer(5, "mb", &mb)); TRY(p.integer(6, "nb", &nb)); TRY(p.integer(7, "nnzb", &nnzb));
  TRY(p.integer(8, "feat_size", &feat)); TRY(p.integer(9, "tile_size", &t));
  TRY(p.integer(10, "group_size", &g));
  TRY(fits_i32(p.fn, "mb", mb)); TRY(fits_i32(p.fn, "nb", nb)); TRY(fits_i32(p.fn, "nnzb", nnzb));
  TRY(fits_i32(p.fn, "feat_size", feat)); TRY(fits_i32(p.fn, "tile_size", t));
  TRY(fits_i32(p.fn, "group_size", g));
  if (t < 1 || g < 1) return fail("sparsetir_tcspmm: tile_size and group_size must be positive");
  TRY(fits_i32(p.fn, "nnzb * group_size", nnzb * g));
  TRY(check_len(p.fn, "a", la, nnzb * t * g));
  TRY(check_len(p.fn, "b", lb, nb * g * feat));
  TRY(check_len(p.fn, "c", lc, mb * t * feat));
  TRY(check_len(p.fn, "indptr", lp, mb + 1));
  TRY(check_len(p.fn, "indices", li, nnzb * g));
  set_void_return(out_ret_value, out_ret_tcode);
  return sparsetir_tcspmm_raw(a, b, c, c_is_f16, static_cast<const int32_t*>(indptr),
                              static_cast<const int32_t*>(indices), (int)mb, (int)nb, (int)nnzb, (int)feat,
                              (int)t, (int)g, p.device_id, sptir::stream_for(p.device_id));
}

int sparsetir_csr_reduce(SPARSETIR_PACKED_ARGS) {
  (void)resource_handle;
  Packed p{"sparsetir_csr_reduce", args, type_codes, num_args};
  int nt = 0;
  while (p.is_tensor(nt)) ++nt;
  if (nt != 3 && nt != 4)
    return fail("sparsetir_csr_reduce: expected (a, b, indptr[, indices][, sizes...]); got %d tensor "
                "arguments", nt);
  void *a = nullptr, *b = nullptr, *indptr = nullptr, *indices = nullptr;
  int64_t la = 0, lb = 0, lp = 0, li = 0;
  TRY(p.tensor(0, "a", kDLFloat, 32, &a, &la));
  TRY(p.tensor(1, "b", kDLFloat, 32, &b, &lb));
  TRY(p.tensor(2, "indptr", kDLInt, 32, &indptr, &lp));
  if (nt == 4) {
    TRY(p.tensor(3, "indices", kDLInt, 32, &indices, &li));
    TRY(check_len(p.fn, "indices", li, la));
  }
  for (int i = nt; i < num_args; ++i) {  // trailing n[, m], nnz of the unspecialised signature
    int64_t v = 0;
    TRY(p.integer(i, "size", &v));
  }
  TRY(check_len(p.fn, "indptr", lp, lb + 1));
  TRY(fits_i32(p.fn, "n", lb)); TRY(fits_i32(p.fn, "nnz", la));
  set_void_return(out_ret_value, out_ret_tcode);
  return sparsetir_csr_reduce_raw(static_cast<const float*>(a), static_cast<float*>(b),
                                  static_cast<const int32_t*>(indptr), (int)lb, (int)la, p.device_id,
                                  sptir::stream_for(p.device_id));
}

int sparsetir_sparse_softmax(SPARSETIR_PACKED_ARGS) {
  (void)resource_handle;
  Packed p{"sparsetir_sparse_softmax", args, type_codes, num_args};
  if (num_args != 4 && num_args != 6)
    return fail("sparsetir_sparse_softmax: num_args should be 4 or 6, got %d", num_args);
  void *a = nullptr, *b = nullptr, *indptr = nullptr, *indices = nullptr;
  int64_t la = 0, lb = 0, lp = 0, li = 0;
  TRY(p.tensor(0, "a", kDLFloat, 32, &a, &la));
  TRY(p.tensor(1, "b", kDLFloat, 32, &b, &lb));
  TRY(p.tensor(2, "indptr", kDLInt, 32, &indptr, &lp));
  TRY(p.tensor(3, "indices", kDLInt, 32, &indices, &li));
  if (num_args == 6) {
    int64_t n = 0, nnz = 0;
    TRY(p.integer(4, "n", &n)); TRY(p.integer(5, "nnz", &nnz));
    TRY(check_len(p.fn, "indptr", lp, n + 1));
    TRY(check_len(p.fn, "a", la, nnz));
  }
  if (lp < 1) return fail("sparsetir_sparse_softmax: indptr must have at least one element");
  TRY(check_len(p.fn, "b", lb, la));
  TRY(check_len(p.fn, "indices", li, la));
  TRY(fits_i32(p.fn, "n", lp - 1)); TRY(fits_i32(p.fn, "nnz", la));
  set_void_return(out_ret_value, out_ret_tcode);
  return sparsetir_sparse_softmax_raw(static_cast<const float*>(a), static_cast<float*>(b),
                                      static_cast<const int32_t*>(indptr), (int)(lp - 1), (int)la,
                                      p.device_id, sptir::stream_for(p.device_id));
}

int sparsetir_csr2bsr(SPARSETIR_PACKED_ARGS) {
  (void)resource_handle;
  Packed p{"sparsetir_csr2bsr", args, type_codes, num_args};
  if (num_args != 7 && num_args != 13)
    return fail("sparsetir_csr2bsr: num_args should be 7 or 13, got %d", num_args);
  void *a = nullptr, *b = nullptr, *ip = nullptr, *ix = nullptr, *op = nullptr, *ox = nullptr;
  int64_t la = 0, lb = 0, lip = 0, lix = 0, lop = 0, lox = 0, blk = 0;
  TRY(p.tensor(0, "a", kDLFloat, 32, &a, &la));
  TRY(p.tensor(1, "b", kDLFloat, 32, &b, &lb));
  TRY(p.tensor(2, "indptr_in", kDLInt, 32, &ip, &lip));
  TRY(p.tensor(3, "indices_in", kDLInt, 32, &ix, &lix));
  TRY(p.tensor(4, "indptr_out", kDLInt, 32, &op, &lop));
  TRY(p.tensor(5, "indices_out", kDLInt, 32, &ox, &lox));
  TRY(p.integer(num_args - 1, "blk_size", &blk));
  if (blk < 1) return fail("sparsetir_csr2bsr: blk_size must be positive");
  if (lip < 1 || lop < 1) return fail("sparsetir_csr2bsr: empty row pointer array");
  if (num_args == 13) {
    int64_t m_in = 0, m_out = 0, nnz_in = 0, nnz_out = 0;
    TRY(p.integer(6, "m_in", &m_in)); TRY(p.integer(8, "m_out", &m_out));
    TRY(p.integer(10, "nnz_in", &nnz_in)); TRY(p.integer(11, "nnz_out", &nnz_out));
    TRY(check_len(p.fn, "indptr_in", lip, m_in + 1));
    TRY(check_len(p.fn, "indptr_out", lop, m_out + 1));
    TRY(check_len(p.fn, "a", la, nnz_in));
    TRY(check_len(p.fn, "indices_out", lox, nnz_out));
  }
  TRY(check_len(p.fn, "indices_in", lix, la));
  TRY(check_len(p.fn, "b", lb, lox * blk * blk));
  if ((lip - 1 + blk - 1) / blk > lop - 1)
    return fail("sparsetir_csr2bsr: the block matrix has fewer block rows than the rows need");
  TRY(fits_i32(p.fn, "m_in", lip - 1)); TRY(fits_i32(p.fn, "nnz_in", la));
  TRY(fits_i32(p.fn, "blk_size", blk));
  set_void_return(out_ret_value, out_ret_tcode);
  return sparsetir_csr2bsr_raw(static_cast<const float*>(a), static_cast<float*>(b),
                               static_cast<const int32_t*>(ip), static_cast<const int32_t*>(ix),
                               static_cast<const int32_t*>(op), static_cast<const int32_t*>(ox),
                               (int)(lip - 1), (int)la, (int)blk, p.device_id,
                               sptir::stream_for(p.device_id));
}

int sparsetir_ellmm(SPARSETIR_PACKED_ARGS) {
  (void)resource_handle;
  Packed p{"sparsetir_ellmm", args, type_codes, num_args};
  if (num_args != 9) return fail("sparsetir_ellmm: num_args should be 9, got %d", num_args);
  void *a = nullptr, *b = nullptr, *c = nullptr, *indices = nullptr;
  int64_t la = 0, lb = 0, lc = 0, li = 0, nb = 0, mb = 0, feat = 0, col = 0, blk = 0;
  TRY(p.tensor(0, "a", kDLFloat, 32, &a, &la));
  TRY(p.tensor(1, "b", kDLFloat, 32, &b, &lb));
  TRY(p.tensor(2, "c", kDLFloat, 32, &c, &lc));
  TRY(p.tensor(3, "indices", kDLInt, 32, &indices, &li));
  TRY(p.integer(4, "nb", &nb)); TRY(p.integer(5, "mb", &mb)); TRY(p.integer(6, "feat_size", &feat));
  TRY(p.integer(7, "col", &col)); TRY(p.integer(8, "blk", &blk));
  TRY(fits_i32(p.fn, "nb", nb)); TRY(fits_i32(p.fn, "mb", mb)); TRY(fits_i32(p.fn, "feat_size", feat));
  TRY(fits_i32(p.fn, "col", col)); TRY(fits_i32(p.fn, "blk", blk));
  if (blk < 1) return fail("sparsetir_ellmm: blk must be positive");
  TRY(check_len(p.fn, "a", la, nb * col * blk * blk));
  TRY(check_len(p.fn, "b", lb, mb * blk * feat));
  TRY(check_len(p.fn, "c", lc, nb * blk * feat));
  TRY(check_len(p.fn, "indices", li, nb * col));
  set_void_return(out_ret_value, out_ret_tcode);
  return sparsetir_ellmm_raw(static_cast<const float*>(a), static_cast<const float*>(b),
                             static_cast<float*>(c), static_cast<const int32_t*>(indices), (int)nb, (int)mb,
                             (int)feat, (int)col, (int)blk, p.device_id, sptir::stream_for(p.device_id));
}

int sparsetir_fusedmm(SPARSETIR_PACKED_ARGS) {
  (void)resource_handle;
  Packed p{"sparsetir_fusedmm", args, type_codes, num_args};
  if (num_args != 6 && num_args != 10)
    return fail("sparsetir_fusedmm: num_args should be 6 or 10, got %d", num_args);
  void *q = nullptr, *k = nullptr, *v = nullptr, *o = nullptr, *indptr = nullptr, *indices = nullptr;
  int64_t lq = 0, lk = 0, lv = 0, lo = 0, lp = 0, li = 0, m = 0, n = 0, nnz = 0, feat = 0;
  TRY(p.tensor(0, "q", kDLFloat, 32, &q, &lq));
  TRY(p.tensor(1, "k", kDLFloat, 32, &k, &lk));
  TRY(p.tensor(2, "v", kDLFloat, 32, &v, &lv));
  TRY(p.tensor(3, "o", kDLFloat, 32, &o, &lo));
  TRY(p.tensor(4, "indptr", kDLInt, 32, &indptr, &lp));
  TRY(p.tensor(5, "indices", kDLInt, 32, &indices, &li));
  if (num_args == 10) {
    TRY(p.integer(6, "m", &m)); TRY(p.integer(7, "n", &n)); TRY(p.integer(8, "nnz", &nnz));
    TRY(p.integer(9, "feat_size", &feat));
  } else {
    m = lp - 1;
    nnz = li;
    if (m < 1 || lq % m != 0) return fail("sparsetir_fusedmm: cannot infer feat_size from len(q) and m");
    feat = lq / m;
    if (feat == 0 || lk % feat != 0) return fail("sparsetir_fusedmm: len(k) is not a multiple of feat_size");
    n = lk / feat;
  }
  TRY(fits_i32(p.fn, "m", m)); TRY(fits_i32(p.fn, "n", n)); TRY(fits_i32(p.fn, "nnz", nnz));
  TRY(fits_i32(p.fn, "feat_size", feat));
  TRY(check_len(p.fn, "q", lq, m * feat));
  TRY(check_len(p.fn, "k", lk, n * feat));
  TRY(check_len(p.fn, "v", lv, n * feat));
  TRY(check_len(p.fn, "o", lo, m * feat));
  TRY(check_len(p.fn, "indptr", lp, m + 1));
  TRY(check_len(p.fn, "indices", li, nnz));
  set_void_return(out_ret_value, out_ret_tcode);
  return sparsetir_fusedmm_raw(static_cast<const float*>(q), static_cast<const float*>(k),
                               static_cast<const float*>(v), static_cast<float*>(o),
                               static_cast<const int32_t*>(indptr), static_cast<const int32_t*>(indices),
                               (int)m, (int)n, (int)nnz, (int)feat, p.device_id,
                               sptir::stream_for(p.device_id));
}

}  // extern "C"
