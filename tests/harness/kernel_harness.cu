// Test harness: single launches of the library's kernels, linked against libpibem_gb300.so, for
// what the C ABI shows only through whole operators.  Host arrays in and out; every function
// returns the device error flag (0: none) or -1 after an exception.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <exception>
#include <vector>

#include "../../pi-bem_gb300/csrc/kernels.h"
#include "../../pi-bem_gb300/csrc/krylov.h"

using namespace pibem;

namespace
{
  template <typename F>
  int guarded(F f)
  {
    try
      {
        return f();
      }
    catch (const std::exception &e)
      {
        std::fprintf(stderr, "kernel_harness: %s\n", e.what());
        return -1;
      }
  }

  // a device copy of n host values
  template <typename T>
  struct Up : DBuf<T>
  {
    Up(const T *v, size_t n) { this->upload(v, n, nullptr); }
    explicit Up(const std::vector<T> &v) : Up(v.data(), v.size()) {}
  };

  template <typename T>
  void down(const DBuf<T> &b, T *out, size_t n)
  {
    b.download(out, n, nullptr);
    PIBEM_CUDA(cudaStreamSynchronize(nullptr));
  }
} // namespace

// The operator table of order p: nof M2L offsets, 8 M2M, 8 L2L, [in][out] each
extern "C" void kh_ops(int p, int nof, const int32_t *offsets, double *ops) { build_ops(p, nof, offsets, ops); }

// M2L products of the FP64-accurate operator, Y[q] = T_op(q) E[src(q)], (hi, lo) pairs; the pairs q
// sorted by operator.  digits: the tensor-core kernel, else the float-float GEMM.
extern "C" int kh_m2l(int p, int nof, const int32_t *offsets, int n_rows, const float *E, int n_pairs,
                      const int32_t *src, const int32_t *op_of, int digits, float *Y)
{
  return guarded([&] {
    const int           K = (p + 1) * (p + 1), nops = nof + 16;
    std::vector<double> ops(size_t(nops) * K * K);
    build_ops(p, nof, offsets, ops.data());
    std::vector<int32_t> start, cnt, op;
    for (int q = 0; q < n_pairs; ++q)
      if (q == 0 || op_of[q] != op_of[q - 1] || cnt.back() == 128)
        {
          start.push_back(q);
          cnt.push_back(1);
          op.push_back(op_of[q]);
        }
      else
        ++cnt.back();
    Up<double>     d_ops(ops);
    Up<int32_t>    d_start(start), d_cnt(cnt), d_op(op), d_src(src, n_pairs);
    Up<float2>     d_E(reinterpret_cast<const float2 *>(E), size_t(n_rows) * K);
    DBuf<float2>   d_off, d_Y;
    DBuf<uint16_t> img, slc;
    DBuf<int16_t>  ecol;
    DBuf<int>      erow, err;
    d_off.alloc(ops.size());
    launch_convert_d2ff(int64_t(ops.size()), d_ops.p, d_off.p, nullptr);
    d_Y.alloc(size_t(n_pairs) * K);
    img.alloc(ozaki_image_values(nops, K));
    ecol.alloc(ozaki_column_values(nops, K));
    slc.alloc(ozaki_slice_values(n_rows, K));
    erow.alloc(n_rows);
    err.alloc(1);
    err.zero(nullptr);
    launch_ozaki_images(d_ops.p, nops, K, img.p, ecol.p, nullptr);
    OperatorDev<double> o;
    o.K               = K;
    o.p               = p;
    o.ch_start        = d_start.p;
    o.ch_cnt          = d_cnt.p;
    o.ch_op           = d_op.p;
    o.q_src           = d_src.p;
    o.max_chunk_pairs = *std::max_element(cnt.begin(), cnt.end());
    o.ops_ff          = d_off.p;
    o.oz_images       = img.p;
    o.oz_ecol         = ecol.p;
    o.dev_err         = err.p;
    if (digits)
      {
        launch_ozaki_slices(n_rows, K, d_E.p, slc.p, erow.p, nullptr);
        launch_ozaki_gemm(o, 1, 0, int(cnt.size()), slc.p, erow.p, n_rows, d_Y.p, nullptr);
      }
    else
      launch_ff_gemm<float2>(o, 1, 0, int(cnt.size()), d_E.p, d_Y.p, nullptr);
    down(d_Y, reinterpret_cast<float2 *>(Y), size_t(n_pairs) * K);
    int e = 0;
    down(err, &e, 1);
    return e;
  });
}

// One L2L level of the FP32 operator: L[box] += T_octant L[par] for n boxes listed by octant (oct:
// the nine bounds), R columns.  ref != 0: the same sums on the host, chain by chain.
extern "C" int kh_l2l(int p, int R, int n_all, int n, const int32_t *box, const int32_t *par, const int32_t *oct,
                      int ref, float *L)
{
  return guarded([&] {
    const int           K = (p + 1) * (p + 1);
    std::vector<double> ops(size_t(16) * K * K);
    build_ops(p, 0, nullptr, ops.data());
    const size_t       lvk = fused_level_ops_floats(K) / 16;
    std::vector<float> lv(16 * lvk, 0.0f);
    for (int o = 0; o < 16; ++o)
      for (int i = 0; i < K * K; ++i)
        lv[o * lvk + i] = float(ops[size_t(o) * K * K + i]);
    if (ref)
      {
        for (int o = 0; o < 8; ++o)
          for (int i = oct[o]; i < oct[o + 1]; ++i)
            for (int r = 0; r < R; ++r)
              for (int k = 0; k < K; ++k)
                {
                  const float *T = &lv[(8 + o) * lvk], *x = L + (size_t(par[i]) * R + r) * K;
                  auto         chain = [&](int a, int b) {
                    float s = 0.0f;
                    for (int j = a; j < b; ++j)
                      s = std::fmaf(T[j * K + k], x[j], s);
                    return s;
                  };
                  L[(size_t(box[i]) * R + r) * K + k] +=
                    K <= 81 ? chain(0, K) :
                              (chain(0, K / 4) + chain(K / 4, K / 2)) + (chain(K / 2, 3 * K / 4) + chain(3 * K / 4, K));
                }
        return 0;
      }
    Up<float>   d_lv(lv), d_L(L, size_t(n_all) * R * K);
    Up<int32_t> d_box(box, n), d_par(par, n);
    DBuf<int>   err;
    err.alloc(1);
    err.zero(nullptr);
    OperatorDev<float> o;
    o.K        = K;
    o.p        = p;
    o.lv_ops   = d_lv.p;
    o.down_box = d_box.p;
    o.down_par = d_par.p;
    o.dev_err  = err.p;
    o.down_oct_ptr.resize(1);
    std::copy(oct, oct + 9, o.down_oct_ptr[0].p);
    launch_l2l_level_fused(o, R, 0, d_L.p, nullptr);
    down(d_L, L, size_t(n_all) * R * K);
    int e = 0;
    down(err, &e, 1);
    return e;
  });
}

// ILU(0) substitutions of R columns of z (n values each) with given factors (CSR, the diagonal's
// positions) and rows by level: a launch per level, else one block per column.
extern "C" int kh_ilu(int n, int R, const int64_t *ptr, const int32_t *col, const double *val, const int64_t *diag,
                      int n_lo, const int64_t *lptr_lo, const int32_t *rows_lo, int n_up, const int64_t *lptr_up,
                      const int32_t *rows_up, int by_level, double *z)
{
  return guarded([&] {
    Up<int64_t>  d_ptr(ptr, n + 1), d_diag(diag, n);
    Up<int32_t>  d_col(col, ptr[n]), d_lo(rows_lo, n), d_up(rows_up, n);
    Up<double>   d_val(val, ptr[n]), d_z(z, size_t(n) * R);
    DBuf<double> y;
    DBuf<int>    err;
    y.alloc(size_t(n) * R);
    err.alloc(1);
    err.zero(nullptr);
    if (by_level)
      launch_ilu_levels(std::vector<int64_t>(lptr_lo, lptr_lo + n_lo + 1), d_lo.p,
                        std::vector<int64_t>(lptr_up, lptr_up + n_up + 1), d_up.p, R, n, d_ptr.p, d_col.p, d_val.p,
                        d_diag.p, d_z.p, nullptr, nullptr, nullptr);
    else
      launch_ilu_apply(n, R, d_lo.p, d_up.p, d_ptr.p, d_col.p, d_val.p, d_diag.p, d_z.p, y.p, nullptr, nullptr,
                       err.p, nullptr);
    down(d_z, z, size_t(n) * R);
    int e = 0;
    down(err, &e, 1);
    return e;
  });
}

// P2M tables T1, T2 (rows of K4 values) of n_leaves leaves, the boxes 0 ... n_leaves - 1, with work
// for the points' expansions of work_bytes
extern "C" int kh_p2m_tables(int p, int n_leaves, const int64_t *row_ptr, const int64_t *contrib_ptr,
                             const int32_t *contrib_q, const double *center, const double *delta, int n_points,
                             const double *qpts, const double *qnrm, const double *qw, int64_t work_bytes,
                             double *T1, double *T2)
{
  return guarded([&] {
    const int            K = (p + 1) * (p + 1), K4 = (K + 3) / 4 * 4;
    const int64_t        rows = row_ptr[n_leaves];
    std::vector<int32_t> box(n_leaves);
    for (int i = 0; i < n_leaves; ++i)
      box[i] = i;
    Up<int64_t>  d_row(row_ptr, n_leaves + 1), d_cp(contrib_ptr, rows + 1);
    Up<int32_t>  d_cq(contrib_q, contrib_ptr[rows]), d_box(box);
    Up<double>   d_c(center, 3 * n_leaves), d_d(delta, n_leaves), d_p(qpts, 3 * n_points), d_n(qnrm, 3 * n_points),
      d_w(qw, 4 * n_points);
    DBuf<double> t1, t2;
    t1.alloc(rows * K4);
    t2.alloc(rows * K4);
    t1.zero(nullptr);
    t2.zero(nullptr);
    P2mTableArgs a;
    a.K = K, a.p = p, a.n_leaves = n_leaves;
    a.row_ptr = d_row.p, a.contrib_ptr = d_cp.p, a.h_row_ptr = row_ptr, a.h_contrib_ptr = contrib_ptr;
    a.leaf_box = d_box.p, a.contrib_q = d_cq.p, a.box_center = d_c.p, a.box_delta = d_d.p;
    a.n_points = n_points, a.qpts = d_p.p, a.qnrm = d_n.p, a.qw = d_w.p;
    a.work_bytes = size_t(work_bytes), a.T1 = t1.p, a.T2 = t2.p;
    launch_p2m_tables(a, nullptr);
    down(t1, T1, size_t(rows) * K4);
    down(t2, T2, size_t(rows) * K4);
    return 0;
  });
}
