// Test harness: single launches of the library's kernels, linked against libpibem_gb300.so, for
// what the C ABI shows only through whole operators.  Host arrays in and out; every function
// returns the device error flag (0: none) or -1 after an exception.
#include <algorithm>
#include <cstdio>
#include <exception>
#include <vector>

#include "../../pi-bem_gb300/csrc/kernels.h"

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
