// fft.cu -- FFTOperator (src/particle.jl:196-535): the transform between a
// position grid and its momentum grid, applied to kets, bras and operators.
//
// The reference multiplies by a phase array (mul_before), runs FFTW's in-place
// fft!/bfft! over the transformed dimensions, and multiplies by a second phase
// array that includes 1/sqrt(N) (mul_after); bras and the rows of an operator
// multiplied from the right go through conj -> opposite-sign transform -> conj,
// which is the same-sign transform of the row with the two phase arrays
// swapped (the DFT matrix is symmetric).  Both phase arrays are Kronecker
// products of per-axis vectors, so a multi-dimensional transform is one pass per
// axis, each pass multiplying by its axis's phases.
//
// Powers of two from 8 on: a thread owns eight elements of a line in registers and
// does radix-8 Stockham stages on them (Van Loan, Computational Frameworks for the
// FFT, 1992; one stage of radix 2 or 4 first where log2 n is no multiple of 3), with
// one exchange through shared memory between two stages; the first stage reads and the
// last one writes global memory.  Other lengths: a direct DFT on the even and odd
// parts of the line.  The last pass applies alpha and beta.
//
// What bounds it is the FP64 pipe, two lanes a clock and SM: 6.5 operations
// a point and radix-8 stage, 3.5 for its twiddles, 4 for each phase array.
// Measured against radix-2 stages through shared memory and the plain sum (a particle
// Hamiltonian, two transforms and two diagonals, us): 4096 points, 64 kets, ComplexF64 103 -> 84,
// ComplexF32 58 -> 36; 256 x 256 points, 8 kets 210 -> 188, double-float 122 -> 98; 800 points,
// 32 kets 2375 -> 117, one ket 2364 -> 42.
//
// In a product transform -- diagonal -- transform (a particle's kinetic energy) the
// first transform's last pass, the diagonal and the second one's first pass are one
// kernel, and a diagonal term beside that product (the potential) is added by the
// last store: 4096 points on 64 kets 84 -> 59 us (three launches for six), 64 points on
// one 30 -> 19 (one launch for four), 256 x 256 on 8 188 -> 152, double-float 92 -> 60.
#include <cmath>
#include <vector>

#include "fft_line.h"
#include "k_gather.cuh"  // DF

namespace qob {
namespace {

void upload_prec(DeviceBuf& d, const std::vector<c128>& v, int precision, bool ff) {
  if (ff) {  // (re hi, re lo, im hi, im lo)
    std::vector<float> q(4 * v.size());
    for (size_t i = 0; i < v.size(); ++i) {
      const float rh = (float)v[i].re, ih = (float)v[i].im;
      q[4 * i] = rh;
      q[4 * i + 1] = (float)(v[i].re - (double)rh);
      q[4 * i + 2] = ih;
      q[4 * i + 3] = (float)(v[i].im - (double)ih);
    }
    d.upload(q.data(), q.size() * sizeof(float));
  } else if (precision == QOB_C128) {
    d.upload(v.data(), v.size() * sizeof(c128));
  } else {
    std::vector<c64> f(v.size());
    for (size_t i = 0; i < v.size(); ++i) f[i] = {(float)v[i].re, (float)v[i].im};
    d.upload(f.data(), f.size() * sizeof(c64));
  }
}

}  // namespace

// f with the arithmetic type of a plan
template <typename F>
static void with_form(int precision, bool ff, F f) {
  if (ff)
    f(gather::DF{});
  else if (precision == QOB_C128)
    f(double{});
  else
    f(float{});
}

void launch_fft_pass(Context& ctx, const Plan& P, size_t a, const void* x, int64_t xes, int64_t xcs, const FftOut& o,
                     int64_t ncols, void* scratch, cudaStream_t s) {
  with_form(P.precision, P.ff, [&](auto r) {
    fft_axis<decltype(r)>(P.fft[a], P.m, x, xes, xcs, o, ncols, scratch, ctx.num_sms, s);
  });
}

bool gather_is_diagonal(const GatherPlan& g) {
  return g.has_diag && g.ngroups == 0 && g.square && !g.phased && g.diag.p;
}

// One diagonal alone: no other groups, passes or sub-plans.
static bool plan_is_diagonal(const Plan& P) {
  return P.kind == Plan::Kind::Sum && P.gather && P.dense.empty() && P.modek.empty() && P.subs.empty() &&
         gather_is_diagonal(*P.gather);
}
// Marks the first transform -- diagonal -- transform of a product whose last axis has an
// FFT: P.turn, and P.mid = the phases between the two (after the first, before the
// second) of that axis.  ops: the factors in application order.
void find_fft_turn(Plan& P, const std::vector<const OpNode*>& ops) {
  for (size_t i = 0; i + 2 < P.chain.size(); ++i) {
    const Plan &A = *P.chain[i], &D = *P.chain[i + 1], &B = *P.chain[i + 2];
    if (A.kind != Plan::Kind::Fft || B.kind != Plan::Kind::Fft || !plan_is_diagonal(D) || D.gather->ff != P.ff || A.fft.size() != B.fft.size() ||
        D.m != A.m || A.m != B.m)
      continue;
    bool same = A.fft.back().pow2;
    for (size_t a = 0; a < A.fft.size(); ++a)
      same = same && A.fft[a].n == B.fft[a].n && A.fft[a].stride == B.fft[a].stride;
    if (!same) continue;
    const int64_t n = A.fft.back().n;
    const bool right = P.side == QOB_RIGHT;
    const std::vector<c128>& post = right ? ops[i]->fft_before : ops[i]->fft_after;
    const std::vector<c128>& pre = right ? ops[i + 2]->fft_after : ops[i + 2]->fft_before;
    std::vector<c128> mid((size_t)n);
    for (int64_t k = 0; k < n; ++k) mid[k] = cmul(post[post.size() - n + k], pre[pre.size() - n + k]);
    upload_prec(P.mid, mid, P.precision, P.ff);
    P.turn = (int)i;
    return;
  }
}

// The three factors at P.turn.  The last axis of the first transform, the diagonal and that
// axis of the second are one pass (three launches in the four-step form), the
// other axes a pass each.  False (nothing done) where the passes one by one are faster: a
// last axis of several whose lines only the four-step form spreads.  Uses slots ws .. ws + 2.
bool launch_fft_turn(Context& ctx, const Plan& P, const void* x, int64_t xes, int64_t xcs, const FftOut& o,
                     int64_t ncols, cudaStream_t s, int ws) {
  const Plan &A = *P.chain[P.turn], &B = *P.chain[P.turn + 2];
  const GatherPlan& d = *P.chain[P.turn + 1]->gather;
  const size_t q = A.fft.size(), esz = P.precision == QOB_C128 ? 16 : 8, bytes = (size_t)P.m * ncols * esz;
  const int64_t lines = A.m / A.fft.back().n * ncols;
  const bool steps = four_step(A.fft.back(), lines, ctx.num_sms);
  if (q > 1 && (steps || (o.add && !A.fft.front().pow2))) return false;
  const void* src = x;
  int64_t ses = xes, scs = xcs;
  int slot = 0;
  auto temp = [&]() {
    void* t = ctx.ws.get(ws + slot, bytes);
    slot ^= 1;
    return FftOut{t, 1, A.m, {1.0, 0.0}, {0.0, 0.0}, nullptr, nullptr, 0, 0};
  };
  auto advance = [&](const FftOut& t) {
    src = t.y;
    ses = 1;
    scs = A.m;
  };
  for (size_t a = 0; a + 1 < q; ++a) {
    const FftOut t = temp();
    launch_fft_pass(ctx, A, a, src, ses, scs, t, ncols, nullptr, s);
    advance(t);
  }
  const FftOut t = q == 1 ? o : temp();
  void* s1 = steps ? ctx.ws.get(ws, bytes) : nullptr;
  void* s2 = steps ? ctx.ws.get(ws + 1, bytes) : nullptr;
  with_form(P.precision, P.ff, [&](auto r) {
    fft_turn<decltype(r)>(A.fft.back(), B.fft.back(), d, P.mid.p, A.m, src, ses, scs, t, ncols, s1, s2, ctx.num_sms, s);
  });
  if (q == 1) return true;
  advance(t);
  for (size_t a = q - 1; a-- > 0;) {
    const FftOut u = a == 0 ? o : temp();
    void* scratch = a == 0 && B.fft[a].n1 > 0 ? ctx.ws.get(ws + 2, bytes) : nullptr;
    launch_fft_pass(ctx, B, a, src, ses, scs, u, ncols, scratch, s);
    if (a > 0) advance(u);
  }
  return true;
}

// LEFT (kets, operator columns): pre = before, post = after.  RIGHT (bras,
// operator rows): pre = after, post = before, same sign.
std::unique_ptr<Plan> compile_fft(const NodeP& op, int side, int precision_code) {
  const bool ff = precision_code == QOB_C128X;
  const int precision = ff ? QOB_C128 : precision_code;
  auto P = std::make_unique<Plan>();
  P->kind = Plan::Kind::Fft;
  P->side = side;
  P->precision = precision;
  P->ff = ff;
  P->m = side == QOB_RIGHT ? op->n : op->m;
  P->n = side == QOB_RIGHT ? op->m : op->n;
  P->root = op.get();
  const std::vector<int64_t>& shape = op->shape_l;
  int64_t off = 0;
  for (size_t a = 0; a < op->fft_sites.size(); ++a) {
    const int site = op->fft_sites[a];
    FftAxis ax;
    ax.n = shape[site];
    ax.stride = 1;
    for (int q = 0; q < site; ++q) ax.stride *= shape[q];
    ax.pow2 = (ax.n & (ax.n - 1)) == 0 && ax.n >= 8;
    const size_t esz = precision == QOB_C128 ? 16 : 8;
    const size_t smem = ((ax.n & (ax.n - 1)) == 0 && ax.n >= 2 ? 2 : 1) * (size_t)ax.n * esz;
    if (smem > 200 * 1024) fail(QOB_ERR_UNSUPPORTED, "FFT axis too long for one block's shared memory");
    ax.sign = op->fft_sign[a] < 0 ? -1 : 1;
    std::vector<c128> tw((size_t)ax.n);
    for (int64_t m = 0; m < ax.n; ++m) {
      const double th = 6.283185307179586476925286766559 * (double)m / (double)ax.n;
      tw[(size_t)m] = {std::cos(th), ax.sign * std::sin(th)};
    }
    std::vector<c128> before(op->fft_before.begin() + off, op->fft_before.begin() + off + ax.n);
    std::vector<c128> after(op->fft_after.begin() + off, op->fft_after.begin() + off + ax.n);
    off += ax.n;
    upload_prec(ax.tw, tw, precision, ff);
    if (ax.pow2 && ax.n >= 512) {
      ax.n1 = int64_t(1) << (log2_of(ax.n) / 2);
      ax.n2 = ax.n / ax.n1;
    }
    upload_prec(ax.pre, side == QOB_RIGHT ? after : before, precision, ff);
    upload_prec(ax.post, side == QOB_RIGHT ? before : after, precision, ff);
    P->fft.push_back(std::move(ax));
  }
  return P;
}

}  // namespace qob

namespace {
qob_op* wrap_node(qob::NodeP n) {
  auto* h = new qob_op;
  h->node = std::move(n);
  return h;
}
}  // namespace

extern "C" int qob_op_fft(qob_ctx* ctx, int nsub, const int64_t* shape, int naxes, const int64_t* axes,
                          const int* sign, const double* before, const double* after, qob_op** out) {
  if (!ctx) return QOB_ERR_ARG;
  try {
    using namespace qob;
    if (!out || nsub < 1 || nsub > kMaxSites || !shape || naxes < 1 || naxes > nsub || !axes || !sign || !before ||
        !after)
      fail(QOB_ERR_ARG, "qob_op_fft: bad arguments");
    auto nd = std::make_shared<OpNode>();
    nd->kind = Kind::Fft;
    nd->shape_l.assign(shape, shape + nsub);
    nd->shape_r = nd->shape_l;
    int64_t len = 1;
    for (int i = 0; i < nsub; ++i) {
      if (shape[i] < 1) fail(QOB_ERR_ARG, "qob_op_fft: bad subsystem length");
      len *= shape[i];
    }
    if (len > INT32_MAX) fail(QOB_ERR_UNSUPPORTED, "dimension exceeds 2^31-1");
    nd->m = nd->n = len;
    int64_t total = 0;
    for (int a = 0; a < naxes; ++a) {
      if (axes[a] < 1 || axes[a] > nsub || (a > 0 && axes[a] <= axes[a - 1]))
        fail(QOB_ERR_ARG, "qob_op_fft: axes must be increasing 1-based subsystem indices");
      nd->fft_sites.push_back((int)axes[a] - 1);
      nd->fft_sign.push_back(sign[a] < 0 ? -1 : 1);
      total += shape[axes[a] - 1];
    }
    for (int64_t k = 0; k < total; ++k) {
      nd->fft_before.push_back({before[2 * k], before[2 * k + 1]});
      nd->fft_after.push_back({after[2 * k], after[2 * k + 1]});
    }
    *out = wrap_node(nd);
    return QOB_OK;
  } catch (const qob::Error& e) {
    ctx->c.err = e.msg;
    return e.code;
  }
}
