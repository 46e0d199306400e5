// The launches of a Mamba-2 block's mixer (convolution, step sizes, chunked scan, skip connection, output gate), forward and backward, from one call:
// the sequence of entry points that ops/ssm.py describes, in its order and with its arguments, for the sizes whose products read their operands in
// place (chunks, head and state sizes that are multiples of 64). No kernels of its own.
// Why: 9 and 27 entry points through Python, each with a dozen converted arguments, a stream lookup and an allocation, kept the host busy for 1.0 ms
// of a block of width 768 whose kernels take 0.4 ms. Scratch is one block that the caller allocates (sx_mixer_workspace).
#include "sx_api.h"

namespace sx {

typedef uint16_t h16;   // bf16 storage

// One walk over the sequence: with `run` off it only finds out how much scratch it takes.
struct Mixer {
  const SxMixerArgs& a;
  cudaStream_t st;
  const bool run;
  int rc = 0;
  long long used = 0;   // bytes of scratch
  // sizes: chunks of a sequence, (chunk, group) matrices, heads of a group, inner width, convolution channels, projection width
  const int nc, rep, di, C;
  const long long n, W, Lp, BC, rP;

  Mixer(const SxMixerArgs& args, cudaStream_t stream, bool go)
      : a(args), st(stream), run(go), nc((args.L + args.Q - 1) / args.Q), rep(args.H / args.G), di(args.H * args.P),
        C(args.H * args.P + 2 * args.G * args.N), n((long long)args.B * nc * args.G), W((long long)di + C + args.H), Lp((long long)nc * args.Q),
        BC((long long)args.B * nc), rP((long long)rep * args.P) {}

  // Buffers in the order of their addresses: take() fills the first gap that is wide enough, drop() gives one back when the last launch that reads it
  // has been issued (they run one after another).
  struct Range { long long at, end; } held[48];
  int n_held = 0;
  char* base() const { return a.work ? static_cast<char*>(a.work) : reinterpret_cast<char*>(256); }   // without scratch: sizes only
  template <typename T>
  T* take(long long count) {
    const long long bytes = (count * (long long)sizeof(T) + 255) / 256 * 256;
    long long at = 0;
    int i = 0;
    for (; i < n_held && held[i].at - at < bytes; ++i) at = held[i].end;
    if (n_held == (int)(sizeof(held) / sizeof(held[0]))) { rc = -3; return nullptr; }
    for (int j = n_held++; j > i; --j) held[j] = held[j - 1];
    held[i] = {at, at + bytes};
    if (at + bytes > used) used = at + bytes;
    return reinterpret_cast<T*>(base() + at);
  }
  void drop(const void* p) {
    int i = 0;
    while (i < n_held && base() + held[i].at != p) ++i;
    if (i == n_held) { rc = -3; return; }
    for (--n_held; i < n_held; ++i) held[i] = held[i + 1];
  }
  template <typename... P>
  void drop(const void* p, P... more) { drop(p); drop(more...); }
  template <typename F>
  void go(F&& f) {
    if (run && rc == 0) rc = f();
  }
  void check(cudaError_t e) {
    if (e != cudaSuccess && rc == 0) rc = -11;
  }
  struct Mat { const void* p; long long ld, stride; bool mn; };   // row pitch, pitch of the batch, reduction over the rows

  // D [batch, M, N] = A B^T (+ D), D dense
  void gemm(Mat A, Mat B, void* D, long long M, long long N, long long K, long long batch, bool f32, bool add = false) {
    go([&] {
      SxGemmArgs g = {};
      g.A = A.p; g.B = B.p; g.D = D;
      g.M = (int)M; g.N = (int)N; g.K = (int)K; g.batch = (int)batch;
      g.lda = A.ld; g.ldb = B.ld; g.ldd = N;
      g.strideA = A.stride; g.strideB = B.stride; g.strideD = M * N;
      g.a_mn = A.mn; g.b_mn = B.mn;
      g.out_fp32 = f32;
      g.alpha = 1.f;
      if (add) { g.C = D; g.ldc = N; g.strideC = M * N; g.c_fp32 = f32; g.beta = 1.f; }
      g.status = a.status;
      return sx_gemm_bf16(&g, st);
    });
  }

  float *dth, *csh, *E, *decay, *tot;
  Mat Bg, Cg;   // by (chunk, group), [n, Q, N]: in the convolution's output for one group, packed otherwise

  void prep() {
    const long long v = BC * a.H * a.Q;
    dth = take<float>(v); csh = take<float>(v); E = take<float>(v); decay = take<float>(v); tot = take<float>(BC * a.H);
    go([&] { return sx_mix_prep((const h16*)a.zx + W - a.H, W, a.dt_bias, a.a_log, dth, csh, E, decay, tot, a.B, nc, a.L, a.H, a.Q, st); });
    const h16* x = (const h16*)a.xbc;
    if (a.G == 1) {
      Bg = {x + di, C, (long long)a.Q * C, false};
      Cg = {x + di + a.N, C, (long long)a.Q * C, false};
      return;
    }
    const long long one = n * a.Q * a.N;
    h16* out = take<h16>(2 * one);
    go([&] { return sx_mix_pack(x + di, C, out, BC * a.Q, a.G, a.Q, a.N, st); });
    Bg = {out, a.N, (long long)a.Q * a.N, false};
    Cg = {out + one, a.N, (long long)a.Q * a.N, false};
  }
  Mat mn(Mat m) { m.mn = true; return m; }
  Mat dense(const void* p, long long rows, long long cols, bool over_rows = false) { return {p, cols, rows * cols, over_rows}; }
  h16* scaled_rows() {
    h16* xw = take<h16>(BC * a.Q * di);
    go([&] { return sx_ssd_scale_rows(a.xbc, decay, xw, BC * a.Q * a.H, a.P, a.H, C, a.Q, a.G, st); });
    return xw;
  }
  h16* heads_first(const void* t, long long ld) {
    h16* out = take<h16>(BC * a.Q * di);
    go([&] { return sx_ssd_heads_first(t, ld, out, BC * a.H * a.Q, a.H, a.Q, a.P, st); });
    return out;
  }
  void zero_tail(void* t, long long cols) {   // rows behind each sequence of a [B, Lp, cols] tensor
    if (run && Lp > a.L) check(cudaMemset2DAsync((h16*)t + a.L * cols, Lp * cols * 2, 0, (Lp - a.L) * cols * 2, a.B, st));
  }

  void forward() {
    const int Q = a.Q, N = a.N, P = a.P, H = a.H;
    zero_tail(a.xbc, C);
    go([&] { return sx_conv1d_fwd((const h16*)a.zx + di, nullptr, a.conv_w, a.conv_b, a.xbc, nullptr, a.B, a.L, C, a.K, 1, W, (int)Lp, st); });
    prep();
    float* S = take<float>(n * rP * N);
    h16* xw = scaled_rows();
    gemm(dense(xw, Q, rP, true), mn(Bg), S, rP, N, Q, n, true);
    drop(xw, decay);
    float* fin = take<float>((long long)a.B * H * P * N);
    go([&] { return sx_ssd_state_fwd(S, tot, nullptr, a.hprev, fin, a.B, nc, H, P * N, st); });
    drop(S, fin);
    const h16* x = (const h16*)a.xbc;
    if (a.fused) {
      go([&] { return sx_ssd_chunk_fwd(x + di + a.G * N, C, x + di, C, x, C, a.hprev, csh, dth, a.D, a.y, BC, H, a.G, a.status, st); });
    } else {
      float* CB = take<float>(n * Q * Q);
      gemm(Cg, Bg, CB, Q, Q, N, n, true);
      h16* M = take<h16>(BC * H * Q * Q);
      go([&] { return sx_ssd_build_m(CB, csh, dth, M, BC, H, a.G, Q, st); });
      drop(CB);
      h16 *xh = heads_first(x, C), *Yi = take<h16>(BC * Q * di);
      gemm(dense(M, Q, Q), dense(xh, Q, P, true), Yi, Q, P, Q, BC * H, false);
      drop(M, xh);
      h16* Yo = take<h16>(BC * Q * di);
      gemm(Cg, dense(a.hprev, rP, N), Yo, Q, rP, N, n, false);
      go([&] { return sx_ssd_combine(Yi, Yo, x, E, a.D, a.y, BC * Q * H, H, Q, P, C, a.G, st); });
    }
    go([&] { return sx_gate_mul_fwd(a.y, a.zx, W, a.out, (long long)a.B * a.L, di, a.L, (int)Lp, st); });
  }

  void backward() {
    const int Q = a.Q, N = a.N, P = a.P, H = a.H;
    const long long rows = (long long)a.B * a.L, vec = BC * Q * H, states = n * rP * N, toks = BC * Q * di;
    const h16* x = (const h16*)a.xbc;
    h16* dy = take<h16>(toks);
    zero_tail(dy, di);
    go([&] { return sx_gate_mul_bwd(a.g, a.y, a.zx, W, dy, a.dzx, rows, di, a.L, (int)Lp, W, st); });
    prep();
    // contribution of earlier chunks, and through them the chunk states
    h16 *Yo = take<h16>(toks), *dye = take<h16>(toks);
    float *dcs = take<float>(vec), *ddrow = take<float>(vec);
    gemm(Cg, dense(a.hprev, rP, N), Yo, Q, rP, N, n, false);
    go([&] { return sx_ssd_bwd_rows1(dy, x, Yo, E, dye, dcs, ddrow, vec, P, H, C, Q, a.G, st); });
    drop(Yo, E);
    float *dC = take<float>(n * Q * N), *dHp = take<float>(states);
    gemm(dense(dye, Q, rP), dense(a.hprev, rP, N, true), dC, Q, N, rP, n, true);
    gemm(dense(dye, Q, rP, true), mn(Cg), dHp, rP, N, Q, n, true);
    drop(dye);
    h16* dS = take<h16>(states);
    float *dtot = take<float>(BC * H), *dinit = take<float>((long long)a.B * H * P * N);
    if (run) check(cudaMemsetAsync(dtot, 0, BC * H * sizeof(float), st));
    go([&] { return sx_ssd_state_bwd(dHp, tot, a.hprev, nullptr, dS, dtot, dinit, a.B, nc, H, P * N, st); });
    drop(dHp, dinit);
    h16* dxw = take<h16>(toks);
    gemm(Bg, dense(dS, rP, N), dxw, Q, rP, N, n, false);
    float* dB = take<float>(n * Q * N);
    h16* xw = scaled_rows();
    gemm(dense(xw, Q, rP), dense(dS, rP, N, true), dB, Q, N, rP, n, true);
    drop(xw, dS);
    // quadratic term within the chunk
    h16 *dyh = heads_first(dy, di), *xh = heads_first(x, C), *dM = take<h16>(BC * H * Q * Q);
    gemm(dense(dyh, Q, P), dense(xh, Q, P), dM, Q, Q, P, BC * H, false);
    drop(xh);
    float *CB = take<float>(n * Q * Q), *rowW = take<float>(vec), *colU = take<float>(vec);
    gemm(Cg, Bg, CB, Q, Q, N, n, true);
    h16 *M = take<h16>(BC * H * Q * Q), *dGh = take<h16>(BC * H * Q * Q);
    go([&] { return sx_ssd_bwd_qq(dM, CB, csh, dth, M, dGh, rowW, colU, BC, H, a.G, Q, st); });
    drop(dM, CB);
    h16* dxi = take<h16>(toks);
    gemm(dense(M, Q, Q, true), dense(dyh, Q, P, true), dxi, Q, P, Q, BC * H, false);
    drop(M, dyh);
    h16* dxbc = take<h16>(BC * Q * C);
    float* ddecay = take<float>(vec);
    go([&] { return sx_ssd_bwd_rows2(dy, x, dxw, dxi, decay, a.D, dxbc, ddecay, vec, H, Q, P, C, a.G, C, st); });
    drop(dy, dxw, dxi);
    const h16* dG = dGh;
    if (rep > 1) {
      h16* sum = take<h16>(n * Q * Q);
      go([&] { return sx_mix_sum(dGh, sum, n, rep, Q * Q, st); });
      dG = sum;
    }
    gemm(dense(dG, Q, Q), mn(Bg), dC, Q, N, Q, n, true, true);
    gemm(dense(dG, Q, Q, true), mn(Cg), dB, Q, N, Q, n, true, true);
    go([&] { return sx_mix_unpack(dB, dC, dxbc + di, C, BC * Q, a.G, Q, N, st); });
    // convolution and step sizes
    float* partial = take<float>((long long)sx_conv1d_bwd_parts(a.B, a.L, C) * (a.K + 1) * C);
    go([&] {
      return sx_conv1d_bwd(dxbc, (const h16*)a.zx + di, nullptr, a.conv_w, a.conv_b, (h16*)a.dzx + di, partial, a.dwdb, a.B, a.L, C, a.K, 1, W, (int)Lp,
                           W, st);
    });
    go([&] {
      return sx_mix_finish((const h16*)a.zx + W - H, W, a.dt_bias, a.a_log, dth, csh, ddecay, dcs, ddrow, rowW, colU, dtot, tot,
                           (h16*)a.dzx + W - H, W, a.part, a.B, nc, a.L, H, Q, st);
    });
  }
};

static bool mixer_ok(const SxMixerArgs& a) {
  return a.B > 0 && a.L > 0 && a.G > 0 && a.H % a.G == 0 && a.Q % 64 == 0 && a.Q >= 64 && a.Q <= 128 && a.P % 64 == 0 && a.P > 0 && a.P <= 256 &&
         a.N % 64 == 0 && a.N > 0 && (!a.fused || (a.Q == 128 && a.N == 128 && a.P == 64));
}
static int mixer_call(const SxMixerArgs& a, cudaStream_t st, bool back) {
  if (!mixer_ok(a) || !a.work) return -1;
  Mixer size(a, st, false);
  back ? size.backward() : size.forward();
  if (size.rc) return size.rc;
  if (size.used > a.work_bytes) return -2;
  Mixer m(a, st, true);
  back ? m.backward() : m.forward();
  return m.rc;
}

}  // namespace sx

// Bytes of scratch of sx_mixer_fwd (backward = 0) or sx_mixer_bwd; negative: sizes that these do not take.
extern "C" long long sx_mixer_workspace(const SxMixerArgs* a, int backward) {
  if (!sx::mixer_ok(*a)) return -1;
  sx::Mixer m(*a, nullptr, false);
  backward ? m.backward() : m.forward();
  return m.rc ? m.rc : m.used;
}
extern "C" int sx_mixer_fwd(const SxMixerArgs* a, cudaStream_t st) { return sx::mixer_call(*a, st, false); }
extern "C" int sx_mixer_bwd(const SxMixerArgs* a, cudaStream_t st) { return sx::mixer_call(*a, st, true); }
