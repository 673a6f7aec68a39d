// Host driver of the learned MVC weight field: parameter block, batches,
// the training step sequence and the per-frame projection (field.h).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "field.h"

namespace cgs {

#define FIELD_TRY(x)                   \
  do {                                 \
    const cudaError_t e_ = (x);        \
    if (e_ != cudaSuccess) return e_;  \
  } while (0)

cudaError_t FieldBuf::ensure(size_t bytes, cudaStream_t s) {
  if (bytes == 0) bytes = 16;
  if (bytes <= cap) return cudaSuccess;
  if (p) cudaFree(p);
  p = nullptr;
  cap = 0;
  FIELD_TRY(cudaMalloc(&p, bytes));
  cap = bytes;
  return cudaMemsetAsync(p, 0, bytes, s);
}

namespace {

uint64_t splitmix64(uint64_t& s) {
  uint64_t z = (s += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// Standard normal samples by the Box-Muller transform on splitmix64 uniforms.
double normal(uint64_t& s) {
  const double u1 = ((splitmix64(s) >> 11) + 1.0) * (1.0 / 9007199254740993.0);
  const double u2 = (splitmix64(s) >> 11) * (1.0 / 9007199254740992.0);
  return std::sqrt(-2.0 * std::log(u1)) * std::cos(6.283185307179586 * u2);
}

uint32_t pad8(uint32_t v) { return (v + 7u) & ~7u; }

// Inverse of a 4 x 4 matrix by Gauss-Jordan elimination with partial
// pivoting; false when singular.
bool invert4(const double (&a)[4][4], double (&inv)[4][4]) {
  double m[4][8];
  for (int i = 0; i < 4; ++i)
    for (int j = 0; j < 8; ++j) m[i][j] = j < 4 ? a[i][j] : (j - 4 == i ? 1.0 : 0.0);
  for (int c = 0; c < 4; ++c) {
    int piv = c;
    for (int r = c + 1; r < 4; ++r)
      if (std::fabs(m[r][c]) > std::fabs(m[piv][c])) piv = r;
    if (!(std::fabs(m[piv][c]) > 0.0)) return false;
    if (piv != c)
      for (int j = 0; j < 8; ++j) std::swap(m[c][j], m[piv][j]);
    const double d = 1.0 / m[c][c];
    for (int j = 0; j < 8; ++j) m[c][j] *= d;
    for (int r = 0; r < 4; ++r)
      if (r != c) {
        const double f = m[r][c];
        for (int j = 0; j < 8; ++j) m[r][j] -= f * m[c][j];
      }
  }
  for (int i = 0; i < 4; ++i)
    for (int j = 0; j < 4; ++j) inv[i][j] = m[i][j + 4];
  return true;
}

}  // namespace

cudaError_t FieldState::init(uint32_t nv, const float* rest_v4, uint64_t seed, cudaStream_t s) {
  V = nv;
  ldV = pad8(nv);
  const uint32_t sizes[kFieldParams] = {kFieldHid * kFieldIn, kFieldHid, kFieldHid * kFieldHid,
                                        kFieldHid,            kFieldHid * kFieldHid, kFieldHid,
                                        kFieldHid * kFieldHid, kFieldHid, nv * kFieldHid, nv};
  uint32_t o = 0;
  for (int k = 0; k < kFieldParams; ++k) {
    off[k] = o;
    o += pad8(sizes[k]);
  }
  off[kFieldParams] = o;
  // encoding: centre and half-extent of the rest cage's bounding box
  float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (uint32_t j = 0; j < nv; ++j)
    for (int d = 0; d < 3; ++d) {
      lo[d] = std::min(lo[d], rest_v4[4 * j + d]);
      hi[d] = std::max(hi[d], rest_v4[4 * j + d]);
    }
  scale = 0.5f * std::max(hi[0] - lo[0], std::max(hi[1] - lo[1], hi[2] - lo[2]));
  if (!(scale > 0.0f)) scale = 1.0f;
  for (int d = 0; d < 3; ++d) enc[d] = 0.5f * (lo[d] + hi[d]);
  enc[3] = 1.0f / scale;
  // M = (Vb Vb^T)^-1, Vb = [1; v_j] over the rest vertices
  double G[4][4] = {}, Gi[4][4];
  for (uint32_t j = 0; j < nv; ++j) {
    const double b[4] = {1.0, rest_v4[4 * j], rest_v4[4 * j + 1], rest_v4[4 * j + 2]};
    for (int a = 0; a < 4; ++a)
      for (int c = 0; c < 4; ++c) G[a][c] += b[a] * b[c];
  }
  if (!invert4(G, Gi)) return cudaErrorInvalidValue;  // degenerate (flat) cage
  for (int a = 0; a < 4; ++a)
    for (int c = 0; c < 4; ++c) M.m[4 * a + c] = (float)Gi[a][c];
  std::vector<float> h(o, 0.0f);
  uint64_t st = seed * 0x2545F4914F6CDD1Dull + 1;
  const int fan[4] = {kFieldIn, kFieldHid, kFieldHid, kFieldHid};
  const int wl[4] = {kW1, kW2, kW3, kW4};
  for (int l = 0; l < 4; ++l) {
    const double sd = std::sqrt(2.0 / fan[l]);
    for (uint32_t i = 0; i < sizes[wl[l]]; ++i) h[off[wl[l]] + i] = (float)(sd * normal(st));
  }
  for (uint32_t i = 0; i < sizes[kW5]; ++i) h[off[kW5] + i] = (float)(1e-3 * normal(st));
  for (uint32_t j = 0; j < nv; ++j) h[off[kB5] + j] = 1.0f / (float)nv;
  FIELD_TRY(p32.ensure((size_t)o * 4, s));
  FIELD_TRY(g32.ensure((size_t)o * 4, s));
  FIELD_TRY(m1.ensure((size_t)o * 4, s));
  FIELD_TRY(m2.ensure((size_t)o * 4, s));
  FIELD_TRY(pb.ensure((size_t)o * 2, s));
  FIELD_TRY(enc_d.ensure(16, s));
  FIELD_TRY(M_d.ensure(64, s));
  FIELD_TRY(rest_d.ensure((size_t)nv * 16, s));
  FIELD_TRY(proj.ensure((size_t)kFieldProj * 4, s));
  FIELD_TRY(proj_rest.ensure((size_t)kFieldProj * 4, s));
  FIELD_TRY(loss.ensure(16, s));
  FIELD_TRY(status.ensure(16, s));
  FIELD_TRY(wT.ensure((size_t)kFieldHid * (3 * kFieldHid + ldV) * 2, s));
  FIELD_TRY(cudaMemsetAsync(m1.p, 0, (size_t)o * 4, s));
  FIELD_TRY(cudaMemsetAsync(m2.p, 0, (size_t)o * 4, s));
  FIELD_TRY(cudaMemsetAsync(g32.p, 0, (size_t)o * 4, s));
  FIELD_TRY(cudaMemcpyAsync(enc_d.p, enc, 16, cudaMemcpyHostToDevice, s));
  FIELD_TRY(cudaMemcpyAsync(M_d.p, M.m, 64, cudaMemcpyHostToDevice, s));
  FIELD_TRY(cudaMemcpyAsync(rest_d.p, rest_v4, (size_t)nv * 16, cudaMemcpyHostToDevice, s));
  step = 0;
  FIELD_TRY(cudaMemcpyAsync(p32.p, h.data(), (size_t)o * 4, cudaMemcpyHostToDevice, s));
  FIELD_TRY(refresh(s));
  return cudaStreamSynchronize(s);  // h goes out of scope
}

FieldNet FieldState::net() const {
  FieldNet n;
  const __nv_bfloat16* b = pb.as<__nv_bfloat16>();
  const float* f = p32.as<float>();
  n.W1b = b + off[kW1];
  n.W2b = b + off[kW2];
  n.W3b = b + off[kW3];
  n.W4b = b + off[kW4];
  n.W5b = b + off[kW5];
  n.b1 = f + off[kB1];
  n.b2 = f + off[kB2];
  n.b3 = f + off[kB3];
  n.b4 = f + off[kB4];
  n.b5 = f + off[kB5];
  return n;
}

BatchLayout::BatchLayout(uint32_t B, uint32_t V, uint32_t ldV, bool train) {
  size_t at = 0;
  auto take = [&](size_t n) {
    const size_t p = at;
    at = (at + n + 255) & ~(size_t)255;
    return p;
  };
  const size_t b = B, H = kFieldHid;
  x = take(b * 12);
  idx = take(b * 4);
  a0 = take(b * kFieldIn * 2);
  for (int l = 0; l < 4; ++l) {
    pre[l] = take(b * H * 4);
    h[l] = take(b * H * 2);
  }
  z = take(b * ldV * 4);
  if (train) {
    dzb = take(b * ldV * 2);
    for (int l = 0; l < 2; ++l) dpreb[l] = take(b * H * 2);
    for (int l = 0; l < 5; ++l) {
      inT[l] = take((l == 0 ? kFieldIn : H) * b * 2);
      dT[l] = take((l == 4 ? ldV : H) * b * 2);
      if (l < 4) dpre[l] = take(b * H * 4);
    }
    dz = take(b * ldV * 4);
    for (int l = 0; l < 5; ++l)
      ws[l] = take((size_t)grad_splits(B) * (l == 4 ? V : H) * (l == 0 ? kFieldIn : H) * 4);
  }
  bytes = at;
}

void FieldState::transposed(__nv_bfloat16* (&w)[4]) const {
  for (int l = 0; l < 4; ++l) w[l] = wT.as<__nv_bfloat16>() + (size_t)l * kFieldHid * kFieldHid;
}

cudaError_t FieldState::refresh(cudaStream_t s) {
  __nv_bfloat16* w[4];
  transposed(w);
  return launch_field_refresh(off, V, ldV, p32.as<float>(), pb.as<__nv_bfloat16>(), w, s);
}

cudaError_t FieldState::forward(const float* points, const float* target, uint32_t n, uint32_t B,
                                uint32_t seed, const float4* rest_verts, float lambda,
                                cudaStream_t s) {
  const bool train = target != nullptr;
  const BatchLayout L(B, V, ldV, train);
  FIELD_TRY(batch.ensure(L.bytes, s));
  FieldBatch fb{};
  fb.points = points;
  fb.n = n;
  fb.B = B;
  fb.seed = seed;
  fb.enc = enc_d.as<float>();
  fb.x = batch.at<float>(L.x);
  fb.idx = batch.at<uint32_t>(L.idx);
  fb.a0 = batch.at<__nv_bfloat16>(L.a0);
  fb.a0T = train ? batch.at<__nv_bfloat16>(L.inT[0]) : nullptr;
  FIELD_TRY(launch_field_gather(fb, s));
  const FieldNet nt = net();
  const __nv_bfloat16* W[4] = {nt.W1b, nt.W2b, nt.W3b, nt.W4b};
  const float* bias[4] = {nt.b1, nt.b2, nt.b3, nt.b4};
  for (int l = 0; l < 4; ++l) {
    GemmArgs g{};
    g.status = status.as<uint32_t>();
    g.A = batch.at<__nv_bfloat16>(l == 0 ? L.a0 : L.h[l - 1]);
    g.lda = g.K = l == 0 ? kFieldIn : kFieldHid;
    g.B = W[l];
    g.ldb = g.K;
    g.M = B;
    g.N = kFieldHid;
    g.C = batch.at<float>(L.pre[l]);
    g.ldc = kFieldHid;
    g.bias = bias[l];
    g.D = batch.at<__nv_bfloat16>(L.h[l]);
    g.ldd = kFieldHid;
    g.DT = train ? batch.at<__nv_bfloat16>(L.inT[l + 1]) : nullptr;
    g.ldt = B;
    FIELD_TRY(launch_gemm_nt(g, kEpiBiasSilu, s));
  }
  GemmArgs g{};
  g.status = status.as<uint32_t>();
  g.A = batch.at<__nv_bfloat16>(L.h[3]);
  g.lda = g.K = kFieldHid;
  g.B = nt.W5b;
  g.ldb = kFieldHid;
  g.M = B;
  g.N = V;
  g.C = batch.at<float>(L.z);
  g.ldc = ldV;
  g.bias = nt.b5;
  FIELD_TRY(launch_gemm_nt(g, kEpiBias, s));
  if (!target) return cudaSuccess;
  FieldLoss fl{};
  fl.z = batch.at<float>(L.z);
  fl.target = target;
  fl.idx = batch.at<uint32_t>(L.idx);
  fl.x = batch.at<float>(L.x);
  fl.verts = rest_verts;
  fl.B = B;
  fl.V = V;
  fl.ldz = ldV;
  fl.lambda = lambda;
  fl.s2 = scale * scale;
  std::memcpy(fl.M, M.m, 64);
  fl.dzb = batch.at<__nv_bfloat16>(L.dzb);
  fl.dzT = batch.at<__nv_bfloat16>(L.dT[4]);
  fl.dz = batch.at<float>(L.dz);
  fl.loss = loss.as<float>();
  return launch_field_loss(fl, s);
}

cudaError_t FieldState::backward(uint32_t B, cudaStream_t s) {
  if (B % 8) return cudaErrorInvalidValue;  // transposed operands have row length B
  const BatchLayout L(B, V, ldV, true);
  __nv_bfloat16* w[4];
  transposed(w);
  // dL/dpre of layer l = (dL/dz or dL/dpre of the layer above) W silu'(pre_l)
  for (int l = 3; l >= 0; --l) {
    GemmArgs g{};
    g.status = status.as<uint32_t>();
    g.A = batch.at<__nv_bfloat16>(l == 3 ? L.dzb : L.dpreb[(l + 1) & 1]);
    g.lda = l == 3 ? ldV : kFieldHid;
    g.K = l == 3 ? V : kFieldHid;
    g.B = w[l];
    g.ldb = g.lda;
    g.M = B;
    g.N = kFieldHid;
    g.pre = batch.at<float>(L.pre[l]);
    g.C = batch.at<float>(L.dpre[l]);
    g.ldc = kFieldHid;
    g.D = l > 0 ? batch.at<__nv_bfloat16>(L.dpreb[l & 1]) : nullptr;
    g.ldd = kFieldHid;
    g.DT = batch.at<__nv_bfloat16>(L.dT[l]);
    g.ldt = B;
    FIELD_TRY(launch_gemm_nt(g, kEpiBack, s));
  }
  // dW_l = (dL/dpre_l or dL/dz)^T (input of the layer), db_l = their column sums
  GemmBatch gb{};
  gb.splits = grad_splits(B);
  for (int l = 0; l < 5; ++l) {
    GemmArgs& g = gb.g[l];
    g.status = status.as<uint32_t>();
    g.A = batch.at<__nv_bfloat16>(L.dT[l]);
    g.B = batch.at<__nv_bfloat16>(L.inT[l]);
    g.lda = g.ldb = g.K = B;
    g.M = l == 4 ? V : kFieldHid;
    g.N = l == 0 ? kFieldIn : kFieldHid;
    g.C = batch.at<float>(L.ws[l]);
    gb.first[l + 1] = gb.first[l] + (g.M + 127) / 128 * ((g.N + 63) / 64);
    gb.sum[l] = batch.at<float>(l == 4 ? L.dz : L.dpre[l]);
    gb.sum_n[l] = g.M;
    gb.sum_ld[l] = l == 4 ? ldV : kFieldHid;
    gb.sum_out[l] = g32.as<float>() + off[2 * l + 1];
  }
  return launch_gemm_grads(gb, s);
}

cudaError_t FieldState::update(uint32_t B, const float* lr, cudaStream_t s) {
  FieldUpdate u{};
  for (int k = 0; k <= kFieldParams; ++k) u.off[k] = off[k];
  u.V = V;
  u.ldV = ldV;
  u.splits = grad_splits(B);
  const BatchLayout L(B, V, ldV, true);
  for (int l = 0; l < 5; ++l) u.ws[l] = batch.at<float>(L.ws[l]);
  u.p = p32.as<float>();
  u.g = g32.as<float>();
  u.m = m1.as<float>();
  u.v = m2.as<float>();
  u.pb = pb.as<__nv_bfloat16>();
  transposed(u.wT);
  u.adam = lr ? 1 : 0;
  if (u.adam) {
    ++step;
    u.lr = *lr;
    u.b1 = 0.9f;
    u.b2 = 0.999f;
    u.eps = 1e-8f;
    u.c1 = (float)(1.0 / (1.0 - std::pow(0.9, (double)step)));
    u.c2 = (float)(1.0 / (1.0 - std::pow(0.999, (double)step)));
  }
  return launch_field_update(u, s);
}

cudaError_t FieldState::eval(uint32_t n, const float* points, float* w, cudaStream_t s) {
  const uint32_t chunk = 65536;
  for (uint32_t done = 0; done < n; done += chunk) {
    const uint32_t B = std::min(chunk, n - done);
    FIELD_TRY(forward(points + 3 * (size_t)done, nullptr, B, B, 0, nullptr, 0.0f, s));
    const BatchLayout L(B, V, ldV, false);
    FIELD_TRY(launch_field_weights(batch.at<float>(L.z), B, V, ldV, batch.at<float>(L.x), rest_d.as<float4>(), M,
                                   w + (size_t)done * V, s));
  }
  return cudaSuccess;
}

cudaError_t FieldState::project(const float4* verts, float* out, cudaStream_t s) const {
  return launch_field_project(net(), V, rest_d.as<float4>(), verts, M_d.as<float>(), out, s);
}

}  // namespace cgs
