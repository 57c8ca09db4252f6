// Decode step of a small fp32 model for up to 8 sequences (Llama.generate's per-token forward, llama3.py:285-321 with L == 1): all
// layers in ONE thread-block cluster of 16 CTAs, then the LM head with its argmax over the whole chip.
//
// A layer of such a model (stories15M: 4 MB of weights) is five short products that depend on one another.  Spread over all SMs
// (decode_mega.cu) each hand-over costs 3 - 4 us of L2 round trips, 17 us per layer; inside a cluster a phase's outputs go straight
// into every CTA's shared memory.  16 SMs draw their share of the weights - one contiguous range of rows per matrix and CTA - from L2 a
// phase or two ahead of its use: 249 KB per CTA and layer, 24 MB per step, which is not what bounds it (10 B/clk of an SM's 64).
//   phase 1  q, k, v rows (RMSNorm folded in, rotary turn) -> every CTA; k, v also to the caches
//   phase 2  attention, a (sequence, head) per CTA and turn -> every CTA
//   phase 3  Wo rows + residual    phase 4  gate, up rows, silu(g) u    phase 5  Wdown rows + residual, each -> every CTA
// Both sides measured: the rule in l3_api.cu (enqueue_decode_nodes).
#include <cooperative_groups.h>

#include <algorithm>

#include "cluster.h"
#include "common.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int CL = 16, TH = 512, NW = TH / 32;
static_assert(NW == CL, "warp w sends a phase's outputs to CTA w");
constexpr int KS = 4;  // most pieces of K a row's sum is split into

struct Lay {  // offsets in floats of one CTA's shared memory
  int a, b, x, att, qkv, res, red, out, out_n, tab, bar, total;
};
__host__ __device__ inline int up4(int v) { return (v + 3) & ~3; }
// N values (a multiple of 4) over the CTAs in whole fours
__host__ __device__ inline int rows_of(int N, int r) { return 4 * ((r + 1) * (N / 4) / CL - r * (N / 4) / CL); }
__host__ __device__ inline int first_of(int N, int r) { return 4 * (r * (N / 4) / CL); }
__host__ __device__ inline int most_rows(int N) { return 4 * ((N / 4 + CL - 1) / CL); }

// two copies spare a barrier per head; with 8 sequences stories15M would pass 227 KB by 1 KB
__host__ __device__ constexpr int red_copies(int nb) { return nb == 8 ? 1 : 2; }

__host__ __device__ inline Lay make_lay(int NL, int D, int HN, int KVHN, int HD, int FD, int nb) {
  const int qkv = (HN + 2 * KVHN) * HD;
  Lay l;
  l.a = 0;                                                          // norm weights | rows of Wqkv, then of w13
  l.b = l.a + D + std::max(most_rows(qkv), 2 * most_rows(FD)) * D;  // rows of Wo, then of Wdown
  l.x = l.b + most_rows(D) * std::max(D, FD);
  l.att = l.x + nb * D;
  l.qkv = l.att + nb * HN * HD;                                     // q | k | v; hidden values
  l.res = l.qkv + nb * std::max(qkv, FD);                           // own rows of x, two buffers
  l.red = l.res + up4(2 * nb * most_rows(D));                       // [warp][HD], then [warp] (max, sum)
  l.out = l.red + red_copies(nb) * (NW * HD + 2 * NW);
  l.out_n = up4(nb * std::max(std::max(most_rows(qkv), 2 * most_rows(FD)), KS * most_rows(D)));
  l.tab = l.out + 2 * l.out_n;                                      // the layers' pointers
  l.bar = l.tab + NL * (int)(sizeof(MegaLayer) / 4);
  l.total = l.bar + 16;
  return l;
}

__device__ __forceinline__ uint32_t s32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_arm(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// False: gave up.  The thread then waits no more, its CTA leaves the layers at the next barrier of all its threads, the others run out of
// data and do the same, and the host finds the error word.
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, bool ok) {
  uint32_t done = 0;
  for (uint32_t n = ok ? 1u << 22 : 1u; !done && n; --n)
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return ok && done;
}
__device__ __forceinline__ void bulk_load(float* dst, const float* src, int n, uint32_t bar) {  // 16-byte pieces on 16-byte boundaries
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(s32(dst)), "l"(src), "r"(n * 4), "r"(bar) : "memory");
}
// Four values into another CTA's shared memory; its barrier counts the bytes as they land
__device__ __forceinline__ void send4(uint32_t dst, float4 v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];"
               ::"r"(dst), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(bar) : "memory");
}

// The share of a warp: row groups g0, g0 + step, ... over values k0 .. k1 of K, to piece `piece` of the output
struct Part { int g0, step, k0, k1, piece; };
__device__ __forceinline__ Part part_of(int K, int ks) {
  const int warp = threadIdx.x >> 5, per = NW / ks, piece = warp % ks, nch = (K + 127) / 128;
  return {warp < per * ks ? warp / ks : 1 << 20, per, piece * nch / ks * 128, min(K, (piece + 1) * nch / ks * 128), piece};
}

// out[piece][b][row] = w[row] . xs[b] over the warp's piece of K, `rows` rows in shared memory, R rows of a warp at a time so that xs
// is read once for R of them.  NORM: xs[b] / rms(xs[b]) * nw in place of xs[b]; each warp sums the squares beside its products (one piece).
template <int NB, int R, bool NORM>
__device__ __forceinline__ void gemv(const float* w, int rows, int K, const Part& p, const float* xs, const float* nw, float eps, float* out) {
  const int lane = threadIdx.x & 31, k0 = p.k0, k1 = p.k1, piece = p.piece;
  for (int g = p.g0; g * R < rows; g += p.step) {
    float acc[R * NB], ss[NB];  // acc[b * R + r]
#pragma unroll
    for (int i = 0; i < R * NB; ++i) acc[i] = 0.f;
#pragma unroll
    for (int b = 0; b < NB; ++b) ss[b] = 0.f;
    const float* wr[R];
#pragma unroll
    for (int r = 0; r < R; ++r) wr[r] = w + min(g * R + r, rows - 1) * K + lane * 4;
    auto step = [&](int k, bool in) {
      const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
      float4 wv[R], n4 = zero;
#pragma unroll
      for (int r = 0; r < R; ++r) wv[r] = in ? *reinterpret_cast<const float4*>(wr[r] + k) : zero;
      if (NORM && in) n4 = *reinterpret_cast<const float4*>(nw + k + lane * 4);
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        float4 xv = in ? *reinterpret_cast<const float4*>(xs + b * K + k + lane * 4) : zero;
        if (NORM) {
          ss[b] = fmaf(xv.x, xv.x, ss[b]); ss[b] = fmaf(xv.y, xv.y, ss[b]); ss[b] = fmaf(xv.z, xv.z, ss[b]); ss[b] = fmaf(xv.w, xv.w, ss[b]);
          xv.x *= n4.x; xv.y *= n4.y; xv.z *= n4.z; xv.w *= n4.w;
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float& t = acc[b * R + r];
          t = fmaf(wv[r].x, xv.x, t); t = fmaf(wv[r].y, xv.y, t); t = fmaf(wv[r].z, xv.z, t); t = fmaf(wv[r].w, xv.w, t);
        }
      }
    };
    int k = k0;  // all lanes take the same way: a loop that some leave early would run its unrolled and its single form
#pragma unroll 2
    for (; k + 128 <= k1; k += 128) step(k, true);
    if (k < k1) step(k, k + lane * 4 < k1);
    __syncwarp();
    warp_sums<R * NB, 16>(acc, lane);
    float rinv = 1.f;
    if (NORM) {
      warp_sums<NB, 16>(ss, lane);  // lane b * (32 / NB) holds sequence b
      rinv = 1.0f / sqrtf(ss[0] / (float)K + eps);
    }
    constexpr int H = steps_of(R * NB), C = (R * NB) >> H, REST = 32 >> H;
    const int base = slot_base<R * NB>(lane);
#pragma unroll
    for (int i = 0; i < C; ++i) {
      const int b = (base + i) / R, row = g * R + (base + i) % R;
      float t = acc[i];
      if (NORM) t *= __shfl_sync(L3_FULL, rinv, b * (32 / NB));
      if ((lane & (REST - 1)) == 0 && row < rows) out[(piece * NB + b) * rows + row] = t;
    }
  }
}

// What bounds a step: five hand-overs a layer, each the latency of a short product, its sums over lanes and one crossing of the cluster.
// So every piece of it is about latency: weights arrive by bulk copies that one thread starts a phase or two ahead; this step's K and V
// rows of the cache are in registers before q is known; a phase's outputs are sent with the bytes counted at the receiver's barrier, in
// place of store, fence and cluster barrier (1300 cycles a phase for that alone, as measured with clock64).
// No buffer needs a second barrier: a CTA that holds all outputs of a phase knows that every CTA has ended that phase's reads, and what
// it writes next is only read behind the next hand-over.  `out`, the residual rows and `red` alternate between two copies, since a warp
// may still read one while the CTA's others are a phase ahead; the barrier of all warps in each phase bounds the distance to one.
template <int NB>
__global__ void __launch_bounds__(TH, 1) decode_cluster_kernel(const __grid_constant__ ClusterArgs a) {
  extern __shared__ __align__(16) float sm[];
  constexpr int U = NB <= 2 ? 8 : 4;  // keys of a thread in registers ahead of their use
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank(), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int D = a.D, HD = a.HD, FD = a.FD, B = a.B, qc = a.HN * HD, kc = a.KVHN * HD, QKV = qc + 2 * kc, rep = a.HN / a.KVHN;
  const Lay l = make_lay(a.NL, D, a.HN, a.KVHN, HD, FD, NB);
  float *sA = sm + l.a, *sB = sm + l.b, *x = sm + l.x, *att = sm + l.att, *qkv = sm + l.qkv;
  const int n1 = rows_of(QKV, rank), f1 = first_of(QKV, rank), n3 = rows_of(D, rank), f3 = first_of(D, rank), nh = rows_of(FD, rank), fh = first_of(FD, rank), n4 = 2 * nh;
  const uint32_t bar0 = s32(sm + l.bar), barA = bar0 + 40, barB = bar0 + 48;  // phase p: bar0 + 8 (p - 1)
  if (tid == 0) {
    for (int i = 0; i < 7; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8 * i));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  const uint32_t bytes[5] = {(uint32_t)(B * QKV * 4), (uint32_t)(B * qc * 4), (uint32_t)(B * D * 4), (uint32_t)(B * FD * 4), (uint32_t)(B * D * 4)};
  auto load = [&](uint32_t bar, float* dst, const float* nw, const void* w, int first, int n, int K) {  // thread 0
    bar_arm(bar, (uint32_t)((nw ? D : 0) + n * K) * 4);
    if (nw) { bulk_load(dst, nw, D, bar); dst += D; }
    bulk_load(dst, (const float*)w + (size_t)first * K, n * K, bar);
  };
  auto load1 = [&](const MegaLayer& ly) { load(barA, sA, ly.norm_in, ly.wqkv, f1, n1, D); };
  auto load3 = [&](const MegaLayer& ly) { load(barB, sB, nullptr, ly.wo, f3, n3, qc); };
  auto load4 = [&](const MegaLayer& ly) { load(barA, sA, ly.norm_post, ly.w13, 2 * fh, n4, D); };
  auto load5 = [&](const MegaLayer& ly) { load(barB, sB, nullptr, ly.w2, f3, n3, FD); };
  const MegaLayer* tab = reinterpret_cast<const MegaLayer*>(sm + l.tab);
  for (int i = tid; i < a.NL * (int)(sizeof(MegaLayer) / 4); i += TH) sm[l.tab + i] = reinterpret_cast<const float*>(a.layers)[i];
  if (tid == 0) {
    for (int p = 0; p < 5; ++p) bar_arm(bar0 + 8 * p, bytes[p]);
    load1(a.layers[0]);
    load3(a.layers[0]);
  }
  pdl_launch();
  pdl_wait();  // the weights above are constants; ids, positions and caches come from the step before
  const int pos = min(max(a.ids ? a.scal[0] : a.scal[2] + a.scal[1] + 1, 0), a.M - 1), T = pos + 1;
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    int id = 0;
    if (b < B) id = a.ids ? a.ids[(size_t)b * a.ids_ld + a.ids_off] : a.d_next[b];
    id = min(max(id, 0), a.vocab - 1);
    for (int i = tid; i < D; i += TH) {
      const float v = b < B ? a.embed[(size_t)id * D + i] : 0.f;
      x[b * D + i] = v;
      if (i >= f3 && i < f3 + n3) sm[l.res + b * n3 + i - f3] = v;
    }
    for (int i = tid; i < qc; i += TH) att[b * qc + i] = 0.f;  // slots without a sequence are never sent
  }
  for (int i = tid; i < NB * FD; i += TH) qkv[i] = 0.f;
  const float scale = 1.0f / sqrtf((float)HD);
  const int lpk = HD <= 64 ? 16 : 32, kpr = TH / lpk, sub = lane & (lpk - 1), key0 = tid / lpk;  // lanes per key, keys per row of threads
  const bool on = sub * 4 < HD;
  // Wo and Wdown: rows in fours and K in pieces so that all warps have work
  const int ks3 = max(1, min(min(KS, (qc + 127) / 128), NW / (n3 / 4))), ks5 = max(1, min(min(KS, (FD + 127) / 128), NW / (n3 / 4)));
  const Part pd = part_of(D, 1), p3 = part_of(qc, ks3), p5 = part_of(FD, ks5);
  // A phase's outputs are finished by ST threads per sequence - a value (or a pair of q, k, v) each, the rule sees to it - then sent.
  // What a thread needs for its pair in phase 1 stays the same in all layers.
  constexpr int ST = TH / NB;
  const int sb = tid / ST, st = tid % ST, col1 = f1 + 2 * st, kvc = col1 < qc + kc ? col1 - qc : col1 - qc - kc;
  const bool act1 = 2 * st < n1, turn = col1 < qc + kc, cached = act1 && col1 >= qc && sb < B;
  float rc = 1.f, rs = 0.f;
  if (act1 && turn) { const int j = (col1 < qc ? col1 : kvc) % HD / 2; rc = a.cos_tab[(size_t)pos * (HD / 2) + j]; rs = a.sin_tab[(size_t)pos * (HD / 2) + j]; }
  const size_t kv_at = cached ? (((size_t)sb * a.KVHN + kvc / HD) * a.M + pos) * HD + kvc % HD : 0;
  const int it_b = rank / a.HN, it_h = rank % a.HN;  // first (sequence, head) of phase 2
  float4 kf[U], vf[U];
  auto fetch = [&](const MegaLayer& ly, int b, int h, int j0) {
    if (b >= B) return;
    const size_t at = ((size_t)(b * a.KVHN + (rep == 1 ? h : h / rep)) * a.M + j0 + key0) * HD + sub * 4;
    const float *ck = (const float*)ly.ck + at, *cv = (const float*)ly.cv + at;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int j = j0 + u * kpr + key0;
      kf[u] = vf[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (on && j < pos) { kf[u] = __ldcg(reinterpret_cast<const float4*>(ck + u * kpr * HD)); vf[u] = __ldcg(reinterpret_cast<const float4*>(cv + u * kpr * HD)); }
    }
  };
  auto send_rows = [&](const float* o, int n, uint32_t to, int ld, int p) {  // o[b][n] -> to + b * ld, warp w to CTA w
    const uint32_t dst = cluster_at(to, warp), bar = cluster_at(bar0 + 8 * (p - 1), warp);
    const int sh = n <= 32 ? 3 : n <= 64 ? 4 : 5;  // lanes for a sequence's fours: 8, 16 or 32
    for (int b = lane >> sh; b < B; b += 32 >> sh)
      for (int i = 4 * (lane & ((1 << sh) - 1)); i < n; i += 4 << sh) send4(dst + (b * ld + i) * 4, *reinterpret_cast<const float4*>(o + b * n + i), bar);
    __syncwarp();
  };
  bool ok = true;
  int flip = 0;  // copy of `out`
  auto out = [&] { return sm + l.out + flip * l.out_n; };
  cl.sync();  // every CTA's barriers are set up before anything is sent
  for (int li = 0; li < a.NL; ++li) {
    const MegaLayer& ly = tab[li];
    const bool more = li + 1 < a.NL;
    const uint32_t par = li & 1;
    auto wait = [&](int p) {  // all outputs of phase p are here
      ok = bar_wait(bar0 + 8 * (p - 1), par, ok);
      if (tid == 0 && more && ok) bar_arm(bar0 + 8 * (p - 1), bytes[p - 1]);
    };
    auto refill = [&] { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); };  // all reads lie behind a barrier: before the next copy
    // ---- 1
    if (NB <= 2) fetch(ly, it_b, it_h, 0);
    ok = bar_wait(barA, 0, ok);
    if (n1 <= 4 * NW) gemv<NB, 4, true>(sA + D, n1, D, pd, x, sA, a.eps, out());
    else gemv<NB, 6, true>(sA + D, n1, D, pd, x, sA, a.eps, out());
    if (NB > 2) fetch(ly, it_b, it_h, 0);
    ok = __syncthreads_and(ok);
    if (!ok) break;
    {
      float* o = out();
      if (act1) {
        float2 v = *reinterpret_cast<float2*>(o + sb * n1 + 2 * st);
        if (turn) {
          v = make_float2(v.x * rc - v.y * rs, v.x * rs + v.y * rc);
          *reinterpret_cast<float2*>(o + sb * n1 + 2 * st) = v;
        }
        if (cached) *reinterpret_cast<float2*>((float*)(turn ? ly.ck : ly.cv) + kv_at) = v;
      }
      __syncthreads();
      send_rows(o, n1, s32(qkv + f1), QKV, 1);
      flip ^= 1;
    }
    if (tid == 0 && ok) { refill(); load4(ly); }
    wait(1);
    // ---- 2: keys of the cache from registers, this step's from the exchange.  Every warp keeps the running maximum of its own keys.
    {
      const uint32_t dst = cluster_at(s32(att), warp), bar = cluster_at(bar0 + 8, warp);
      int copy = 0, b = it_b, h = it_h;
      while (b < B) {
        const int g = rep == 1 ? h : h / rep;
        const float *knew = qkv + b * QKV + qc + g * HD, *vnew = knew + kc;
        const float4 qv = on ? *reinterpret_cast<const float4*>(qkv + b * QKV + h * HD + sub * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        float m = -INFINITY, sum = 0.f;
        float4 o4 = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int j0 = 0; j0 < T; j0 += U * kpr) {
          if (j0) fetch(ly, b, h, j0);
          float s[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (j0 + u * kpr + key0 == pos && on) { kf[u] = *reinterpret_cast<const float4*>(knew + sub * 4); vf[u] = *reinterpret_cast<const float4*>(vnew + sub * 4); }
            s[u] = qv.x * kf[u].x;
            s[u] = fmaf(qv.y, kf[u].y, s[u]); s[u] = fmaf(qv.z, kf[u].z, s[u]); s[u] = fmaf(qv.w, kf[u].w, s[u]);
          }
          __syncwarp();
          if (lpk == 32) {
#pragma unroll
            for (int u = 0; u < U; ++u) s[u] += __shfl_xor_sync(L3_FULL, s[u], 16);
          }
          warp_sums<U, 8>(s, lane);  // lanes: key mine of U, one or two lanes each in a group of 16
          const int mine = U == 8 ? (lane >> 1) & 7 : (lane >> 2) & 3;
          const bool in = j0 + mine * kpr + key0 < T;
          const float sc = in ? s[0] * scale : -INFINITY;
          float mt = fmaxf(m, sc);
#pragma unroll
          for (int o = 16; o > 8 / U; o >>= 1) mt = fmaxf(mt, __shfl_xor_sync(L3_FULL, mt, o));
          const float pr = in ? expf(sc - mt) : 0.f;
          if (j0) {
            const float corr = m == -INFINITY ? 0.f : expf(m - mt);
            sum *= corr; o4.x *= corr; o4.y *= corr; o4.z *= corr; o4.w *= corr;
          }
          m = mt;
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const float p = __shfl_sync(L3_FULL, pr, (lane & 16) | u * (16 / U));
            sum += p;
            o4.x = fmaf(p, vf[u].x, o4.x); o4.y = fmaf(p, vf[u].y, o4.y); o4.z = fmaf(p, vf[u].z, o4.z); o4.w = fmaf(p, vf[u].w, o4.w);
          }
        }
        const int b0 = b, h0 = h;
        for (h += CL; h >= a.HN; h -= a.HN) ++b;
        fetch(ly, b, h, 0);
        if (lpk == 16) {
          sum += __shfl_xor_sync(L3_FULL, sum, 16);
          o4.x += __shfl_xor_sync(L3_FULL, o4.x, 16); o4.y += __shfl_xor_sync(L3_FULL, o4.y, 16);
          o4.z += __shfl_xor_sync(L3_FULL, o4.z, 16); o4.w += __shfl_xor_sync(L3_FULL, o4.w, 16);
        }
        float *red = sm + l.red + copy * (NW * HD + 2 * NW), *ms = red + NW * HD;
        if (on && lane < lpk) *reinterpret_cast<float4*>(red + warp * HD + sub * 4) = o4;
        if (lane == 0) { ms[2 * warp] = m; ms[2 * warp + 1] = sum; }
        __syncthreads();
        // every warp weighs the warps' shares for itself and sends them to its CTA
        const float mw = ms[2 * (lane & (NW - 1))], lw = ms[2 * (lane & (NW - 1)) + 1];
        float mx = mw;
#pragma unroll
        for (int o = NW / 2; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(L3_FULL, mx, o));
        float wt = mw == -INFINITY ? 0.f : expf(mw - mx), tot = wt * lw;
#pragma unroll
        for (int o = NW / 2; o > 0; o >>= 1) tot += __shfl_xor_sync(L3_FULL, tot, o);
        wt /= tot;
        // half a warp takes half of the shares
        const int half = lane >> 4;
        for (int d0 = 0; d0 < HD; d0 += 64) {
          const int d = min(d0 + 4 * (lane & 15), HD - 4);
          float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int w = 0; w < NW / 2; ++w) {
            const float4 r4 = *reinterpret_cast<const float4*>(red + (2 * w + half) * HD + d);
            const float t = __shfl_sync(L3_FULL, wt, 2 * w + half);
            v.x = fmaf(t, r4.x, v.x); v.y = fmaf(t, r4.y, v.y); v.z = fmaf(t, r4.z, v.z); v.w = fmaf(t, r4.w, v.w);
          }
          v.x += __shfl_xor_sync(L3_FULL, v.x, 16); v.y += __shfl_xor_sync(L3_FULL, v.y, 16);
          v.z += __shfl_xor_sync(L3_FULL, v.z, 16); v.w += __shfl_xor_sync(L3_FULL, v.w, 16);
          if (!half && d0 + 4 * lane < HD) send4(dst + (b0 * qc + h0 * HD + d) * 4, v, bar);
          __syncwarp();
        }
        if (red_copies(NB) == 1) __syncthreads();
        else copy ^= 1;
      }
    }
    wait(2);
    // ---- 3 and 5: rows of the residual stream, x[own] + out -> every CTA
    auto add_rows = [&](int p, int ks) {
      const float *o = out(), *old = sm + l.res + (p == 5 ? NB * n3 : 0);
      float* now = sm + l.res + (p == 5 ? 0 : NB * n3);
      if (st < n3) {
        float v = o[sb * n3 + st];
        for (int s = 1; s < ks; ++s) v += o[(s * NB + sb) * n3 + st];
        now[sb * n3 + st] = v + old[sb * n3 + st];
      }
      __syncthreads();
      send_rows(now, n3, s32(x + f3), D, p);
      flip ^= 1;
    };
    ok = bar_wait(barB, 0, ok);
    gemv<NB, 4, false>(sB, n3, qc, p3, att, nullptr, 0.f, out());
    __syncthreads();
    add_rows(3, ks3);
    if (tid == 0 && ok) { refill(); load5(ly); }
    wait(3);
    // ---- 4
    ok = bar_wait(barA, 1, ok);
    if (n4 <= 4 * NW) gemv<NB, 4, true>(sA + D, n4, D, pd, x, sA, a.eps, out());
    else gemv<NB, 6, true>(sA + D, n4, D, pd, x, sA, a.eps, out());
    __syncthreads();
    {
      float* o = out();
      float v = 0.f;
      if (st < nh) { const float2 gu = *reinterpret_cast<const float2*>(o + sb * n4 + 2 * st); v = silu_ref(gu.x) * gu.y; }
      flip ^= 1;  // the other copy: no thread reads it any more
      o = out();
      if (st < nh) o[sb * nh + st] = v;
      __syncthreads();
      send_rows(o, nh, s32(qkv + fh), FD, 4);
      flip ^= 1;
    }
    if (tid == 0 && more && ok) { refill(); load1(tab[li + 1]); }
    wait(4);
    // ---- 5
    ok = bar_wait(barB, 1, ok);
    gemv<NB, 4, false>(sB, n3, FD, p5, qkv, nullptr, 0.f, out());
    __syncthreads();
    add_rows(5, ks5);
    if (tid == 0 && more && ok) { refill(); load3(tab[li + 1]); }
    wait(5);
  }
  for (int i = tid; i < n3 * B; i += TH) {
    const int b = i / n3, row = i % n3;
    a.x[(size_t)b * D + f3 + row] = x[b * D + f3 + row];
  }
  if (!ok) *a.err = 1;
  cl.sync();  // nobody leaves while something is on its way to it
  if (!ok) __nanosleep(1000000);  // what this CTA did not wait for lands before its shared memory is given up
}

// LM head: its argmax and the step's bookkeeping, or (LOGITS) the logits.  The layers ahead of it run on 16 SMs; on the others this kernel is
// resident meanwhile, one CTA each, and draws its rows of W into shared memory (stories15M: 192 of 243 rows, 29 of 37 MB; the rest is asked
// into L2).  Behind the wait there is the norm of x, a pass over shared memory and the merge of the maxima.  Four rows per warp and turn,
// eight lanes per row, four chains of sums per lane: of stories15M's 288 terms a chain has nine, as in the row-streaming GEMV (one chain of 36
// is 1.4 times as far from 64 bits).  stories15M, one sequence: from the layers' end to the step's 10.9 -> 8.3 us (a wait, three passes of few microseconds,
// two rounds of atomics), a forward step with its logits 125.5 -> 113.5 us.
constexpr int HT = 512, HW = HT / 32;
template <int NB, bool LOGITS>
__global__ void __launch_bounds__(HT, 1) cluster_head_kernel(ClusterHeadArgs a, int keep) {
  extern __shared__ __align__(16) float sh[];  // [keep][D] rows of W | [NB][D] normed x
  __shared__ unsigned long long s_best[HW][NB];
  __shared__ __align__(8) unsigned long long s_bar;
  __shared__ int s_last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, sub = lane & 7;
  float* xs = sh + (size_t)keep * a.D;
  const int r_lo = (int)((long long)a.VS * blockIdx.x / gridDim.x), r_hi = (int)((long long)a.VS * (blockIdx.x + 1) / gridDim.x);
  const int n_s = min(keep, r_hi - r_lo);
  const float* W = a.w + (size_t)r_lo * a.D;
  const uint32_t bar = s32(&s_bar);
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    bar_arm(bar, (uint32_t)(n_s * a.D * 4));
    const int piece = max(1, 4096 / a.D);  // rows per copy
    for (int r = 0; r < n_s; r += piece) bulk_load(sh + (size_t)r * a.D, W + (size_t)r * a.D, min(piece, n_s - r) * a.D, bar);
    for (int r = n_s; r < r_hi - r_lo; r += piece) l2_prefetch_bulk(W + (size_t)r * a.D, (uint32_t)(min(piece, r_hi - r_lo - r) * a.D * 4));
  }
  __syncthreads();
  pdl_launch();
  pdl_wait();  // W is constant; x comes from the kernel before
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const float* x = a.x + (size_t)min(b, a.B - 1) * a.D;
    float ss = 0.f;
    for (int i = lane * 4; i < a.D; i += 128) {
      const float4 v = *reinterpret_cast<const float4*>(x + i);
      ss = fmaf(v.x, v.x, ss); ss = fmaf(v.y, v.y, ss); ss = fmaf(v.z, v.z, ss); ss = fmaf(v.w, v.w, ss);
    }
    const float rinv = 1.0f / sqrtf(warp_sum(ss) / (float)a.D + a.eps);
    for (int i = tid; i < a.D; i += HT) xs[b * a.D + i] = x[i] * rinv * a.norm[i];
  }
  const bool ok = bar_wait(bar, 0, true);
  __syncthreads();
  unsigned long long best[NB];
#pragma unroll
  for (int b = 0; b < NB; ++b) best[b] = 0ull;
  auto four_rows = [&](const float* rows, int r0, int end, auto load) {  // rows r0 .. r0 + 3 of this CTA's, those below `end`
    const int r = r0 + (lane >> 3);
    const float* w = rows + (size_t)min(r, end - 1) * a.D;
    float2 lo[NB], hi[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) lo[b] = hi[b] = make_float2(0.f, 0.f);
    constexpr int AHEAD = NB <= 4 ? 9 : 3;  // of eight sequences nine do not fit the registers
#pragma unroll AHEAD
    for (int k = sub * 4; k < a.D; k += 32) {
      const float4 wv = load(w + k);
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const float4 xv = *reinterpret_cast<const float4*>(xs + b * a.D + k);
        lo[b] = fma2(make_float2(wv.x, wv.y), make_float2(xv.x, xv.y), lo[b]);
        hi[b] = fma2(make_float2(wv.z, wv.w), make_float2(xv.z, xv.w), hi[b]);
      }
    }
    __syncwarp();
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      float t = (lo[b].x + lo[b].y) + (hi[b].x + hi[b].y);
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(L3_FULL, t, o);
      if (LOGITS) {
        if (sub == 0 && r < end && b < a.B) a.logits[(size_t)b * a.VS + r_lo + r] = t;
      } else {
        const unsigned long long key = r < end && t == t ? argmax_key(t, r_lo + r) : 0ull;
        best[b] = key > best[b] ? key : best[b];
      }
    }
  };
  for (int r0 = n_s + warp * 4; r0 < r_hi - r_lo; r0 += HW * 4) four_rows(W, r0, r_hi - r_lo, [](const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); });
  for (int r0 = warp * 4; r0 < n_s; r0 += HW * 4) four_rows(sh, r0, n_s, [](const float* p) { return *reinterpret_cast<const float4*>(p); });
  if (!ok) {  // gave up: the host finds the error word; what is in flight lands before the shared memory is given up
    *a.err = 1;
    __nanosleep(1000000);
  }
  if constexpr (!LOGITS) {
#pragma unroll
    for (int b = 0; b < NB; ++b) {
#pragma unroll
      for (int o = 16; o >= 8; o >>= 1) {
        const unsigned long long k = __shfl_xor_sync(L3_FULL, best[b], o);
        best[b] = k > best[b] ? k : best[b];
      }
      if (lane == 0) s_best[warp][b] = best[b];
    }
    __syncthreads();
    if (tid < NB && tid < a.B) {
      unsigned long long k = 0ull;
      for (int w = 0; w < HW; ++w) k = s_best[w][tid] > k ? s_best[w][tid] : k;
      if (k) atomicMax(a.best + tid, k);
      __threadfence();
    }
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      s_last = atomicAdd(a.done, 1) == (int)gridDim.x - 1;
      __threadfence();
    }
    __syncthreads();
    if (!s_last) return;
    const int step = a.scal[1] + 1, pos = a.scal[2] + step;
    __syncthreads();
    if (tid < a.B) {
      const unsigned long long k = atomicExch(a.best + tid, 0ull);
      const int idx = k ? (int)(0xffffffffu - (uint32_t)(k & 0xffffffffull)) : 0;
      a.d_next[tid] = idx;
      a.d_tokens[(size_t)tid * a.M + step] = (int64_t)idx;
    }
    if (tid == 0) { a.scal[1] = step; a.scal[0] = pos; *a.done = 0; }
  }
}

int batch_slots(int B) { return B <= 1 ? 1 : B <= 2 ? 2 : B <= 4 ? 4 : 8; }

void fill_cfg(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, size_t smem, bool pdl, cudaStream_t s) {
  cfg = cudaLaunchConfig_t{};
  cfg.gridDim = dim3(CL);
  cfg.blockDim = dim3(TH);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CL; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl ? 2 : 1;
}

template <int NB>
cudaError_t prepare() {
  static bool done[16] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (done[dev & 15]) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(decode_cluster_kernel<NB>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(decode_cluster_kernel<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  done[dev & 15] = e == cudaSuccess;
  return e;
}

template <int NB>
cudaError_t launch_t(const ClusterArgs& a, cudaStream_t s) {
  const cudaError_t e = prepare<NB>();
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[2];
  fill_cfg(cfg, at, (size_t)make_lay(a.NL, a.D, a.HN, a.KVHN, a.HD, a.FD, NB).total * 4, a.pdl, s);
  return cudaLaunchKernelEx(&cfg, decode_cluster_kernel<NB>, a);
}

}  // namespace

int decode_cluster_max_batch(int NL, int D, int HN, int KVHN, int HD, int FD, int M) {
  // whole 16-byte pieces everywhere; a CTA's rows of a matrix fit its shared memory at once.  One CTA walks a head's keys, so only
  // short contexts: at 512 keys a head's caches (200 KB) take about as long as the rest of a layer
  if (D % 4 || FD % 4 || HD % 4 || HD > 128 || HN * HD != D || HN % KVHN || M > 512 || D / 4 < CL || FD / 4 < CL || KVHN * HD < 4 || NL > 64) return 0;
  int best = 0;
  for (int nb = 1; nb <= 8; nb *= 2)
    if ((size_t)make_lay(NL, D, HN, KVHN, HD, FD, nb).total * 4 <= 227 * 1024 && most_rows((HN + 2 * KVHN) * HD) / 2 <= TH / nb && most_rows(D) <= TH / nb &&
        most_rows(FD) <= TH / nb)
      best = nb;
  if (!best || prepare<1>() != cudaSuccess || prepare<2>() != cudaSuccess || prepare<4>() != cudaSuccess || prepare<8>() != cudaSuccess) { cudaGetLastError(); return 0; }
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[2];
  fill_cfg(cfg, at, (size_t)make_lay(NL, D, HN, KVHN, HD, FD, best).total * 4, false, nullptr);
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, decode_cluster_kernel<8>, &cfg) != cudaSuccess) { cudaGetLastError(); return 0; }
  return n > 0 ? best : 0;
}

cudaError_t launch_decode_cluster(const ClusterArgs& a, cudaStream_t s) {
  switch (batch_slots(a.B)) {
    case 1: return launch_t<1>(a, s);
    case 2: return launch_t<2>(a, s);
    case 4: return launch_t<4>(a, s);
    default: return launch_t<8>(a, s);
  }
}

template <int NB, bool LOGITS>
static cudaError_t launch_head_t(const ClusterHeadArgs& a, int n_sm, cudaStream_t s) {
  constexpr int ROOM = 220 * 1024;  // beside 16 x NB + 16 bytes of static shared memory
  static bool done[16] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!done[dev & 15]) {
    const cudaError_t e = cudaFuncSetAttribute(cluster_head_kernel<NB, LOGITS>, cudaFuncAttributeMaxDynamicSharedMemorySize, ROOM);
    if (e != cudaSuccess) return e;
    done[dev & 15] = true;
  }
  const int row = a.D * 4, grid = std::max(1, std::min(n_sm > 2 * CL ? n_sm - CL : n_sm, (a.VS + 3) / 4)), most = (a.VS + grid - 1) / grid;
  const int keep = std::min((most + 3) / 4 * 4, (ROOM - NB * row) / row / 4 * 4);
  return launch_k(cluster_head_kernel<NB, LOGITS>, dim3(grid), dim3(HT), (size_t)(keep + NB) * row, s, a, keep);
}

cudaError_t launch_cluster_head(const ClusterHeadArgs& a, int n_sm, cudaStream_t s) {
  const bool lg = a.logits != nullptr;
  switch (batch_slots(a.B)) {
    case 1: return lg ? launch_head_t<1, true>(a, n_sm, s) : launch_head_t<1, false>(a, n_sm, s);
    case 2: return lg ? launch_head_t<2, true>(a, n_sm, s) : launch_head_t<2, false>(a, n_sm, s);
    case 4: return lg ? launch_head_t<4, true>(a, n_sm, s) : launch_head_t<4, false>(a, n_sm, s);
    default: return lg ? launch_head_t<8, true>(a, n_sm, s) : launch_head_t<8, false>(a, n_sm, s);
  }
}
