// Second derivatives of the graph message in one pass per owner row (C = 32 or 64).
//
// The adjoint of (dx, dsh, dg) = A(x, sh, g; v) with cotangents hx, hs, hg of all three is the gradient of
//   <v, F(hx, sh, g) + F(x, hs, g) + F(x, sh, hg)>,
// three adjoint launches (sender rows), three forward launches (receiver rows) and the additions between them, most of all
// those of the [E, P C] gate gradients.  Here a sender pass builds both geometries of an edge, b(sh) and b(hs), reads the
// cotangent row once and forms
//   z_i = sum_k b(sh)_ik v_k,  y_i = sum_k b(hs)_ik v_k            per path p
//   gx_i += y_i g_p + z_i hg_p       gg_p = sum_i hx_i z_i + x_i y_i       gsh from (x_i hg_p + hx_i g_p) v_k,
// and a receiver pass gv_k += hg_p sum_i x_i b(sh)_ik + g_p sum_i (hx_i b(sh)_ik + x_i b(hs)_ik).
// Gate rows g and hg come through the same ring of bulk copies as in tp_tma_kernels.cuh, two rows a slot.  Both
// sets of features and geometries are live, which takes about 200 registers: eight warps per SM instead of twelve.
// Training step of 32,768 atoms (1.05 M edges, both interactions): 56.2 -> 51.4 ms.
#pragma once
#include "tp_tma_kernels.cuh"

namespace ictc {

constexpr int kSecondStages = 3, kSecondWarps = 8;

template <class S, class F, int CPL> struct SecondLayout {
  static constexpr int C = 32 * CPL;
  static constexpr int R = (F::NB + 31) / 32, NBP = R * 32;
  static constexpr unsigned GATE_BYTES = S::NP * C * 4, SLOT_BYTES = 2 * GATE_BYTES;
  static constexpr unsigned BAR_OFF = kSecondStages * SLOT_BYTES;
  static constexpr unsigned GEO_OFF = BAR_OFF + ((kSecondStages * 8 + 15) / 16) * 16;
  static constexpr unsigned RED_OFF = GEO_OFF + 4 * NBP * sizeof(Vec<CPL>);      // two edges, two geometries
  static constexpr int RED_PITCH = 36;
  static constexpr unsigned BYTES = ((RED_OFF + S::NH * RED_PITCH * 4 + 127) / 128) * 128;
};

// The ring of gate rows of one warp: slot s holds g and hg of an edge.
template <class S, class L> struct SecondRing {
  unsigned char* mine;
  unsigned bars;
  int slot = 0;
  unsigned parity = 0;

  __device__ SecondRing(unsigned char* smem, int lane) : mine(smem), bars(smem_addr(smem + L::BAR_OFF)) {
    if (lane == 0) {
#pragma unroll
      for (int s = 0; s < kSecondStages; ++s) mbar_init(bars + s * 8, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
  }
  __device__ void issue(int s, const TpArgs& a, const TpTangents& t, int e, int lane) {
    if (lane) return;
    const unsigned bar = bars + s * 8;
    mbar_expect_tx(bar, L::SLOT_BYTES);
    bulk_g2s(smem_addr(mine + s * L::SLOT_BYTES), a.g + int64_t(e) * (S::NP * L::C), L::GATE_BYTES, bar);
    bulk_g2s(smem_addr(mine + s * L::SLOT_BYTES + L::GATE_BYTES), t.hg + int64_t(e) * (S::NP * L::C), L::GATE_BYTES, bar);
  }
  // false: the time limit ran out; the copies that are still in flight have been waited for
  __device__ bool wait(int64_t it, int64_t end) {
    if (mbar_wait(bars + slot * 8, parity)) return true;
    for (int s = 0; s < kSecondStages; ++s) {
      const bool refilled = s < slot;
      if (it - slot + s + (refilled ? kSecondStages : 0) < end) mbar_wait(bars + s * 8, refilled ? parity ^ 1u : parity);
    }
    return false;
  }
  __device__ void advance() {
    if (++slot == kSecondStages) {
      slot = 0;
      parity ^= 1;
    }
  }
};

template <class S, class F, int CPL>
__global__ void __launch_bounds__(32, kSecondWarps) tp_second_adjoint_kernel(TpArgs a, TpTangents t) {
  using V = Vec<CPL>;
  using L = SecondLayout<S, F, CPL>;
  constexpr int C = L::C;
  extern __shared__ __align__(128) unsigned char tma_smem[];
  const int lane = threadIdx.x;
  const int64_t owner = blockIdx.x;
  SecondRing<S, L> ring(tma_smem, lane);
  V* geo = reinterpret_cast<V*>(tma_smem + L::GEO_OFF);
  float* red = reinterpret_cast<float*>(tma_smem + L::RED_OFF);
  BTerm bt[L::R];
#pragma unroll
  for (int r = 0; r < L::R; ++r) bt[r] = (r * 32 + lane < F::NB) ? F::ap(r * 32 + lane) : BTerm{0, 0.f, 0, 0.f};
  V x[S::NX], hx[S::NX], dx[S::NX];
#pragma unroll
  for (int i = 0; i < S::NX; ++i) {
    const int64_t at = owner * (S::NX * C) + lane * CPL + i * C;
    x[i] = V::load(a.x + at);
    hx[i] = V::load(t.hx + at);
    dx[i] = V::dup(0.f);
  }
  const int64_t begin = ldg(a.rowptr + owner), end = ldg(a.rowptr + owner + 1);
  auto edge_at = [&](int64_t it) -> int { return int(a.order ? ldg(a.order + it) : it); };
#pragma unroll
  for (int k = 0; k < kSecondStages; ++k)
    if (begin + k < end) ring.issue(k, a, t, edge_at(begin + k), lane);
  int e_cur = begin < end ? edge_at(begin) : 0;
  int r_cur = begin < end ? int(ldg(a.nbr + e_cur)) : 0;
  float shv = 0.f, hsv = 0.f;
  if (begin < end && lane < S::NH) {
    shv = ldg(a.sh + int64_t(e_cur) * S::NH + lane);
    hsv = ldg(t.hs + int64_t(e_cur) * S::NH + lane);
  }
  int buf = 0;
  for (int64_t it = begin; it < end; ++it, buf ^= 1) {
    const int e = e_cur;
    const float sh_now = shv, hs_now = hsv;
    const float* vp = a.v + int64_t(r_cur) * (S::NO * C) + lane * CPL;
    const int e_fill = it + kSecondStages < end ? edge_at(it + kSecondStages) : 0;
    if (it + 1 < end) {
      e_cur = edge_at(it + 1);
      r_cur = int(ldg(a.nbr + e_cur));
      if (lane < S::NH) {
        shv = ldg(a.sh + int64_t(e_cur) * S::NH + lane);
        hsv = ldg(t.hs + int64_t(e_cur) * S::NH + lane);
      }
    }
    V *sb = geo + 2 * buf * L::NBP, *sbh = sb + L::NBP;
    build_geometry<F::NB, CPL, L::R>(bt, sh_now, lane, sb);
    build_geometry<F::NB, CPL, L::R>(bt, hs_now, lane, sbh);
    if (!ring.wait(it, end)) {
      if (lane == 0 && a.status) atomicExch(a.status, 3);
      return;
    }
    const unsigned char* base = tma_smem + ring.slot * L::SLOT_BYTES + lane * (CPL * 4);
    const bool scaled = a.mask || a.w;
    const V mu = V::dup(a.mask ? ldg(a.mask + e) : 1.f);
    auto scale = [&](int p, V g) -> V {
      if (!scaled) return g;
      return vmul(g, a.w ? vmul(mu, V::load(a.w + p * C + lane * CPL)) : mu);
    };
    float* ggp = a.dg + int64_t(e) * (S::NP * C) + lane * CPL;
    __syncwarp();   // both geometries visible to every lane
    V dsh[S::NH];
#pragma unroll
    for (int j = 0; j < S::NH; ++j) dsh[j] = V::dup(0.f);
    F::second_fused(
        x, hx, [&](int k) -> V { return V::load(vp + k * C); },
        [&](int p) -> V { return scale(p, lds_vec<CPL>(base + p * (C * 4))); },
        [&](int p) -> V { return scale(p, lds_vec<CPL>(base + L::GATE_BYTES + p * (C * 4))); }, sb, sbh, dx, dsh,
        [&](int p, V val) { scale(p, val).store(ggp + p * C); });
    // harmonics' gradient: lane r adds up component r over the lanes' partial sums
#pragma unroll
    for (int j = 0; j < S::NH; ++j) red[j * L::RED_PITCH + lane] = dsh[j].hsum();
    __syncwarp();   // every lane is done with the slot and the geometry; the partial sums are visible
    if (it + kSecondStages < end) ring.issue(ring.slot, a, t, e_fill, lane);
    if (lane < S::NH) {
      const float4* row = reinterpret_cast<const float4*>(red + lane * L::RED_PITCH);
      float tot = 0.f;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float4 part = row[q];
        tot += (part.x + part.y) + (part.z + part.w);
      }
      a.dsh[int64_t(e) * S::NH + lane] = tot;
    }
    __syncwarp();   // the partial sums may be overwritten
    ring.advance();
  }
#pragma unroll
  for (int i = 0; i < S::NX; ++i) dx[i].store(a.dx + owner * (S::NX * C) + lane * CPL + i * C);
}

template <class S, class F, int CPL>
__global__ void __launch_bounds__(32, kSecondWarps) tp_second_forward_kernel(TpArgs a, TpTangents t) {
  using V = Vec<CPL>;
  using L = SecondLayout<S, F, CPL>;
  constexpr int C = L::C;
  extern __shared__ __align__(128) unsigned char tma_smem[];
  const int lane = threadIdx.x;
  const int64_t n = blockIdx.x;
  SecondRing<S, L> ring(tma_smem, lane);
  V* geo = reinterpret_cast<V*>(tma_smem + L::GEO_OFF);
  BTerm bt[L::R];
#pragma unroll
  for (int r = 0; r < L::R; ++r) bt[r] = (r * 32 + lane < F::NB) ? F::fb(r * 32 + lane) : BTerm{0, 0.f, 0, 0.f};
  V acc[S::NO];
#pragma unroll
  for (int k = 0; k < S::NO; ++k) acc[k] = V::dup(0.f);
  const int64_t begin = ldg(a.rowptr + n), end = ldg(a.rowptr + n + 1);
  auto edge_at = [&](int64_t it) -> int { return int(a.order ? ldg(a.order + it) : it); };
#pragma unroll
  for (int k = 0; k < kSecondStages; ++k)
    if (begin + k < end) ring.issue(k, a, t, edge_at(begin + k), lane);
  int e_cur = begin < end ? edge_at(begin) : 0;
  int r_cur = begin < end ? int(ldg(a.nbr + e_cur)) : 0;
  float shv = 0.f, hsv = 0.f;
  if (begin < end && lane < S::NH) {
    shv = ldg(a.sh + int64_t(e_cur) * S::NH + lane);
    hsv = ldg(t.hs + int64_t(e_cur) * S::NH + lane);
  }
  int buf = 0;
  for (int64_t it = begin; it < end; ++it, buf ^= 1) {
    const int e = e_cur;
    const float sh_now = shv, hs_now = hsv;
    V x[S::NX], hx[S::NX], ge[S::NP], hge[S::NP];
#pragma unroll
    for (int i = 0; i < S::NX; ++i) {
      const int64_t at = int64_t(r_cur) * (S::NX * C) + lane * CPL + i * C;
      x[i] = V::load(a.x + at);
      hx[i] = V::load(t.hx + at);
    }
    const int e_fill = it + kSecondStages < end ? edge_at(it + kSecondStages) : 0;
    if (it + 1 < end) {
      e_cur = edge_at(it + 1);
      r_cur = int(ldg(a.nbr + e_cur));
      if (lane < S::NH) {
        shv = ldg(a.sh + int64_t(e_cur) * S::NH + lane);
        hsv = ldg(t.hs + int64_t(e_cur) * S::NH + lane);
      }
    }
    V *sb = geo + 2 * buf * L::NBP, *sbh = sb + L::NBP;
    build_geometry<F::NB, CPL, L::R>(bt, sh_now, lane, sb);
    build_geometry<F::NB, CPL, L::R>(bt, hs_now, lane, sbh);
    if (!ring.wait(it, end)) {
      if (lane == 0 && a.status) atomicExch(a.status, 4);
      return;
    }
    const unsigned char* base = tma_smem + ring.slot * L::SLOT_BYTES + lane * (CPL * 4);
#pragma unroll
    for (int p = 0; p < S::NP; ++p) {
      ge[p] = lds_vec<CPL>(base + p * (C * 4));
      hge[p] = lds_vec<CPL>(base + L::GATE_BYTES + p * (C * 4));
    }
    if (a.mask || a.w) {
      const V mu = V::dup(a.mask ? ldg(a.mask + e) : 1.f);
#pragma unroll
      for (int p = 0; p < S::NP; ++p) {
        const V s = a.w ? vmul(mu, V::load(a.w + p * C + lane * CPL)) : mu;
        ge[p] = vmul(ge[p], s);
        hge[p] = vmul(hge[p], s);
      }
    }
    __syncwarp();   // geometries visible; the compiler may still read the slot below
    F::second_forward(x, hx, ge, hge, sb, sbh, acc);
    __syncwarp();   // every lane is done with the slot
    if (it + kSecondStages < end) ring.issue(ring.slot, a, t, e_fill, lane);
    ring.advance();
  }
  float* op = a.out + n * (S::NO * C) + lane * CPL;
#pragma unroll
  for (int k = 0; k < S::NO; ++k) acc[k].store(op + k * C);
}

template <class S, class F, int CPL> int launch_second(const TpArgs& a, const TpTangents& t, bool forward, cudaStream_t st) {
  using L = SecondLayout<S, F, CPL>;
  if (forward) {
    auto kernel = tp_second_forward_kernel<S, F, CPL>;
    static const int attr = set_smem(kernel, L::BYTES);
    if (attr != ICTC_OK) return attr;
    kernel<<<(unsigned)a.N, 32, L::BYTES, st>>>(a, t);
    return finish_launch("tp_second_forward");
  }
  auto kernel = tp_second_adjoint_kernel<S, F, CPL>;
  static const int attr = set_smem(kernel, L::BYTES);
  if (attr != ICTC_OK) return attr;
  kernel<<<(unsigned)a.N, 32, L::BYTES, st>>>(a, t);
  return finish_launch("tp_second_adjoint");
}

template <class S, int ID> int second_dispatch(const TpArgs& a, const TpTangents& t, bool forward, cudaStream_t st) {
  if (a.C == 64) return launch_second<S, TpFast<ID, 2>, 2>(a, t, forward, st);
  return launch_second<S, TpFast<ID, 1>, 1>(a, t, forward, st);
}

template <class S, int ID> TpOps make_ops_tma() {
  return TpOps{S::NX, S::NH, S::NP, S::NO, S::NNZ, &launch_edge_forward<S>, &graph_forward_dispatch_tma<S, ID>,
               &adjoint_dispatch_tma<S, ID>, &second_dispatch<S, ID>};
}

}  // namespace ictc
