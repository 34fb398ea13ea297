// Paged key-value cache: append of new keys/values and batch decode attention over the pages.
//
// The cache is the reference's: a pool of pages, each one tensor [layers, 2, kv_heads, page_size,
// head_dim] (kernel_src/src/loquetier/utils/kvcache.py:40-60; flashinfer's paged_kv_t with pointer
// storage, kernel_src/third_party/flashinfer/include/flashinfer/page.cuh:45-64), reached through a
// device array of page addresses, a page index pointer per request and the number of valid entries
// of each request's last page.  Keys are stored as projected - NOT rotated; the rotary position
// embedding is applied when they are read (decode.cuh:108-111), to the query at position
// seq_len - 1 (:489-494).
//
//   append_kv_kernel   one new token per request   (AppendPagedKVCacheDecodeKernel, page.cuh:368-396)
//                      or a run of tokens per request (AppendPagedKVCachePrefillKernel, page.cuh:411-444)
//   paged_decode_kernel  o = softmax(rope(q) . rope(K)^T / sqrt(d)) . V per request and head
//                        (BatchDecodeWithPagedKVCacheKernel, decode.cuh:451-620)
//
// Decode is HBM-bound: every K and V entry of a (request, kv head) is read exactly once, whatever the
// number of query heads that share the kv head - they are the columns of one tensor-core tile.  Long
// sequences of small batches are cut into up to `splits` ranges of key tiles so that the machine is filled; the
// partial softmax states go through a workspace and the CTA that finishes last (a ticket, no waiting)
// merges them in range order - a fixed order, so the result does not depend on scheduling.  In batches of long
// requests that need no ranges the longest go first, so that the launch ends on its shortest CTAs.
#pragma once
#include "smlm_common.cuh"

namespace smlm {

constexpr int kPdDim = 128;          // head dimension served
constexpr int kPdStages = 2;         // tiles of 16 keys in flight per warp
constexpr int kPdMaxSplits = 16;
constexpr int kPdRec = kPdDim + 4;   // floats of a parked softmax state: m, d, two unused, then o[128] (16-byte aligned)

struct PdArgs {
  void* o;                        // [B, Nq, 128]
  const void* q;                  // [B, Nq, 128]
  const void* const* kv_ptrs;     // page addresses
  const int32_t* kv_indptr;       // [B + 1]
  const int32_t* last_page_offset;  // [B]
  int* err;                       // error word (bits of smlm_common.cuh), may be null
  int* tickets;                   // [B * Nkv], zero between launches
  float* partial;                 // [B * Nq * splits * kPdRec]
  int batch, num_kv_heads, num_layers, layer_idx, page_size, splits, total_pages;
  int sort_pages;                 // pages in use from which on the longest requests may go first; negative: never
  float log2_theta;               // log2(rope base)
};

struct AppendArgs {
  const void* const* kv_ptrs;
  const int32_t* kv_indptr;
  const int32_t* last_page_offset;
  const void* k;                  // [tokens, Nkv, 128]
  const void* v;
  const int32_t* append_indptr;   // [B + 1] for init_kv; null for append_kv (one token per request)
  int* err;
  int batch, num_kv_heads, num_layers, layer_idx, page_size, total_pages;
};

// ---------------------------------------------------------------------------------------------
// append
// ---------------------------------------------------------------------------------------------

// grid: (B * Nkv, token chunks); 16 threads move one 256-byte row each, 8 rows per step
template <typename T>
__global__ void __launch_bounds__(128) append_kv_kernel(const AppendArgs a) {
  const int b = blockIdx.x / a.num_kv_heads;
  const int h = blockIdx.x - b * a.num_kv_heads;
  const int tx = threadIdx.x & 15, row = threadIdx.x >> 4;
  pdl_wait();
  const int p0 = a.kv_indptr[b], p1 = a.kv_indptr[b + 1];
  const int npg = p1 - p0;
  if (npg <= 0 || p0 < 0 || p1 > a.total_pages) {
    if (npg != 0 && threadIdx.x == 0 && a.err != nullptr) atomicOr(a.err, kErrBadIndptr);
    return;
  }
  const int P = a.page_size;
  const int seq_len = (npg - 1) * P + a.last_page_offset[b];
  int src0, n;
  if (a.append_indptr == nullptr) {
    src0 = b;
    n = 1;
  } else {
    src0 = a.append_indptr[b];
    n = a.append_indptr[b + 1] - src0;
  }
  if (n <= 0) return;
  if (n > seq_len) {  // more new tokens than the pages hold
    if (threadIdx.x == 0 && a.err != nullptr) atomicOr(a.err, kErrBadIndptr);
    return;
  }
  const int start = seq_len - n;
  const T* K = static_cast<const T*>(a.k);
  const T* V = static_cast<const T*>(a.v);
  const size_t kv_delta = static_cast<size_t>(a.num_kv_heads) * P * kPdDim;
  // four tokens per thread and step: their page addresses and source rows are fetched together, so that a
  // step costs one round of memory latency instead of four
  constexpr int U = 4;
  const int stride = gridDim.y * 8;
  for (int j0 = blockIdx.y * 8 + row; j0 < n; j0 += U * stride) {
    T* kd[U];
    uint4 kk[U], vv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int j = j0 + u * stride;
      kd[u] = nullptr;
      kk[u] = vv[u] = make_uint4(0u, 0u, 0u, 0u);
      if (j < n) {
        const int pos = start + j;
        T* page = static_cast<T*>(const_cast<void*>(a.kv_ptrs[p0 + pos / P]));
        if (page == nullptr || (reinterpret_cast<uintptr_t>(page) & 15) != 0) {
          if (tx == 0 && a.err != nullptr) atomicOr(a.err, kErrBadPointer);
        } else {
          kd[u] = page + ((static_cast<size_t>(a.layer_idx) * 2 * a.num_kv_heads + h) * P + pos % P) * kPdDim + tx * 8;
        }
        const size_t so = (static_cast<size_t>(src0 + j) * a.num_kv_heads + h) * kPdDim + tx * 8;
        kk[u] = __ldg(reinterpret_cast<const uint4*>(K + so));
        vv[u] = __ldg(reinterpret_cast<const uint4*>(V + so));
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (kd[u] != nullptr) {
        *reinterpret_cast<uint4*>(kd[u]) = kk[u];
        *reinterpret_cast<uint4*>(kd[u] + kv_delta) = vv[u];
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------
// decode
// ---------------------------------------------------------------------------------------------

constexpr int kPdWarps = 4;                          // each warp streams its own tiles of 16 keys
constexpr int kPdTile = 16;
constexpr int kPdTileBytes = kPdTile * kPdDim * 2;   // one tile of K (or V) of one head: 4 KB
constexpr int kPdWarpRing = kPdStages * 2 * kPdTileBytes;
constexpr int kPdQOff = kPdWarps * kPdWarpRing;      // rotated queries [8 rows][128]
constexpr int kPdRotOff = kPdQOff + 8 * kPdDim * 2;  // frequency pairs: step of a warp, step of 8 keys, frequencies
constexpr int kPdSmem = kPdRotOff + 2 * 512 + 256;
constexpr int kPdStep = kPdWarps * kPdTile;          // keys between two tiles of a warp
constexpr int kPdMaxSorted = 192;                    // requests whose ranks a CTA finds for itself
constexpr int kPdReseed = 16;                        // tiles after which the rotation is computed afresh

// 8 x 8 transpose of 16-bit elements over a warp
__device__ __forceinline__ uint32_t movm_t(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(r) : "r"(v));
  return r;
}
// (c, s) of an angle turned by (c1, s1), two angles at once
__device__ __forceinline__ void turn_f32x2(uint64_t& c, uint64_t& s, uint64_t c1, uint64_t s1) {
  const uint64_t n = fma_f32x2(c, c1, mul_f32x2(s ^ 0x8000000080000000ull, s1));
  s = fma_f32x2(s, c1, mul_f32x2(c, s1));
  c = n;
}

// One CTA = one (request, kv head, range of key tiles).  The keys of a tile are the rows of the MMA and the
// G query heads that share the kv head its columns, so every key and value is read once for all of them and no
// row is padding:
//   S^T[16 keys, 8 heads] = K . Q^T  and  O^T[128, 8 heads] += V^T . P^T  with mma.sync m16n8k16, fp32 accumulation.
// Each warp owns every fourth tile of the range and a private ring of shared-memory stages filled with
// 16-byte cp.async copies (no CTA-wide barrier in the loop).
//
// The keys are rotated in registers between ldmatrix and the MMA: a lane's fragments hold, for keys g and g + 8
// of the tile, a dimension and (four k steps later) its partner 64 dimensions on.  A lane keeps the cosines and
// sines of key g for its 16 frequencies, turns them by 8 keys for the other key and by the warp's step for its next
// tile, and computes them afresh every 16 tiles (16 turns: the error of one).  The rotated keys are rounded to
// the storage type - what a cache that stores rotated keys holds anyway.
//
// What bounds it: with the keys' rows rotated in place in shared memory (two loads and two stores per key and
// lane) and the heads as the rows of a half-empty tile, a tile of 16 keys took a warp about 960 instructions and
// the 12 warps of an SM could not issue them as fast as the keys arrive; this form takes about 660.  The maxima are
// exchanged (six shuffles) and the sums rescaled only in tiles that raise one, which a vote finds out.  They are raised by
// any excess: the weights are rounded to 16 bits, and the key that sets the maximum has the weight one exactly.  Raising
// them late, at an excess of 2^8, made the results' error against 64 bits 2.4 % larger (geometric mean, up to 7.5 %).
// Measured, append + decode of 128 requests with contexts 512..4096 drawn evenly, 32 / 8 heads (1236 MB), longest first:
// 287 us before, 217 us now (5.7 TB/s) as one call among others on new inputs; 199-210 us replayed from a graph.
template <typename T, int G>
__global__ void __launch_bounds__(kPdWarps * 32, 3) paged_decode_kernel(const PdArgs a) {
  extern __shared__ __align__(128) unsigned char pd_smem[];
  __shared__ int s_last;
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;       // MMA fragment coordinates: row g, column pair t

  const int S = a.splits;
  const int s = blockIdx.x % S;
  const int kvh = blockIdx.x / S % a.num_kv_heads;
  int b = blockIdx.x / S / a.num_kv_heads;
  const int Nq = a.num_kv_heads * G;
  const int P = a.page_size;
  const int head0 = kvh * G;

  pdl_wait();
  if (a.sort_pages >= 0) {
    // the request whose number of pages has rank b: every CTA counts for itself (whatever the table holds, the
    // ranks are a permutation of the requests)
    int* len = reinterpret_cast<int*>(pd_smem);
    const int n4 = (a.batch + 3) & ~3;
    // what the requests hold counts; the table may be longer (a captured step keeps its arguments)
    const int used = max(0, min(a.kv_indptr[a.batch] - a.kv_indptr[0], a.total_pages));
    int uneven = 0;   // long requests, and one of them holds more than 5/4 of the mean
    for (int i = tid; i < n4; i += kPdWarps * 32) {
      const int n = i < a.batch ? a.kv_indptr[i + 1] - a.kv_indptr[i] : INT32_MIN;
      len[i] = n;
      uneven |= used >= a.sort_pages && 4LL * n * a.batch > 5LL * used;
    }
    if (__syncthreads_or(uneven)) {
      for (int i = tid; i < a.batch; i += kPdWarps * 32) {
        const int mine = len[i];
        int rank = 0;
        for (int k = 0; k < n4; k += 4) {   // (entries past the batch are never ahead: smallest, and behind)
          const int4 v = *reinterpret_cast<const int4*>(len + k);
          rank += (v.x > mine || (v.x == mine && k < i)) + (v.y > mine || (v.y == mine && k + 1 < i)) +
                  (v.z > mine || (v.z == mine && k + 2 < i)) + (v.w > mine || (v.w == mine && k + 3 < i));
        }
        if (rank == b) s_last = i;
      }
      __syncthreads();
      b = s_last;
    }
    __syncthreads();   // the ranks' space is the ring's, s_last serves the ranges later
  }
  const int bh = b * a.num_kv_heads + kvh;
  int p0 = a.kv_indptr[b], p1 = a.kv_indptr[b + 1];
  if (p0 < 0 || p1 < p0 || p1 > a.total_pages) {
    if (tid == 0 && a.err != nullptr) atomicOr(a.err, kErrBadIndptr);
    p1 = p0 = 0;
  }
  const int npages = p1 - p0;
  int last_valid = npages > 0 ? a.last_page_offset[b] : 0;
  if (last_valid < 0 || last_valid > P) {
    if (tid == 0 && a.err != nullptr) atomicOr(a.err, kErrBadIndptr);
    last_valid = 0;
  }
  const int seq_len = npages > 0 ? (npages - 1) * P + last_valid : 0;
  const int ntiles = (seq_len + kPdTile - 1) / kPdTile;
  // The ranges follow from the request's own length, whatever else the batch or its page table holds.  Longer ranges for
  // the shorter requests of an uneven batch (a share of the machine each) were up to 17 % faster (20 requests of 100..4000
  // keys and 4 kv heads, 24 against 29 us) but rounded more weights: every warp's largest is exact, and with fewer ranges
  // there are fewer of them (error against 64 bits up to 1 % larger).
  const int per = max((ntiles + S - 1) / S, kPdWarps);        // a tile per warp at least
  const int ranges = max(1, (ntiles + per - 1) / per);        // ranges this request is cut into
  if (s >= ranges) return;
  const int tile0 = s * per;
  const int ntl = max(0, min(ntiles, tile0 + per) - tile0);   // tiles of this CTA
  const int ntw = ntl > warp ? (ntl - warp + kPdWarps - 1) / kPdWarps : 0;   // tiles of this warp

  // ---- the rotated, pre-scaled queries, the B operand: [8 rows][128] in shared memory ----
  // Angles are kept in half-turns (angle / pi): sincospif reduces its argument exactly, whereas the
  // library is built with fast math, under which sincosf loses accuracy at the angles long sequences reach.
  const uint32_t sbase = smem_u32(pd_smem);
  const uint32_t qs = sbase + kPdQOff;
  {
    const int row = tid >> 4;                 // 8 rows x 16 threads
    const int d0 = (tid & 15) * 4;            // dims d0..d0+3 and their partners d0+64..
    float own[4] = {0.f, 0.f, 0.f, 0.f}, par[4] = {0.f, 0.f, 0.f, 0.f};
    if (row < G) {
      const T* qp = static_cast<const T*>(a.q) + (static_cast<size_t>(b) * Nq + head0 + row) * kPdDim;
      const uint2 uo = *reinterpret_cast<const uint2*>(qp + d0);
      const uint2 up = *reinterpret_cast<const uint2*>(qp + d0 + 64);
      const float2 o0 = unpack2<T>(uo.x), o1 = unpack2<T>(uo.y), q0 = unpack2<T>(up.x), q1 = unpack2<T>(up.y);
      own[0] = o0.x; own[1] = o0.y; own[2] = o1.x; own[3] = o1.y;
      par[0] = q0.x; par[1] = q0.y; par[2] = q1.x; par[3] = q1.y;
    }
    const float qscale = 1.4426950408889634f * rsqrtf(static_cast<float>(kPdDim));   // log2(e) / sqrt(d)
    float ro[4], rp[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float f = exp2f(-a.log2_theta * static_cast<float>(2 * (d0 + i)) * (1.0f / kPdDim)) * 0.31830988618379067f;
      float sn, cs;
      sincospif(static_cast<float>(max(seq_len - 1, 0)) * f, &sn, &cs);
      ro[i] = (own[i] * cs - par[i] * sn) * qscale;
      rp[i] = (par[i] * cs + own[i] * sn) * qscale;
    }
    const int c_own = d0 >> 3, c_par = (d0 + 64) >> 3;
    const uint32_t off = (d0 & 7) * 2;
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};\n" ::"r"(qs + row * 256 + ((c_own ^ row) << 4) + off),
                 "r"(pack2<T>(ro[0], ro[1])), "r"(pack2<T>(ro[2], ro[3])) : "memory");
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};\n" ::"r"(qs + row * 256 + ((c_par ^ row) << 4) + off),
                 "r"(pack2<T>(rp[0], rp[1])), "r"(pack2<T>(rp[2], rp[3])) : "memory");
  }
  // the turns by the warp's step and by 8 keys, and the frequencies: (cos, cos, sin, sin) of two frequencies each
  float* rot = reinterpret_cast<float*>(pd_smem + kPdRotOff);
  if (tid < 64) {
    const float f = exp2f(-a.log2_theta * static_cast<float>(2 * tid) * (1.0f / kPdDim)) * 0.31830988618379067f;
    float sn, cs;
    float* r = rot + (tid >> 1) * 4 + (tid & 1);
    sincospif(static_cast<float>(kPdStep) * f, &sn, &cs);
    r[0] = cs;
    r[2] = sn;
    sincospif(8.0f * f, &sn, &cs);
    r[128] = cs;
    r[130] = sn;
    rot[256 + tid] = f;
  }
  __syncthreads();
  uint32_t qf[8][2];   // B operand: dimensions 16 ks ..., column = head
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = lane & 7, chunk = 4 * i + (lane >> 3);
    uint32_t f4[4];
    ldsm_x4(f4, qs + r * 256 + ((chunk ^ r) << 4));
    qf[2 * i][0] = f4[0];
    qf[2 * i][1] = f4[1];
    qf[2 * i + 1][0] = f4[2];
    qf[2 * i + 1][1] = f4[3];
  }

  // ---- this warp's ring and its loader ----
  const uint32_t ring = sbase + warp * kPdWarpRing;
  const size_t head_off = (static_cast<size_t>(a.layer_idx) * 2 * a.num_kv_heads + kvh) * P * kPdDim;
  const size_t kv_delta = static_cast<size_t>(a.num_kv_heads) * P * kPdDim;
  bool bad_ptr = false;
  const int lp = 31 - __clz(P);   // the page size is a power of two (checked by the host)
  // The two halves of a tile (keys 0-7 and 8-15) each lie inside one page (pages hold a multiple of 8
  // entries).  Their addresses are looked up one tile ahead, so that the loads of the page table are
  // in flight while the previous tile is being computed and never sit in front of the copies.
  const T* half_ptr[2] = {nullptr, nullptr};
  auto lookup = [&](int j) {
    half_ptr[0] = half_ptr[1] = nullptr;
    if (j < ntw) {
      const int key0 = (tile0 + warp + j * kPdWarps) * kPdTile;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int gk = key0 + 8 * h;
        if (gk < seq_len) {
          const T* page = static_cast<const T*>(a.kv_ptrs[p0 + (gk >> lp)]);
          if (page == nullptr || (reinterpret_cast<uintptr_t>(page) & 15) != 0) bad_ptr = true;
          else half_ptr[h] = page + head_off + static_cast<size_t>(gk & (P - 1)) * kPdDim;
        }
      }
    }
  };
  // lane l copies chunk l & 15 of the keys 2 k + (l >> 4); chunk c of key e sits at slot c ^ (e & 7)
  const int cch = lane & 15, ckey = lane >> 4;
  const uint32_t dst_row = ckey * 256;
  auto issue = [&](int j) {   // j-th tile of this warp; its addresses were looked up before
    if (j < ntw) {
      const int key0 = (tile0 + warp + j * kPdWarps) * kPdTile;
      const uint32_t kst = ring + (j % kPdStages) * (2 * kPdTileBytes) + dst_row;
      const int valid = seq_len - key0 - ckey;   // key 2 k of this lane exists if 2 k < valid
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const bool have = half_ptr[h] != nullptr;
        const T* src = have ? half_ptr[h] + ckey * kPdDim + cch * 8 : static_cast<const T*>(a.q);
        const T* vsrc = have ? src + kv_delta : src;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const bool ok = have && 8 * h + 2 * k < valid;                    // keys past the end read as zeros
          const int step = ok ? 2 * k * kPdDim : 0;
          const uint32_t dst = kst + (8 * h + 2 * k) * 256 + ((cch ^ (2 * k + ckey)) << 4);
          cp_async16(dst, src + step, ok);
          cp_async16(dst + kPdTileBytes, vsrc + step, ok);
        }
      }
    }
    cp_async_commit();
    lookup(j + 1);
  };
  lookup(0);
#pragma unroll
  for (int j = 0; j < kPdStages - 1; ++j) issue(j);

  // cosines and sines of key g of the tile: pair p = 2 ks + h holds the frequencies 16 ks + 8 h + 2 t and the next
  uint64_t cc[8], ss[8];
  float m_run[2] = {-INFINITY, -INFINITY};   // heads 2 t and 2 t + 1
  float l_run[2] = {0.f, 0.f};               // this lane's keys' share of the sums
  float o[8][4];                             // dims 16 i + g and + 8, heads 2 t and 2 t + 1
#pragma unroll
  for (int i = 0; i < 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;

  const int lm = lane >> 3, lr = lane & 7;
  const uint32_t k_row = ((lm & 1) * 8 + lr) * 256, k_x = ((lm >> 1) ^ lr) << 4;             // matrices: key half, dim half
  const uint32_t v_row = kPdTileBytes + ((lm >> 1) * 8 + lr) * 256, v_x = ((lm & 1) ^ lr) << 4;  // dim half, key half

  for (int j = 0; j < ntw; ++j) {
    issue(j + kPdStages - 1);
    const int key0 = (tile0 + warp + j * kPdWarps) * kPdTile;
    if (j % kPdReseed == 0) {
#pragma unroll
      for (int p = 0; p < 8; ++p) {
        const float2 f = *reinterpret_cast<const float2*>(rot + 256 + 8 * p + 2 * t);
        const float pos = static_cast<float>(key0 + g);
        float s0, s1, c0, c1;
        fast_sincospi(pos * f.x, &s0, &c0);
        fast_sincospi(pos * f.y, &s1, &c1);
        cc[p] = pack_f32x2(c0, c1);
        ss[p] = pack_f32x2(s0, s1);
      }
    }
    cp_async_wait<kPdStages - 1>();
    __syncwarp();
    const uint32_t kst = ring + (j % kPdStages) * (2 * kPdTileBytes);
    // S^T = K . Q^T with the keys rotated on the way (a dimension's k step and its partner's accumulate separately)
    float sc[2][4];
#pragma unroll
    for (int n = 0; n < 2; ++n) sc[n][0] = sc[n][1] = sc[n][2] = sc[n][3] = 0.f;
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      uint32_t own[4], par[4];
      const uint32_t ka = kst + k_row + (k_x ^ (ks << 5));
      ldsm_x4(own, ka);
      ldsm_x4(par, ka + 128);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int p = 2 * ks + h;
        const ulonglong2 t8 = *reinterpret_cast<const ulonglong2*>(rot + 128 + (4 * p + t) * 4);
        const ulonglong2 tw = *reinterpret_cast<const ulonglong2*>(rot + (4 * p + t) * 4);
        uint64_t c = cc[p], s = ss[p];
#pragma unroll
        for (int e = 0; e < 2; ++e) {   // key g, then key g + 8
          const float2 x = unpack2<T>(own[2 * h + e]), y = unpack2<T>(par[2 * h + e]);
          const uint64_t ko = pack_f32x2(x.x, x.y), kp = pack_f32x2(y.x, y.y);
          float a0, a1, b0, b1;
          unpack_f32x2(fma_f32x2(ko, c, mul_f32x2(kp, s ^ 0x8000000080000000ull)), a0, a1);   // ko c - kp s
          unpack_f32x2(fma_f32x2(kp, c, mul_f32x2(ko, s)), b0, b1);                           // kp c + ko s
          own[2 * h + e] = pack2<T>(a0, a1);
          par[2 * h + e] = pack2<T>(b0, b1);
          if (e == 0) turn_f32x2(c, s, t8.x, t8.y);
        }
        turn_f32x2(cc[p], ss[p], tw.x, tw.y);
      }
      mma16816<T>(sc[0], own, qf[ks][0], qf[ks][1]);
      mma16816<T>(sc[1], par, qf[ks + 4][0], qf[ks + 4][1]);
    }
    // running softmax: keys g and g + 8 of heads 2 t and 2 t + 1
    float x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = sc[0][i] + sc[1][i];
    if (key0 + kPdTile > seq_len) {
      if (key0 + g >= seq_len) x[0] = x[1] = -INFINITY;
      if (key0 + g + 8 >= seq_len) x[2] = x[3] = -INFINITY;
    }
    float mx[2] = {fmaxf(x[0], x[2]), fmaxf(x[1], x[3])};
    if (__any_sync(0xffffffffu, mx[0] > m_run[0] || mx[1] > m_run[1])) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
#pragma unroll
        for (int d = 4; d < 32; d <<= 1) mx[q] = fmaxf(mx[q], __shfl_xor_sync(0xffffffffu, mx[q], d));
        const float mn = fmaxf(m_run[q], mx[q]);
        const float rescale = exp2f(m_run[q] - mn);   // exp2f(-inf) = 0 on the first tile
        m_run[q] = mn;
        l_run[q] *= rescale;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          o[i][q] *= rescale;
          o[i][q + 2] *= rescale;
        }
      }
    }
    float pr[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) pr[i] = exp2f(x[i] - m_run[i & 1]);
    l_run[0] += pr[0] + pr[2];
    l_run[1] += pr[1] + pr[3];
    // O^T += V^T . P^T ; P comes as [key][heads] and is transposed into the B operand
    const uint32_t pb0 = movm_t(pack2<T>(pr[0], pr[1])), pb1 = movm_t(pack2<T>(pr[2], pr[3]));
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      uint32_t vf[4];
      ldsm_x4_t(vf, kst + v_row + ((i >> 2) << 7) + (v_x ^ ((i & 3) << 5)));
      mma16816<T>(o[i], vf, pb0, pb1);
    }
    __syncwarp();   // the stage is free for the copy issued in the next iteration
  }
  cp_async_wait<0>();
  if (__any_sync(0xffffffffu, bad_ptr) && lane == 0 && a.err != nullptr) atomicOr(a.err, kErrBadPointer);
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int d = 4; d < 32; d <<= 1) l_run[q] += __shfl_xor_sync(0xffffffffu, l_run[q], d);
  __syncthreads();   // every warp is done with its ring: it becomes the merge area

  // ---- merge the warps in warp order (a fixed order): per (warp, head) m, l, 2 unused, o[128]; thread = dim ----
  float* red = reinterpret_cast<float*>(pd_smem);
  constexpr int REC = kPdRec;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int h = 2 * t + q;
    if (h < G) {
      float* r = red + (warp * 8 + h) * REC;
      if (g == 0) {
        r[0] = m_run[q];
        r[1] = l_run[q];
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        r[4 + 16 * i + g] = o[i][q];
        r[4 + 16 * i + 8 + g] = o[i][q + 2];
      }
    }
  }
  __syncthreads();
  T* O = static_cast<T*>(a.o) + (static_cast<size_t>(b) * Nq + head0) * kPdDim + tid;
  float* part = a.partial + (static_cast<size_t>(b) * Nq + head0) * S * REC;   // [head][range]
#pragma unroll
  for (int h = 0; h < G; ++h) {
    float m = -INFINITY, l = 0.f, acc = 0.f;
#pragma unroll
    for (int w = 0; w < kPdWarps; ++w) {
      const float* r = red + (w * 8 + h) * REC;
      if (r[1] != 0.f) m = fmaxf(m, r[0]);   // an empty state carries no information
    }
#pragma unroll
    for (int w = 0; w < kPdWarps; ++w) {
      const float* r = red + (w * 8 + h) * REC;
      if (r[1] != 0.f) {
        const float wt = exp2f(r[0] - m);
        l += r[1] * wt;
        acc += r[4 + tid] * wt;
      }
    }
    if (ranges == 1) {
      O[h * kPdDim] = static_cast<T>(l == 0.f ? 0.f : acc * (1.0f / l));   // no keys: zeros; a NaN stays one
    } else {
      float* r = part + (static_cast<size_t>(h) * S + s) * REC;
      if (tid == 0) {
        r[0] = m;
        r[1] = l;
      }
      r[4 + tid] = acc;
    }
  }
  if (ranges == 1) return;

  // ---- several ranges: the last CTA of the (request, kv head) merges the parked states in range order ----
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    const int old = atomicAdd(a.tickets + bh, 1);
    s_last = old == ranges - 1;
    if (old == ranges - 1) a.tickets[bh] = 0;   // leave the workspace ready for the next launch
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
#pragma unroll 1
  for (int h = 0; h < G; ++h) {
    const float* r0 = part + static_cast<size_t>(h) * S * REC;
    float mz[kPdMaxSplits], lz[kPdMaxSplits], oz[kPdMaxSplits];
    float m = -INFINITY, l = 0.f, acc = 0.f;
#pragma unroll
    for (int z = 0; z < kPdMaxSplits; ++z) {
      mz[z] = lz[z] = oz[z] = 0.f;
      if (z < ranges) {
        mz[z] = __ldcg(r0 + z * REC);
        lz[z] = __ldcg(r0 + z * REC + 1);
        oz[z] = __ldcg(r0 + z * REC + 4 + tid);
      }
    }
#pragma unroll
    for (int z = 0; z < kPdMaxSplits; ++z)
      if (lz[z] != 0.f) m = fmaxf(m, mz[z]);
#pragma unroll
    for (int z = 0; z < kPdMaxSplits; ++z) {
      if (lz[z] != 0.f) {
        const float wt = exp2f(mz[z] - m);
        l += lz[z] * wt;
        acc += oz[z] * wt;
      }
    }
    O[h * kPdDim] = static_cast<T>(l == 0.f ? 0.f : acc * (1.0f / l));
  }
}

}  // namespace smlm
