// Phase 2 of the Schur reduction, column-owned with each visit's couplings staged as one contiguous run ("runs").
// Included by schur.cu (after the helpers it uses).
//
// A visit is a coupling c2 of block column r2 (a point that observes camera r2). The pairs of the visit are (c1, c2) for
// the point's couplings c1 <= c2, and C stores a point's couplings one after another, so everything the visit's pairs
// read of C is one contiguous run [c of the point's first coupling, end of C_c2). A CTA owns a column (or a part of
// one, an item) and walks its visits in segments that fit shared memory. Per segment:
// 1. every visit's run is copied into shared memory by one bulk (TMA) copy from the 16-byte boundary at or below it;
// 2. W = E' C_c2 (E' = s_e E^-1 s_e) of every visit is formed in FP64 from shared memory, rounded to the storage type
//    and kept there; the same pass adds C_c2' z' to the column's gradient sums and C_c2' W to its diagonal block;
// 3. the segment's off-diagonal pairs, grouped by S block, are multiplied out of shared memory: a block's pairs are dealt
//    to 1, 2, 4, ... lanes of a warp (units), so that the units of a segment are about equally long and there are enough
//    of them for the CTA's warps; the units, longest first, make batches of 32. A lane accumulates C_c1' W_c2 of its
//    pairs in registers, the lanes of a block add theirs up by shuffles and the first adds the block to the item's
//    tile, kept block by block in shared memory.
// After the last segment the tile, times the conditioning scales of its rows and columns, is subtracted from S (with
// atomics when the column is split into several items) and the gradient sums from g_S. In FP32 the items of a split
// column leave their sums of its diagonal block in dpart, and k_runs_diag adds them up in FP64 and subtracts them once: S
// holds R there, far larger than an item's part, and every subtraction rounds it (60 cameras, 6,000 points, several items a
// column, S against 64 bits over three inputs: 9.0e-8 to 1.2e-7 with a subtraction per item, 5.3e-8 to 6.4e-8 now; the
// launch costs 3 us).
#pragma once

constexpr int kRunThreads = 128;
constexpr long long kCopyFault = -2;   // Status::failed: a bulk copy did not complete within its wait limit
constexpr int kRunMaxVisits = 512;   // visits of a segment

template <class T>
struct RunArgs {
  const int4* items;        // two per item: {r2, first segment, segments, the column's only item}, {first block, blocks, 0, 0}
  const int4* segs;         // {place of the segment's record in `blob`, its 16-byte chunks, visits | batches << 16, bytes of its bulk copies}
  // Per segment, in 16-byte chunks: the visits {first entry of the run in C, its length, its place in the segment's
  // buffer, point}; per batch and lane {block of the column | unit length << 16 | log2 of its lanes << 28};
  // per batch the place of its codes; the codes, four iterations at a time, a chunk per lane {place of C_c1 in the
  // buffer | visit << 16}
  const uint4* blob;
  int64_t nitems, Clen, dense_nr;
  const int64_t* block_base;
  const int32_t *block_stride, *block_r1, *boffsets_r;
  const T* C;
  const double *EZ, *Einv, *z, *s_r, *s_e;
  const int32_t *r_dims, *e_dims, *eoffsets, *boffsets_e;
  T* S;
  double* g;
  Status* st;
  const int32_t* prob_of_cam;
  const long long* prob_fail;
  unsigned long long* queue;
  double* dpart;            // FP32: per item of a split column its sums of the diagonal block, column by column, mdr apart
  int tile_bytes, blob_bytes, wr, ts, mdr, mde;   // shared-memory layout (wr, ts, mdr, mde for k_runs_any only)
};

// 16-byte chunks of the bulk copy of a run (first entry x, y entries): all it touches, short of C's end
template <class T>
__host__ __device__ inline int run_chunks(int x, int y, int64_t Clen) {
  constexpr int EPC = 16 / (int)sizeof(T);
  const int ph = x & (EPC - 1), n = (ph + y + EPC - 1) / EPC;
  const int64_t whole = (Clen - (x - ph)) / EPC;
  return whole < n ? (int)whole : n;
}

// Copies a segment's record into shared memory.
__device__ __forceinline__ void run_blob(uint4* dst, const uint4* __restrict__ blob, const int4& seg) {
  for (int i = threadIdx.x; i < seg.y; i += kRunThreads) run_cp16(dst + i, blob + seg.x + i, 16);
}

// Copies the runs of a segment's visits into its buffer, a bulk copy per visit issued by the visit's thread. C starts on a
// 16-byte boundary and a run's place in the buffer has the same offset within 16 bytes as its first entry in C. A run
// that ends in C's last, partial chunk takes that chunk's entries with plain loads.
template <class T>
__device__ __forceinline__ void run_stage(const RunArgs<T>& a, T* buf, const int4* vis, int nv, uint64_t* bar) {
  constexpr int EPC = 16 / (int)sizeof(T);
  for (int v = threadIdx.x; v < nv; v += kRunThreads) {
    const int4 r = vis[v];
    const int ph = r.x & (EPC - 1);
    const int c0 = r.x - ph, n = run_chunks<T>(r.x, r.y, a.Clen);
    if (n > 0) bulk_g2s(buf + (r.z - ph), a.C + c0, 16 * n, bar);
    for (int i = max(ph, n * EPC); i < ph + r.y; ++i) buf[r.z - ph + i] = a.C[c0 + i];
  }
}

// Waits for the segment's bulk copies (every thread calls it). A wait that gives up records a fault (the reduction
// reports it), waits once more so that the copies do not outlive the CTA, and true is returned to every thread.
__device__ __forceinline__ bool run_failed(uint64_t* bar, uint32_t phase, Status* st) {
  const bool gave_up = !mbar_wait(bar, phase);
  if (!__syncthreads_or(gave_up)) return false;
  if (threadIdx.x == 0) atomicMin(&st->failed, kCopyFault);
  mbar_wait(bar, phase);
  return true;
}

// N consecutive entries of shared memory whose address is a multiple of A entries (A entries fill at most 16 bytes)
template <int N, int A, class T>
__device__ __forceinline__ void ld_smem(const T* p, T* out) {
  if constexpr (A * sizeof(T) >= 16) {
    constexpr int V = 16 / sizeof(T);
#pragma unroll
    for (int i = 0; i + V <= N; i += V) {
      const uint4 x = *reinterpret_cast<const uint4*>(p + i);
      __builtin_memcpy(out + i, &x, 16);
    }
#pragma unroll
    for (int i = N / V * V; i < N; ++i) out[i] = p[i];
  } else if constexpr (A * sizeof(T) == 8 && sizeof(T) == 4) {
#pragma unroll
    for (int i = 0; i + 2 <= N; i += 2) {
      const float2 x = *reinterpret_cast<const float2*>(p + i);
      out[i] = x.x;
      out[i + 1] = x.y;
    }
    if (N & 1) out[N - 1] = p[N - 1];
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) out[i] = p[i];
  }
}

// N entries to a 16-byte boundary of shared memory
template <int N, class T>
__device__ __forceinline__ void st_smem(T* p, const T* in) {
  constexpr int V = 16 / sizeof(T);
#pragma unroll
  for (int i = 0; i + V <= N; i += V) {
    uint4 x;
    __builtin_memcpy(&x, in + i, 16);
    *reinterpret_cast<uint4*>(p + i) = x;
  }
#pragma unroll
  for (int i = N / V * V; i < N; ++i) p[i] = in[i];
}

// The layout of an exact-size kernel: the record stride of W (a multiple of 16 bytes, odd in 16-byte units where that
// costs at most one, so that the lanes' records spread over the banks), the stride of a block in the tile, and the
// alignment of a coupling block in entries.
template <class T, int DR, int DE>
struct RunShape {
  static constexpr int EPC = 16 / (int)sizeof(T);
  static constexpr int W16 = (DR * DE + EPC - 1) / EPC;
  static constexpr int WR = (W16 | 1) * EPC;
  static constexpr int TS = (DR * DR + EPC - 1) / EPC * EPC;
  static constexpr int AL = (DR * DE) % EPC == 0 ? EPC : (DR * DE) % 2 == 0 ? 2 : 1;
};

// Every retained block of DR variables, every eliminated one of DE = 3 (E' and z' from the factor kernel's record).
// A lane owns CW columns of its unit's block (DR / CW passes over the batch).
template <class T, int DR, int CW>
__global__ void __launch_bounds__(kRunThreads, 2) k_runs(RunArgs<T> a) {
  constexpr int DE = 3, NT = kRunThreads, NW = NT / 32, B = DR * DE, TRI = DR * (DR + 1) / 2, PARTS = DR / CW;
  using Sh = RunShape<T, DR, DE>;
  static_assert(DR % CW == 0, "parts of equal width");
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ int s_item, s_bat;
  __shared__ double gp[NW][DR];
  __shared__ __align__(8) uint64_t bar;
  __shared__ T dgp[NW][TRI];
  if (!live(a.st)) return;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  uint32_t phase = 0;
  if (tid == 0) {
    mbar_init(&bar, 1);
    mbar_fence_init();
  }
  T* tile = reinterpret_cast<T*>(sm);
  auto blob = [&](int i) { return reinterpret_cast<uint4*>(sm + a.tile_bytes + (i & 1) * a.blob_bytes); };
  T* buf = reinterpret_cast<T*>(sm + a.tile_bytes + 2 * a.blob_bytes);
  for (;;) {
    if (tid == 0) s_item = (int)atomicAdd(a.queue, 1ull);
    __syncthreads();
    const int item = s_item;
    if (item >= a.nitems) break;
    const int4 it = a.items[2 * item], ib = a.items[2 * item + 1];
    const int r2 = it.x, nblk = ib.y;
    if (a.prob_fail && a.prob_fail[a.prob_of_cam[r2]] != NONE) {   // the column's problem failed: its S stays reset
      __syncthreads();
      continue;
    }
    for (int i = tid; i < nblk * Sh::TS; i += NT) tile[i] = T(0);
    double ga[DR];
#pragma unroll
    for (int w = 0; w < DR; ++w) ga[w] = 0.0;
    T dg[TRI];
#pragma unroll
    for (int i = 0; i < TRI; ++i) dg[i] = T(0);
    // the next segment's record is copied while a segment is worked on
    int4 seg = __ldg(a.segs + it.y);
    run_blob(blob(0), a.blob, seg);
    run_cp_commit();
    for (int sg = 0; sg < it.z; ++sg) {
      const int4 next = sg + 1 < it.z ? __ldg(a.segs + it.y + sg + 1) : make_int4(0, 0, 0, 0);
      const uint4* rec = blob(sg);
      const int nv = seg.z & 0xffff, nb = seg.z >> 16;
      const int4* vis = reinterpret_cast<const int4*>(rec);
      const uint32_t* lanes = reinterpret_cast<const uint32_t*>(rec + nv);
      const int* first = reinterpret_cast<const int*>(lanes + 32 * nb);
      const uint4* codes = rec + nv + 8 * nb + (nb + 3) / 4;
      run_cp_wait<0>();
      if (tid == 0) mbar_arrive_expect_tx(&bar, (uint32_t)seg.w);
      fence_proxy_async_shared();
      __syncthreads();   // the segment's record is in, and the other record and the buffer are free
      if (tid == 0) s_bat = 0;
      run_stage(a, buf, vis, nv, &bar);
      run_blob(blob(sg + 1), a.blob, next);
      run_cp_commit();
      // W, the gradient sums and the diagonal block, a thread per visit; the point's record is in flight with the copies
      double Ep[12];
      auto point = [&](int v) {
        const double2* ez = reinterpret_cast<const double2*>(a.EZ + 12 * (int64_t)vis[v].w);
#pragma unroll
        for (int i = 0; i < 6; ++i) { const double2 x = __ldg(ez + i); Ep[2 * i] = x.x; Ep[2 * i + 1] = x.y; }
      };
      if (tid < nv) point(tid);
      if (run_failed(&bar, phase, a.st)) return;
      phase ^= 1;
      for (int v = tid; v < nv; v += NT) {
        const int4 vr = vis[v];
        T* wv = buf + v * Sh::WR;
        if (v != tid) point(v);
        T c[B];
        ld_smem<B, Sh::AL>(buf + vr.z + vr.y - B, c);
        T wr[B];
#pragma unroll
        for (int w = 0; w < DR; ++w) {
          const double c0 = (double)c[3 * w], c1 = (double)c[3 * w + 1], c2 = (double)c[3 * w + 2];
#pragma unroll
          for (int t = 0; t < 3; ++t) wr[3 * w + t] = T(Ep[t] * c0 + Ep[t + 3] * c1 + Ep[t + 6] * c2);
          ga[w] += c0 * Ep[9] + c1 * Ep[10] + c2 * Ep[11];
        }
        st_smem<B>(wv, wr);
#pragma unroll
        for (int cc = 0; cc < DR; ++cc)
#pragma unroll
          for (int rho = 0; rho <= cc; ++rho) {
            T x = dg[cc * (cc + 1) / 2 + rho];
            x = fma(c[3 * rho], wr[3 * cc], x);
            x = fma(c[3 * rho + 1], wr[3 * cc + 1], x);
            x = fma(c[3 * rho + 2], wr[3 * cc + 2], x);
            dg[cc * (cc + 1) / 2 + rho] = x;
          }
      }
      __syncthreads();
      for (;;) {
        int b = 0;
        if (lane == 0) b = atomicAdd(&s_bat, 1);
        b = __shfl_sync(0xffffffffu, b, 0);
        if (b >= nb * PARTS) break;
        const int part = PARTS == 1 ? 0 : b % PARTS;
        const int bi = PARTS == 1 ? b : b / PARTS;
        const uint32_t lr = lanes[32 * bi + lane];
        const int len = (int)((lr >> 16) & 0xfff), iters = __shfl_sync(0xffffffffu, len, 0);   // lane 0 holds the longest
        const uint4* pc = codes + first[bi] + lane;
        T acc[CW][DR];
#pragma unroll
        for (int c = 0; c < CW; ++c)
#pragma unroll
          for (int rho = 0; rho < DR; ++rho) acc[c][rho] = T(0);
        for (int i0 = 0; i0 < iters; i0 += 4) {
          const uint4 cur = pc[8 * i0];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t code = i == 0 ? cur.x : i == 1 ? cur.y : i == 2 ? cur.z : cur.w;
            if (i0 + i < len) {
              T p[B], w[CW * DE];
              ld_smem<B, Sh::AL>(buf + (code & 0xffff), p);
              ld_smem<CW * DE, PARTS == 1 ? Sh::EPC : 1>(buf + (code >> 16) * Sh::WR + part * CW * DE, w);
#pragma unroll
              for (int c = 0; c < CW; ++c)
#pragma unroll
                for (int rho = 0; rho < DR; ++rho) {
                  T x = acc[c][rho];
                  x = fma(p[3 * rho], w[3 * c], x);
                  x = fma(p[3 * rho + 1], w[3 * c + 1], x);
                  x = fma(p[3 * rho + 2], w[3 * c + 2], x);
                  acc[c][rho] = x;
                }
            }
          }
        }
        // the lanes of a block (a power of two, side by side) add up
        const int lg = (int)(lr >> 28), levels = __reduce_max_sync(0xffffffffu, lg);
        for (int j = 0; j < levels; ++j) {
#pragma unroll
          for (int c = 0; c < CW; ++c)
#pragma unroll
            for (int rho = 0; rho < DR; ++rho) {
              const T x = __shfl_down_sync(0xffffffffu, acc[c][rho], 1 << j);
              if (j < lg) acc[c][rho] += x;
            }
        }
        if (len > 0 && (lane & ((1 << lg) - 1)) == 0) {
          T* tb = tile + (size_t)(lr & 0xffff) * Sh::TS + part * CW * DR;
          T old[CW * DR];
          ld_smem<CW * DR, PARTS == 1 ? Sh::EPC : 1>(tb, old);
#pragma unroll
          for (int c = 0; c < CW; ++c)
#pragma unroll
            for (int rho = 0; rho < DR; ++rho) old[c * DR + rho] += acc[c][rho];
          if constexpr (PARTS == 1) {
            st_smem<CW * DR>(tb, old);
          } else {
#pragma unroll
            for (int i = 0; i < CW * DR; ++i) tb[i] = old[i];
          }
        }
      }
      seg = next;
    }
    __syncthreads();   // every batch is in the tile
    // the column's sums, per warp and then over the warps in warp order
#pragma unroll
    for (int w = 0; w < DR; ++w) {
      double x = ga[w];
      for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      if (lane == 0) gp[wid][w] = x;
    }
#pragma unroll
    for (int i = 0; i < TRI; ++i) {
      T x = dg[i];
      for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      if (lane == 0) dgp[wid][i] = x;
    }
    __syncthreads();
    if (tid < TRI) {   // the column's last block is the diagonal one; no batch writes it
      int cc = 0;
      while ((cc + 1) * (cc + 2) / 2 <= tid) ++cc;
      const int rho = tid - cc * (cc + 1) / 2;
      if (it.w || sizeof(T) == 8) {
        T x = dgp[0][tid];
        for (int w = 1; w < NW; ++w) x += dgp[w][tid];
        tile[(size_t)(nblk - 1) * Sh::TS + cc * DR + rho] = x;
      } else {
        double x = 0.0;
        for (int w = 0; w < NW; ++w) x += (double)dgp[w][tid];
        a.dpart[(int64_t)item * DR * DR + cc * DR + rho] = x;
      }
    }
    __syncthreads();
    const int64_t stride = a.block_stride ? (int64_t)__ldg(a.block_stride + ib.x) : a.dense_nr;
    double fc[DR];
#pragma unroll
    for (int w = 0; w < DR; ++w) fc[w] = a.s_r ? a.s_r[DR * (int64_t)r2 + w] : 1.0;
    for (int rr = tid; rr < nblk * DR; rr += NT) {
      const int k = rr / DR, rho = rr - k * DR;
      const double f = a.s_r ? a.s_r[DR * (int64_t)__ldg(a.block_r1 + ib.x + k) + rho] : 1.0;
      T* Sr = a.S + __ldg(a.block_base + ib.x + k) + rho;
      const T* tr = tile + (size_t)k * Sh::TS + rho;
      if (it.w) {
        T old[DR];
#pragma unroll
        for (int w = 0; w < DR; ++w) old[w] = Sr[w * stride];
#pragma unroll
        for (int w = 0; w < DR; ++w) Sr[w * stride] = old[w] - T((double)tr[w * DR] * (f * fc[w]));
      } else if (sizeof(T) == 8 || k < nblk - 1) {
#pragma unroll
        for (int w = 0; w < DR; ++w) atomicAdd(Sr + w * stride, -T((double)tr[w * DR] * (f * fc[w])));
      }
    }
    if (tid < DR) {
      double x = 0.0;
      for (int w = 0; w < NW; ++w) x += gp[w][tid];
      atomicAdd(a.g + DR * (int64_t)r2 + tid, -(a.s_r ? a.s_r[DR * (int64_t)r2 + tid] : 1.0) * x);
    }
    __syncthreads();   // the item's shared memory is free for the next one
  }
}

// Any block sizes up to 16, MDR bounding the retained ones (kernel parameters mdr, mde: the plan's largest): a thread
// per (visit, column of C_c2) forms W, the products run over a pair's d_e variables one at a time (an outer product of
// a column of C_c1' and one of W per variable), a lane owning CW columns of its unit's block.
template <class T, int MDR, int CW>
__global__ void __launch_bounds__(kRunThreads, 2) k_runs_any(RunArgs<T> a) {
  constexpr int NT = kRunThreads;
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ int s_item, s_bat;
  __shared__ double gs[16];
  __shared__ __align__(8) uint64_t bar;
  __shared__ unsigned char vde[kRunMaxVisits];
  if (!live(a.st)) return;
  const int tid = threadIdx.x, lane = tid & 31;
  uint32_t phase = 0;
  if (tid == 0) {
    mbar_init(&bar, 1);
    mbar_fence_init();
  }
  T* tile = reinterpret_cast<T*>(sm);
  auto blob = [&](int i) { return reinterpret_cast<uint4*>(sm + a.tile_bytes + (i & 1) * a.blob_bytes); };
  T* buf = reinterpret_cast<T*>(sm + a.tile_bytes + 2 * a.blob_bytes);
  const int mdr = a.mdr, mde = a.mde;
  for (;;) {
    if (tid == 0) s_item = (int)atomicAdd(a.queue, 1ull);
    if (tid < 16) gs[tid] = 0.0;
    __syncthreads();
    const int item = s_item;
    if (item >= a.nitems) break;
    const int4 it = a.items[2 * item], ib = a.items[2 * item + 1];
    const int r2 = it.x, nblk = ib.y;
    const int d2 = __ldg(a.r_dims + r2), ro2 = __ldg(a.boffsets_r + r2);
    const int parts = (d2 + CW - 1) / CW;
    const int grp = tid / d2, wcol = tid - grp * d2, ngrp = NT / d2;
    for (int i = tid; i < nblk * a.ts; i += NT) tile[i] = T(0);
    double ga = 0.0;
    T dg[MDR];
#pragma unroll
    for (int i = 0; i < MDR; ++i) dg[i] = T(0);
    // the next segment's record is copied while a segment is worked on
    int4 seg = __ldg(a.segs + it.y);
    run_blob(blob(0), a.blob, seg);
    run_cp_commit();
    for (int sg = 0; sg < it.z; ++sg) {
      const int4 next = sg + 1 < it.z ? __ldg(a.segs + it.y + sg + 1) : make_int4(0, 0, 0, 0);
      const uint4* rec = blob(sg);
      const int nv = seg.z & 0xffff, nb = seg.z >> 16;
      const int4* vis = reinterpret_cast<const int4*>(rec);
      const uint32_t* lanes = reinterpret_cast<const uint32_t*>(rec + nv);
      const int* first = reinterpret_cast<const int*>(lanes + 32 * nb);
      const uint4* codes = rec + nv + 8 * nb + (nb + 3) / 4;
      run_cp_wait<0>();
      if (tid == 0) mbar_arrive_expect_tx(&bar, (uint32_t)seg.w);
      fence_proxy_async_shared();
      __syncthreads();   // the segment's record is in, and the other record and the buffer are free
      if (tid == 0) s_bat = 0;
      run_stage(a, buf, vis, nv, &bar);
      run_blob(blob(sg + 1), a.blob, next);
      run_cp_commit();
      if (run_failed(&bar, phase, a.st)) return;
      phase ^= 1;
      if (grp < ngrp)
        for (int v = grp; v < nv; v += ngrp) {
          const int4 vr = vis[v];
          const int e = vr.w, de = __ldg(a.e_dims + e), so = __ldg(a.boffsets_e + e);
          const double* Ei = a.Einv + __ldg(a.eoffsets + e);
          const T* cb = buf + vr.z + vr.y - d2 * de;
          T* wv = buf + v * a.wr + wcol * mde;
          for (int t = 0; t < de; ++t) {
            double x = 0.0;
            for (int s = 0; s < de; ++s) x += __ldg(Ei + t + de * s) * ((a.s_e ? a.s_e[so + s] : 1.0) * (double)cb[wcol * de + s]);
            const double se = a.s_e ? a.s_e[so + t] : 1.0;
            wv[t] = T(se * x);
            ga += (double)cb[wcol * de + t] * (se * __ldg(a.z + so + t));
          }
#pragma unroll
          for (int rho = 0; rho < MDR; ++rho)
            if (rho <= wcol) {
              T x = dg[rho];
              for (int t = 0; t < de; ++t) x = fma(cb[rho * de + t], wv[t], x);
              dg[rho] = x;
            }
          if (wcol == 0) vde[v] = (unsigned char)de;
        }
      __syncthreads();
      for (;;) {
        int b = 0;
        if (lane == 0) b = atomicAdd(&s_bat, 1);
        b = __shfl_sync(0xffffffffu, b, 0);
        if (b >= nb * parts) break;
        const int bi = b / parts, c0 = (b % parts) * CW;
        const uint32_t lr = lanes[32 * bi + lane];
        const int len = (int)((lr >> 16) & 0xfff), iters = __shfl_sync(0xffffffffu, len, 0);
        const int d1 = len > 0 ? __ldg(a.r_dims + __ldg(a.block_r1 + ib.x + (int)(lr & 0xffff))) : 0;
        const uint4* pc = codes + first[bi] + lane;
        uint4 cur = pc[0];
        T acc[CW][MDR];
#pragma unroll
        for (int c = 0; c < CW; ++c)
#pragma unroll
          for (int rho = 0; rho < MDR; ++rho) acc[c][rho] = T(0);
        for (int i = 0; i < iters; ++i) {
          const uint32_t code = (i & 3) == 0 ? cur.x : (i & 3) == 1 ? cur.y : (i & 3) == 2 ? cur.z : cur.w;
          if (i < len) {
            const int v = (int)(code >> 16), de = vde[v];
            const T* p = buf + (code & 0xffff);
            const T* w = buf + v * a.wr + c0 * mde;
            for (int s = 0; s < de; ++s) {
              T q[MDR];
#pragma unroll
              for (int rho = 0; rho < MDR; ++rho) q[rho] = rho < d1 ? p[rho * de + s] : T(0);
#pragma unroll
              for (int c = 0; c < CW; ++c) {
                const T x = c0 + c < d2 ? w[c * mde + s] : T(0);
#pragma unroll
                for (int rho = 0; rho < MDR; ++rho) acc[c][rho] = fma(q[rho], x, acc[c][rho]);
              }
            }
          }
          if ((i & 3) == 3 && i + 1 < iters) cur = pc[8 * (i + 1)];
        }
        const int lg = (int)(lr >> 28), levels = __reduce_max_sync(0xffffffffu, lg);
        for (int j = 0; j < levels; ++j) {
#pragma unroll
          for (int c = 0; c < CW; ++c)
#pragma unroll
            for (int rho = 0; rho < MDR; ++rho) {
              const T x = __shfl_down_sync(0xffffffffu, acc[c][rho], 1 << j);
              if (j < lg) acc[c][rho] += x;
            }
        }
        if (len > 0 && (lane & ((1 << lg) - 1)) == 0) {
          T* tb = tile + (size_t)(lr & 0xffff) * a.ts + c0 * mdr;
#pragma unroll
          for (int c = 0; c < CW; ++c)
#pragma unroll
            for (int rho = 0; rho < MDR; ++rho)
              if (c0 + c < d2 && rho < d1) tb[c * mdr + rho] += acc[c][rho];
        }
      }
      seg = next;
    }
    __syncthreads();
    // the column's sums: the diagonal block into the tile's last block, the gradient into shared memory
    if (grp < ngrp) {
      T* td = tile + (size_t)(nblk - 1) * a.ts + wcol * mdr;
#pragma unroll
      for (int rho = 0; rho < MDR; ++rho)
        if (rho <= wcol) atomicAdd(td + rho, dg[rho]);
      atomicAdd(gs + wcol, ga);
    }
    __syncthreads();
    if (!it.w && sizeof(T) == 4)
      for (int x = tid; x < mdr * d2; x += NT) a.dpart[(int64_t)item * mdr * mdr + x] = (double)tile[(size_t)(nblk - 1) * a.ts + x];
    const int64_t stride = a.block_stride ? (int64_t)__ldg(a.block_stride + ib.x) : a.dense_nr;
    for (int x = tid; x < nblk * mdr; x += NT) {
      const int k = x / mdr, rho = x - k * mdr;
      const int r1 = __ldg(a.block_r1 + ib.x + k);
      if (rho >= __ldg(a.r_dims + r1)) continue;
      const double f = a.s_r ? a.s_r[__ldg(a.boffsets_r + r1) + rho] : 1.0;
      T* Sr = a.S + __ldg(a.block_base + ib.x + k) + rho;
      const T* tr = tile + (size_t)k * a.ts + rho;
      for (int w = 0; w < d2; ++w) {
        if (r1 == r2 && (rho > w || (!it.w && sizeof(T) == 4))) continue;
        const T y = T((double)tr[w * mdr] * (f * (a.s_r ? a.s_r[ro2 + w] : 1.0)));
        if (it.w) Sr[w * stride] -= y;
        else atomicAdd(Sr + w * stride, -y);
      }
    }
    if (tid < d2) atomicAdd(a.g + ro2 + tid, -(a.s_r ? a.s_r[ro2 + tid] : 1.0) * gs[tid]);
    __syncthreads();
  }
}

// FP32: the diagonal blocks of the split columns ({r2, first item, items, block}): a thread per entry of the upper triangle.
// Launched beside the end of k_runs (programmatic serialisation), it waits for that kernel's results itself.
template <class T>
__global__ void __launch_bounds__(128) k_runs_diag(RunArgs<T> a, int64_t nsplit, const int4* __restrict__ split) {
  const int64_t id = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int per = a.mdr * a.mdr, e = (int)(id % per), w = e / a.mdr, rho = e - w * a.mdr;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (id / per >= nsplit || !live(a.st)) return;
  const int4 c = __ldg(split + id / per);
  if (rho > w || w >= __ldg(a.r_dims + c.x) || (a.prob_fail && a.prob_fail[a.prob_of_cam[c.x]] != NONE)) return;
  const double* part = a.dpart + (int64_t)c.y * per + e;
  double x = 0.0;
  for (int i = 0; i < c.z; ++i) x += part[(int64_t)i * per];
  const int64_t stride = a.block_stride ? (int64_t)__ldg(a.block_stride + c.w) : a.dense_nr;
  const int64_t ro = __ldg(a.boffsets_r + c.x);
  a.S[__ldg(a.block_base + c.w) + rho + w * stride] -= T(x * ((a.s_r ? a.s_r[ro + rho] : 1.0) * (a.s_r ? a.s_r[ro + w] : 1.0)));
}

// ------------------------------------------------------------------------------------------------------------------
// The schedule of one storage type, built with the plan
// ------------------------------------------------------------------------------------------------------------------
struct RunInput {
  int64_t nrb, neb, Clen;
  int nsm;   // the device's SMs
  const int64_t *r_dims, *e_dims, *eptr, *eret, *coffsets;
  const std::vector<int32_t>*rptr, *rentry, *entry_elim;
  const std::vector<int64_t>*bcolptr, *browval;
};

// Whether C stores each point's couplings one after another (then a visit's pairs read one contiguous run).
static bool runs_contiguous(const RunInput& in) {
  for (int64_t e = 0; e < in.neb; ++e)
    for (int64_t c = in.eptr[e] + 1; c < in.eptr[e + 1]; ++c)
      if (in.coffsets[c] != in.coffsets[c - 1] + in.r_dims[in.eret[c - 1]] * in.e_dims[e]) return false;
  return true;
}

template <class T>
static bool build_run_schedule(RunSchedule& R, const RunInput& in, int exact, int mdr, int mde, cudaStream_t s, SmallBufs& small) {
  constexpr int EPC = 16 / (int)sizeof(T);
  R.exact = exact;
  R.mdr = mdr;
  R.mde = mde;
  if (exact == 6) { R.wr = RunShape<T, 6, 3>::WR; R.ts = RunShape<T, 6, 3>::TS; }
  else if (exact == 7) { R.wr = RunShape<T, 7, 3>::WR; R.ts = RunShape<T, 7, 3>::TS; }
  else if (exact == 8) { R.wr = RunShape<T, 8, 3>::WR; R.ts = RunShape<T, 8, 3>::TS; }
  else if (exact == 9) { R.wr = RunShape<T, 9, 3>::WR; R.ts = RunShape<T, 9, 3>::TS; }
  else {
    R.wr = ((mdr * mde + EPC - 1) / EPC | 1) * EPC;
    R.ts = (mdr * mdr + EPC - 1) / EPC * EPC;
  }
  const std::vector<int32_t>&rptr = *in.rptr, &rentry = *in.rentry, &entry_elim = *in.entry_elim;
  int64_t max_blk = 0, nvis = 0;
  for (int64_t r2 = 0; r2 < in.nrb; ++r2) {
    max_blk = std::max<int64_t>(max_blk, (*in.bcolptr)[r2 + 1] - (*in.bcolptr)[r2]);
    nvis += rptr[r2 + 1] - rptr[r2];
  }
  if (nvis == 0 || max_blk > 65535) return false;
  // Shared memory of a CTA: the column's tile, two segment records, a segment's W records and runs. CTAs per SM: as many
  // as the registers allow (three for 6 x 6 FP32 blocks, else two) if that leaves a segment 40 KB, else fewer: a longer
  // segment gives each block more pairs per addition to the tile (1000 cameras and 200k points, FP32: 250 us with three,
  // 273 with two, 332 with four; FP64 461 with two, 622 with three).
  const int64_t tile = max_blk * R.ts * (int64_t)sizeof(T);
  const int kCtas = sizeof(T) == 4 && exact == 6 ? 3 : 2;
  int64_t budget = 0;
  for (int k = kCtas; k >= 1; --k) {
    budget = std::min<int64_t>((228 * 1024) / k - 1024 - 2560, 222 * 1024) / 16 * 16;
    if (budget - tile >= 40 * 1024 || k == 1) break;
  }
  // a segment's buffer and two records share the rest: a record (16 bytes a visit, 4 a pair, padding) is held to a
  // seventh of it
  if (budget - tile < 24 * 1024) return false;
  const int64_t blob_cap = (budget - tile) / 7 / 16;   // 16-byte chunks
  const int64_t cap = std::min<int64_t>((budget - tile - 32 * blob_cap) / (int64_t)sizeof(T), 65535 - EPC) / EPC * EPC;   // entries
  // Items: four per resident CTA over all columns where that leaves an item 150 visits (every item of a split column adds
  // its whole tile to S with atomics), else as many as there are resident CTAs, of 24 to 150 visits. 1000 cameras and
  // 200k points, FP32: 250 us; with six per CTA and no lower bound the same there, but a scene of 40 cameras and 8000
  // points took 36 us instead of 25.
  const int64_t slots = in.nsm * kCtas;
  const int64_t avg = std::max<int64_t>({24, nvis / (slots * 4), std::min<int64_t>(150, nvis / slots)});
  const int64_t segv = std::min<int64_t>(avg, kRunMaxVisits);
  struct ColOut {
    std::vector<int4> items, segs;
    std::vector<uint4> blob;
  };
  std::vector<ColOut> out(in.nrb);
  int bad = 0;
  int64_t max_chunks = 0;
#pragma omp parallel reduction(| : bad) reduction(max : max_chunks)
  {
    struct Group { int32_t slot, len, lg; };
    std::vector<Group> groups;
    std::vector<int32_t> slot_of(in.nrb, -1), cnt, first, lanes_of, fill;
    std::vector<int32_t> p_slot;
    std::vector<uint32_t> p_code, lane, codes;
    std::vector<int32_t> place;
    std::vector<int4> vis;
#pragma omp for schedule(dynamic, 8)
    for (int64_t r2 = 0; r2 < in.nrb; ++r2) {
      const int64_t q0 = rptr[r2], nv = rptr[r2 + 1] - q0;
      if (nv == 0) continue;
      const int64_t kb = (*in.bcolptr)[r2], nblk = (*in.bcolptr)[r2 + 1] - kb, d2 = in.r_dims[r2];
      if (nblk == 0 || (*in.browval)[kb + nblk - 1] != r2) { bad = 1; continue; }   // the diagonal block closes the column
      for (int64_t k = 0; k < nblk; ++k) slot_of[(*in.browval)[kb + k]] = (int32_t)k;
      ColOut& o = out[r2];
      const int64_t want = std::max<int64_t>(1, (nv + avg / 2) / avg);   // items of this column
      const int64_t per_seg = std::min<int64_t>(segv, (nv + want - 1) / want);
      for (int64_t v0 = 0; v0 < nv && !bad;) {
        // the segment's visits: as many as fit
        int64_t used = 0, np_est = 0, v1 = v0;
        while (v1 < nv && v1 - v0 < per_seg) {
          const int32_t c2 = rentry[q0 + v1];
          const int64_t e = entry_elim[c2], p0 = in.coffsets[in.eptr[e]];
          const int64_t len = in.coffsets[c2] + d2 * in.e_dims[e] - p0, ph = p0 & (EPC - 1);
          const int64_t need = R.wr + (ph + len + EPC - 1) / EPC * EPC;
          // the record: visits, codes (padded: at most a third over, and a partly filled batch), lanes and places
          const int64_t pairs = np_est + (c2 - in.eptr[e]);
          const int64_t chunks = (v1 - v0 + 1) + pairs / 2 + 9 * (std::min<int64_t>(pairs, 2 * nblk + 128) / 32 + 2) + 160;
          if (used + need > cap || (v1 > v0 && chunks > blob_cap)) break;
          used += need;
          np_est = pairs;
          ++v1;
        }
        if (v1 == v0) { bad = 1; break; }   // one visit's run exceeds the buffer
        const int64_t sv = v1 - v0;
        int64_t pos = sv * R.wr;
        vis.clear();
        lane.clear();
        codes.clear();
        place.clear();
        p_slot.clear();
        p_code.clear();
        cnt.assign(nblk, 0);
        first.assign(nblk, 0);
        lanes_of.assign(nblk, 0);
        for (int64_t v = v0; v < v1; ++v) {
          const int32_t c2 = rentry[q0 + v];
          const int64_t e = entry_elim[c2], c_first = in.eptr[e], p0 = in.coffsets[c_first];
          const int64_t len = in.coffsets[c2] + d2 * in.e_dims[e] - p0, ph = p0 & (EPC - 1);
          const int64_t dst = pos + ph;
          pos += (ph + len + EPC - 1) / EPC * EPC;
          vis.push_back(make_int4((int32_t)p0, (int32_t)len, (int32_t)dst, (int32_t)e));
          for (int64_t c1 = c_first; c1 < c2; ++c1) {
            const int32_t sl = slot_of[in.eret[c1]];
            if (sl < 0) { bad = 1; continue; }
            p_slot.push_back(sl);
            p_code.push_back((uint32_t)(dst + in.coffsets[c1] - p0) | ((uint32_t)(v - v0) << 16));
            cnt[sl] += 1;
          }
        }
        // units: a block's pairs of this segment dealt to the fewest lanes (a power of two) that hold at most U each, U
        // for half as many lanes as the CTA has (9 x 3 blocks, 803 cameras: 264 us; U for all its lanes 298 us, with one
        // lane per block 504 us, two of the four warps waiting)
        const int64_t np = (int64_t)p_slot.size();
        const int U = (int)std::max<int64_t>(2, (np + 63) / 64);
        groups.clear();
        for (int64_t k = 0; k < nblk; ++k) {
          if (cnt[k] == 0) continue;
          int lg = 0;
          while (lg < 5 && (cnt[k] + (1 << lg) - 1) >> lg > U) ++lg;
          groups.push_back({(int32_t)k, (cnt[k] + (1 << lg) - 1) >> lg, lg});
        }
        std::stable_sort(groups.begin(), groups.end(), [](const Group& x, const Group& y) { return x.len != y.len ? x.len > y.len : x.lg > y.lg; });
        // batches: the groups in order, each at the next multiple of its lanes
        int64_t nb = 0;
        for (size_t i = 0; i < groups.size();) {
          const int32_t iters = groups[i].len;
          const int64_t base = (int64_t)codes.size();
          place.push_back((int32_t)(base / 4));
          lane.resize(32 * (nb + 1), 0u);
          int L = 0;
          for (; i < groups.size(); ++i) {
            const Group& u = groups[i];
            const int n = 1 << u.lg, at = (L + n - 1) / n * n;
            if (at + n > 32) break;
            first[u.slot] = (int32_t)(base + 4 * at);
            lanes_of[u.slot] = u.lg;
            for (int l = 0; l < n; ++l) {
              const int len = (cnt[u.slot] + n - 1 - l) >> u.lg;   // pairs l, l + n, ...
              lane[32 * nb + at + l] = (uint32_t)u.slot | ((uint32_t)len << 16) | ((uint32_t)u.lg << 28);
            }
            L = at + n;
          }
          codes.resize(base + (iters + 3) / 4 * 128, 0u);
          if (iters > 0xfff) bad = 1;
          ++nb;
        }
        fill.assign(nblk, 0);
        for (int64_t i = 0; i < np; ++i) {
          const int32_t sl = p_slot[i], k = fill[sl]++, lg = lanes_of[sl];
          const int32_t l = k & ((1 << lg) - 1), q = k >> lg;
          codes[first[sl] + 4 * l + (q / 4) * 128 + (q & 3)] = p_code[i];
        }
        place.resize((place.size() + 3) / 4 * 4, 0);
        const int64_t b0 = (int64_t)o.blob.size(), chunks = sv + 8 * nb + (int64_t)place.size() / 4 + (int64_t)codes.size() / 4;
        if (chunks > blob_cap) { bad = 1; break; }
        max_chunks = std::max(max_chunks, chunks);
        o.blob.resize(b0 + chunks);
        uint4* w = o.blob.data() + b0;
        std::memcpy(w, vis.data(), 16 * vis.size());
        std::memcpy(w += sv, lane.data(), 4 * lane.size());
        std::memcpy(w += 8 * nb, place.data(), 4 * place.size());
        std::memcpy(w += place.size() / 4, codes.data(), 4 * codes.size());
        int64_t bytes = 0;
        for (const int4& v : vis) bytes += 16 * (int64_t)run_chunks<T>(v.x, v.y, in.Clen);
        if (nb > 0x7fff) { bad = 1; break; }
        o.segs.push_back(make_int4((int32_t)b0, (int32_t)chunks, (int32_t)(sv | (nb << 16)), (int32_t)bytes));
        v0 = v1;
      }
      const int64_t ns = (int64_t)o.segs.size(), ni = std::min<int64_t>(want, ns);
      for (int64_t i = 0; i < ni; ++i) {
        const int64_t a = i * ns / ni, b = (i + 1) * ns / ni;
        o.items.push_back(make_int4((int32_t)r2, (int32_t)a, (int32_t)(b - a), ni == 1 ? 1 : 0));
        o.items.push_back(make_int4((int32_t)kb, (int32_t)nblk, 0, 0));
      }
      for (int64_t k = 0; k < nblk; ++k) slot_of[(*in.browval)[kb + k]] = -1;
    }
  }
  if (bad) return false;
  // the columns' parts one after another (the blob is tens of MB: uninitialised memory, filled by all threads)
  std::vector<int64_t> at_i(in.nrb + 1, 0), at_s(in.nrb + 1, 0), at_b(in.nrb + 1, 0);
  for (int64_t r = 0; r < in.nrb; ++r) {
    at_i[r + 1] = at_i[r] + (int64_t)out[r].items.size();
    at_s[r + 1] = at_s[r] + (int64_t)out[r].segs.size();
    at_b[r + 1] = at_b[r] + (int64_t)out[r].blob.size();
  }
  const int64_t n_b = at_b[in.nrb];
  if (n_b >= INT32_MAX) return false;
  std::vector<int4> items(at_i[in.nrb]), segs(at_s[in.nrb]);
  const HostArray<uint4> blob(n_b);
#pragma omp parallel for schedule(dynamic, 8)
  for (int64_t r = 0; r < in.nrb; ++r) {
    ColOut& o = out[r];
    for (size_t i = 0; i < o.items.size(); ++i) {
      items[at_i[r] + i] = o.items[i];
      if (i % 2 == 0) items[at_i[r] + i].y += (int32_t)at_s[r];
    }
    for (size_t i = 0; i < o.segs.size(); ++i) {
      segs[at_s[r] + i] = o.segs[i];
      segs[at_s[r] + i].x += (int32_t)at_b[r];
    }
    if (!o.blob.empty()) std::memcpy(blob.get() + at_b[r], o.blob.data(), sizeof(uint4) * o.blob.size());
    o = ColOut();
  }
  small.add(R.items_d, items, s);
  small.add(R.segs, segs, s);
  small.add(R.blob, blob, s);
  std::vector<int4> split;   // FP32: the split columns
  for (size_t i = 0; sizeof(T) == 4 && i < items.size(); i += 2)
    if (items[i].w == 0) {
      if (split.empty() || split.back().x != items[i].x) split.push_back(make_int4(items[i].x, (int32_t)(i / 2), 0, items[i + 1].x + items[i + 1].y - 1));
      split.back().z += 1;
    }
  R.nsplit = (int64_t)split.size();
  if (R.nsplit) {
    small.add(R.split, split, s);
    small.reserve(R.dpart, sizeof(double) * (items.size() / 2) * mdr * mdr);
  }
  R.items = (int64_t)items.size() / 2;
  R.tile_bytes = (int)((tile + 15) / 16 * 16);
  R.blob_bytes = (int)(16 * max_chunks);
  R.smem = R.tile_bytes + 2 * R.blob_bytes + (int)(cap * (int64_t)sizeof(T));
  R.ok = true;
  return true;
}
