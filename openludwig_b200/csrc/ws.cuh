// Warp-specialised persistent stream-collide (FP32 populations).
//
// One CTA per SM walks a static share of the work items (blocks of one level
// for the drop-in entry point, (descriptor, block) items for the block pool).
// Its 544 threads have two roles:
//   * 1 producer warp only starts copies.  It reads the neighbour-table row of
//     item j+1 and, once stage buffer j & 1 is free, starts the TMA bulk copies
//     (cp.async.bulk, completion counted in bytes on an mbarrier) of item j's
//     contiguous arrays: 27 population planes, 3 velocity planes, sponge,
//     obstacle, wall distance, and the 64-cell layers of the two z neighbours
//     (9 population planes each and their velocities) -- 72 KB, moved without
//     registers or request slots.
//   * 16 consumer warps, one cell per thread, per item: write the remaining
//     out-of-block pull sources, which each thread loaded for this item one
//     item earlier (a neighbour's value, the precomputed ghost value, or,
//     without a ghost row, pull_boundary as in the one-CTA-per-block kernel),
//     into the stage slots of the cells that pull them; barrier; WALE from the
//     staged velocities; pull; release the buffer; issue the out-of-block
//     loads of item j+1 into registers; collide and store to global memory.
//
// Stage.  Each population plane k lands shifted by 8 c_y + 64 c_z slots in a
// plane of kSPlane = 72 + 512 + 72 slots, so the value cell t pulls in
// direction k sits at S[k][t - c_x]: one conflict-free shared load at a
// compile-time offset.  (The shifts reach 72 cells either way; every landing
// address stays 32-byte aligned.)  A z neighbour's layer continues its plane
// on the side the shift left free; the slots whose source lies in the other
// neighbours are overwritten after the landing.  Velocities: 512 own values,
// then the 6 x 64 values beyond the faces (a face without a neighbour repeats
// the cell beside it, the zero-gradient fallback of the WALE gradients).
//
// Why this split (measured on B200): an SM has to keep ~60-90 KB in flight to
// draw its share of HBM bandwidth, which bulk copies do and loader warps do
// not.  With one stage buffer the next landing could only start after the
// pulls and had to end before the next item, so the consumers waited for it:
// 905 us per coarse step of cube_3lvl; with two buffers, z layers by bulk copy
// and one barrier 766 us (sphere_ddf 291 -> 260 us, the thermal kernel built
// the same way 245 -> 222 us).  Of the 3176 out-of-block sources 968 lie in the
// z neighbours' contiguous layers and come by bulk copy; the consumers carry
// the other 2208 (5 registers a thread instead of 7), each found by one 8-byte
// table entry whose plane offset is formed once per launch.
//
// Hand-over uses mbarriers ("landed": bulk bytes plus the producer's arrival;
// "free": one arrival per consumer warp, both per buffer) and one named barrier
// of the consumers per item, after the out-of-block values are written.  A
// buffer lands again only after every consumer has pulled from it, so no
// barrier is needed before the writes.  Every mbarrier wait is bounded in time:
// a wait that runs out sets a bit in the fault word, and the warps give up
// together (consumers through the same named barrier, the producer after its
// copies in flight have landed), so no thread is left at a barrier and the
// kernel always ends.  The staged values are the ones the one-CTA-per-block
// kernel pulls, and the cell update is the same code.
#pragma once
#include "stream_collide.cuh"

namespace ol {

constexpr int kWsProducers = 32;                   // 1 producer warp
constexpr int kWsThreads = BCELLS + kWsProducers;  // 544
// descriptor / neighbour-offset slots (item j uses j & 7): the producer fetches
// item j+1 before buffer j & 1 is free, while a consumer may still update j-3
constexpr int kWsRing = 8;
constexpr int kSPad = 72;                         // stage slots before cell 0 (and after 511)
constexpr int kSPlane = kSPad + BCELLS + kSPad;   // 656 floats = 2624 bytes

// The table that ol_staging_tables exports (kWsTableTotal words; the loader table
// below is made from it): the kHaloEntries
// out-of-block pulls in the order of the staging table (k | dir << 5 | source
// cell << 10 | destination cell << 19), the kWsVelEntries face-halo velocity
// entries (face dir | own cell beside the slot << 5), then per pull its stage
// slot k * kSPlane + kSPad + destination cell - c_x(k).
constexpr int kWsVelEntries = 6 * 64;
constexpr int kWsTableSize = kHaloEntries + kWsVelEntries;
constexpr int kWsSlotOffset = kWsTableSize;
constexpr int kWsTableTotal = kWsTableSize + kHaloEntries;
// The loader table in device memory: two words per pull, {source cell |
// k << 9, dir | stage slot << 5 | staging-table index << 20}; first the
// kWsInner pulls the consumers always carry, then the 2 x kWsZFace pulls from
// the -z and +z face neighbours (carried only where that neighbour is absent).
constexpr int kWsZFace = 484;
constexpr int kWsInner = kHaloEntries - 2 * kWsZFace;  // 2208
constexpr int kWsLoaderWords = 2 * kHaloEntries;
constexpr int kDirZlo = 4, kDirZhi = 22;

// Dynamic shared memory (bytes): two buffers, then the loader table.
constexpr int kWsVPlane = BCELLS + kWsVelEntries;             // 896 floats
constexpr int kWsS = 0;                                       // float [27][kSPlane]
constexpr int kWsV = kWsS + 27 * kSPlane * 4;                 // float [3][kWsVPlane]
constexpr int kWsSP = kWsV + 3 * kWsVPlane * 4;               // float [512]
constexpr int kWsWD = kWsSP + BCELLS * 4;                     // float [512]
constexpr int kWsOB = kWsWD + BCELLS * 4;                     // uint8 [512]
constexpr int kWsBuf = kWsOB + BCELLS;                        // 86,208
constexpr int kWsTab = 2 * kWsBuf;                            // uint2 [kHaloEntries]
constexpr int kWsBytes = kWsTab + kWsLoaderWords * 4;         // 197,824
static_assert(kWsV % 16 == 0 && (kWsVPlane * 4) % 16 == 0 && kWsSP % 16 == 0 && kWsOB % 16 == 0 &&
                  kWsBuf % 16 == 0 && (kSPlane * 4) % 32 == 0 && (kSPad * 4) % 32 == 0,
              "bulk-copy destinations stay 16-byte aligned");
constexpr int kWsHaloPerConsumer = (kWsInner + BCELLS - 1) / BCELLS;  // 5
// A wait that has not completed after this long (ns) is treated as lost.
constexpr unsigned long long kWsWaitNs = 2000000000ull;
// Bits of the fault word.
constexpr int kWsFaultConsumerWait = 1, kWsFaultLoaderWait = 2;

// Per-device loader table (built once; null on failure).
const uint32_t *ws_loader_device();

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("{ .reg .b64 st; mbarrier.arrive.shared::cta.b64 st, [%0]; }" ::"r"(
                   smem_addr(bar))
               : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; "
      "selp.u32 %0, 1, 0, p; }"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Wait for the completion of the phase of `bar` with parity `parity`,
// bounded by kWsWaitNs of wall time and 2^26 polls; false (and `code` set in
// *fault) when the bound runs out.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, int *fault, int code) {
  if (mbar_test(bar, parity)) return true;
  const unsigned long long t0 = global_ns();
  for (uint32_t i = 0; i < (1u << 26); ++i) {
    if (mbar_test(bar, parity)) return true;
    if ((i & 63) == 63 && global_ns() - t0 > kWsWaitNs) break;
  }
  if (fault) atomicOr(fault, code);
  return false;
}

// Barrier of the 512 consumer threads only (named barrier 1); returns whether
// all of them passed a non-zero predicate.
__device__ __forceinline__ bool consumer_sync_and(int pred) {
  int r;
  asm volatile(
      "{ .reg .pred p, q; setp.ne.s32 p, %1, 0; bar.red.and.pred q, 1, %2, p; "
      "selp.s32 %0, 1, 0, q; }"
      : "=r"(r)
      : "r"(pred), "n"(BCELLS)
      : "memory");
  return r != 0;
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }" ::"r"(
                   smem_addr(bar)),
               "r"(bytes)
               : "memory");
}
// TMA bulk copy global -> shared (no multicast), completion counted on bar.
__device__ __forceinline__ void bulk_copy(void *dst, const void *src, uint32_t bytes,
                                          uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}

// A loader table entry with the plane offset of this launch:
// {k * dstride + source cell (mod 2^32), dir | slot << 5 | index << 20}.
__host__ __device__ __forceinline__ uint2 ws_entry(uint2 e, int64_t dstride) {
  return make_uint2((e.x >> 9) * (uint32_t)dstride + (e.x & 511), e.y);
}
// The table into shared memory (by the consumers, while the producer starts the first copies).
__device__ __forceinline__ void ws_load_table(uint2 *tabs, const uint32_t *__restrict__ tab,
                                              int64_t dstride, int t) {
#pragma unroll
  for (int m = 0; m < (kHaloEntries + BCELLS - 1) / BCELLS; ++m) {
    const int i = t + BCELLS * m;
    if (i >= kHaloEntries) break;
    tabs[i] = ws_entry(__ldg((const uint2 *)tab + i), dstride);
  }
}
// Whether the 27 planes reach beyond 32-bit element offsets (over 159 M cells).
__host__ __device__ __forceinline__ bool ws_wide(int64_t dstride) { return 27 * dstride > 0xFFFFFFFFll; }
__host__ __device__ __forceinline__ int ws_slot(uint2 e) { return (e.y >> 5) & 0x7FFF; }
// Element offset of entry e's source in the neighbour block whose first cell is nb.
__host__ __device__ __forceinline__ int64_t ws_source(uint2 e, int nb, int64_t dstride, bool wide) {
  if (!wide) return (int64_t)(e.x + (uint32_t)nb);
  const int k = ws_slot(e) / kSPlane;
  return k * dstride + (uint32_t)(e.x - (uint32_t)k * (uint32_t)dstride) + nb;
}

// The z neighbours' layers of the 9 population planes that pull across that
// face, by lane 0..8 (-z) and 9..17 (+z), where the neighbour exists.
__device__ __forceinline__ void ws_copy_zlayers(const float *fin, int64_t dstride, const int *nb,
                                                int lane, float *S, uint64_t *bar) {
  if (lane >= 18) return;
  const bool hi = lane >= 9;
  const int base = nb[hi ? kDirZhi : kDirZlo];
  if (base < 0) return;
  // c_z = +1 pulls across the -z face from the neighbour's z = 7 layer
  const int k = hi ? lane - 9 : lane + 18;
  const int at = k * kSPlane + kSPad + 8 * cy_of(k) + (hi ? BCELLS - 64 : 0);
  bulk_copy(S + at, fin + (size_t)k * dstride + base + (hi ? 0 : BCELLS - 64), 256, bar);
}

// The producer warp's bulk copies of block b into a buffer (lane 0 announces
// the bytes, then arrives; the bytes complete the phase).
template <bool WALE>
__device__ __forceinline__ void ws_produce(const LevelDev &L, int b, const int *nb, int lane,
                                           unsigned char *buf, uint64_t *bar) {
  constexpr uint32_t kPlane = BCELLS * 4;
  const int64_t own0 = (L.block_offset + b) * BCELLS;
  const bool wd = L.sp.wall_model_active == 1 && L.wall_dist;
  const float *fin = (const float *)L.f_in;
  const uint32_t layers = 9 * 256 * ((nb[kDirZlo] >= 0) + (nb[kDirZhi] >= 0));
  const uint32_t bytes = 27 * kPlane + layers + (WALE ? 3 * kPlane + 6 * 256 : 0) + kPlane +
                         BCELLS + (wd ? kPlane : 0);
  if (lane == 0) mbar_expect_tx(bar, bytes);
  __syncwarp();
  float *const S = (float *)(buf + kWsS);
  float *const V = (float *)(buf + kWsV);
  if (lane < 27) {
    // plane k = lane shifted by 8 c_y + 64 c_z slots (a multiple of 8)
    bulk_copy(S + lane * kSPlane + kSPad + 8 * cy_of(lane) + 64 * cz_of(lane),
              fin + (size_t)lane * L.dstride + own0, kPlane, bar);
  } else if (lane < 30) {
    if (WALE)
      bulk_copy(V + (lane - 27) * kWsVPlane, L.vel_in + (size_t)(lane - 27) * L.dstride + own0,
                kPlane, bar);
  } else if (lane == 30) {
    bulk_copy(buf + kWsSP, L.sponge + own0, kPlane, bar);
  } else {
    bulk_copy(buf + kWsOB, L.obstacle + own0, BCELLS, bar);
    if (wd) bulk_copy(buf + kWsWD, L.wall_dist + own0, kPlane, bar);
  }
  ws_copy_zlayers(fin, L.dstride, nb, lane, S, bar);
  if (WALE && lane >= 18 && lane < 24) {
    // the velocities beyond the z faces (the own layer where there is no neighbour)
    const int c = (lane - 18) % 3;
    const bool hi = lane >= 21;
    const int base = nb[hi ? kDirZhi : kDirZlo];
    const int64_t src = base >= 0 ? (int64_t)base + (hi ? 0 : BCELLS - 64)
                                  : own0 + (hi ? BCELLS - 64 : 0);
    bulk_copy(V + c * kWsVPlane + BCELLS + (hi ? 320 : 256),
              L.vel_in + (size_t)c * L.dstride + src, 256, bar);
  }
}

// Out-of-block pull sources of consumer thread t (table entries t + 512 m; one
// per absent z face) into registers.
struct HaloRegs {
  float f[kWsHaloPerConsumer];
  float z[2];
};
__device__ __forceinline__ void ws_halo_load(const float *__restrict__ fin, int64_t dstride,
                                             bool wide, const float *__restrict__ ghost_row,
                                             const int *nb, int t, const uint2 *tabs,
                                             HaloRegs &h) {
#pragma unroll
  for (int m = 0; m < kWsHaloPerConsumer; ++m) {
    const int i = t + BCELLS * m;
    h.f[m] = 0.0f;
    if (i >= kWsInner) continue;
    const uint2 e = tabs[i];
    const int base = nb[e.y & 31];
    if (base >= 0) h.f[m] = __ldg(fin + ws_source(e, base, dstride, wide));
    else if (ghost_row) h.f[m] = __ldg(ghost_row + (e.y >> 20));
  }
  h.z[0] = h.z[1] = 0.0f;
  if (ghost_row && t < kWsZFace) {
    if (nb[kDirZlo] < 0) h.z[0] = __ldg(ghost_row + (tabs[kWsInner + t].y >> 20));
    if (nb[kDirZhi] < 0) h.z[1] = __ldg(ghost_row + (tabs[kWsInner + kWsZFace + t].y >> 20));
  }
}
// The same values into the stage.  bc: the block has absent neighbours and no
// ghost row, so the sources there are evaluated by `boundary(k, x, y, z)`.
template <class BC>
__device__ __forceinline__ void ws_halo_store(float *S, const int *nb, int t, const uint2 *tabs,
                                              const HaloRegs &h, bool bc, BC boundary) {
  auto eval = [&](uint2 e) {
    const int slot = ws_slot(e), k = slot / kSPlane;
    const int d = slot - k * kSPlane - kSPad + cx_of(k);
    return boundary(k, d & 7, (d >> 3) & 7, d >> 6);
  };
#pragma unroll
  for (int m = 0; m < kWsHaloPerConsumer; ++m) {
    const int i = t + BCELLS * m;
    if (i >= kWsInner) continue;
    const uint2 e = tabs[i];
    float v = h.f[m];
    if (bc && nb[e.y & 31] < 0) v = eval(e);
    S[ws_slot(e)] = v;
  }
  if (t < kWsZFace) {
    if (nb[kDirZlo] < 0) {
      const uint2 e = tabs[kWsInner + t];
      S[ws_slot(e)] = bc ? eval(e) : h.z[0];
    }
    if (nb[kDirZhi] < 0) {
      const uint2 e = tabs[kWsInner + kWsZFace + t];
      S[ws_slot(e)] = bc ? eval(e) : h.z[1];
    }
  }
}

// Velocities beyond the x and y faces: thread t < 256 holds those of cell
// t & 63 of face t >> 6 (-x, +x, -y, +y).
__device__ __forceinline__ void ws_vel_load(const LevelDev &L, int b, const int *nb, int t,
                                            float (&v)[3]) {
  if (t >= 256) return;
  const int face = t >> 6, q = t & 63;
  const bool yf = face >= 2, hi = face & 1;
  const int dir = yf ? (hi ? 16 : 10) : (hi ? 14 : 12);
  const int step = yf ? 56 : 7;  // across the block along the axis
  const int oc = (yf ? (q & 7) + 64 * (q >> 3) : 8 * q) + (hi ? step : 0);
  const int base = nb[dir];
  const int64_t src = base >= 0 ? (int64_t)base + oc + (hi ? -step : step)
                                : (L.block_offset + b) * BCELLS + oc;
#pragma unroll
  for (int c = 0; c < 3; ++c) v[c] = __ldg(L.vel_in + (size_t)c * L.dstride + src);
}
// WALE eddy viscosity of cell t from the staged velocities.
__device__ __forceinline__ float ws_wale(const float *V, int t, float c_wale) {
  const int x = t & 7, y = (t >> 3) & 7, z = t >> 6;
  const float *const H = V + BCELLS;
  const int yz = y + 8 * z, xz = x + 8 * z, xy = x + 8 * y;
  const float *const pe = x < 7 ? V + t + 1 : H + 64 + yz;
  const float *const pw = x > 0 ? V + t - 1 : H + yz;
  const float *const pn = y < 7 ? V + t + 8 : H + 192 + xz;
  const float *const ps = y > 0 ? V + t - 8 : H + 128 + xz;
  const float *const pt = z < 7 ? V + t + 64 : H + 320 + xy;
  const float *const pb = z > 0 ? V + t - 64 : H + 256 + xy;
  WaleVel w;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    w.e[c] = pe[c * kWsVPlane]; w.w[c] = pw[c * kWsVPlane];
    w.n[c] = pn[c * kWsVPlane]; w.s[c] = ps[c * kWsVPlane];
    w.t[c] = pt[c * kWsVPlane]; w.b[c] = pb[c * kWsVPlane];
  }
  return wale_from(w, c_wale);
}

// Both operators: the regularized-BGK update needs fewer registers than the
// cumulant one; its levels took 335 us per coarse step of a 2-level sphere of
// 32 cells with one CTA per block and 202 us here.
// LOW: a level (not a pool, whose items differ) with omega_3 = omega_4 = 1; the
// general update left out of the kernel's code saves instruction fetches (766 ->
// 758 us per coarse step of cube_3lvl).
template <int OP, bool WALE, bool BATCHED, bool LOW = false>
__global__ void __launch_bounds__(kWsThreads, 1)
    k_sc_ws(const __grid_constant__ LevelDev L0, const LevelDev *__restrict__ descs,
            const WorkItem *__restrict__ items, int n_items, const uint32_t *__restrict__ tab,
            int *fault) {
  extern __shared__ __align__(16) unsigned char ws_smem[];
  __shared__ __align__(16) LevelDev Ls[BATCHED ? kWsRing : 1];
  __shared__ int nbb[kWsRing][27];
  __shared__ int blk[kWsRing];
  __shared__ const float *grow[kWsRing];  // the item's ghost row (null: none)
  __shared__ int absent[kWsRing];         // some neighbour of the item is absent
  __shared__ __align__(8) uint64_t bars[5];
  uint64_t *const landed = &bars[0], *const lfree = &bars[2];
  uint64_t *const ready = &bars[4];  // items 0 and 1 are described
  uint2 *const tabs = (uint2 *)(ws_smem + kWsTab);
  const int t = threadIdx.x;
  const int n = BATCHED ? n_items : L0.n_blocks;
  const int first = blockIdx.x;
  const int cnt = first < n ? (n - 1 - first) / (int)gridDim.x + 1 : 0;
  // every descriptor of a pool has the pool's plane stride
  const int64_t dstride = BATCHED ? descs[items[first].desc].dstride : L0.dstride;
  const bool wide = ws_wide(dstride);
  if (t == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(landed + i, 1);            // the producer's expect_tx arrival + the bulk bytes
      mbar_init(lfree + i, BCELLS / 32);   // one arrival per consumer warp
    }
    mbar_init(ready, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  if (t >= BCELLS) {
    // ------------------------------------------------------------ producer
    const int lane = t - BCELLS;
    pdl_wait();  // f_in, vel_in: written by the launches before this one
    // descriptor and neighbour offsets of item p into ring slot p & 7
    auto fetch = [&](int p) {
      const int r = p & (kWsRing - 1);
      const int it = first + p * (int)gridDim.x;
      int b = it;
      if (BATCHED) {
        const WorkItem w = items[it];
        static_assert(sizeof(LevelDev) % 4 == 0, "descriptor copy");
        for (int q = lane; q < (int)(sizeof(LevelDev) / 4); q += 32)
          ((uint32_t *)&Ls[r])[q] = ((const uint32_t *)(descs + w.desc))[q];
        b = w.block;
        __syncwarp();
      }
      const LevelDev &L = BATCHED ? Ls[r] : L0;
      int nb = 1;
      if (lane < 27) {
        nb = L.nbr[b + L.nbr_stride * lane];
        nbb[r][lane] = nb > 0 ? (int)((L.block_offset + nb - 1) * BCELLS) : -1;
      }
      const bool miss = __any_sync(0xffffffffu, nb <= 0);
      if (lane == 0) {
        blk[r] = b;
        absent[r] = miss;
        grow[r] = miss ? ghost_row_of(L, b) : nullptr;
      }
      __syncwarp();
    };
    // item 0's and item 1's offsets are published with item 0's copies;
    // item j+1's with item j's, so consumers can load ahead
    fetch(0);
    if (cnt > 1) fetch(1);
    if (lane == 0) mbar_arrive(ready);
    int j = 0;
    for (; j < cnt; ++j) {
      const int r = j & (kWsRing - 1), bi = j & 1;
      if (j >= 1 && j + 1 < cnt) fetch(j + 1);
      // buffer bi is free once the consumers have pulled item j-2
      const bool ok =
          j < 2 || mbar_wait(lfree + bi, ((j - 2) >> 1) & 1, fault, kWsFaultLoaderWait);
      if (!__all_sync(0xffffffffu, ok)) break;
      if (j >= 2) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      ws_produce<WALE>(BATCHED ? Ls[r] : L0, blk[r], nbb[r], lane, ws_smem + bi * kWsBuf,
                       landed + bi);
    }
    // bulk copies still in flight (a loop left early) land before the CTA exits
    if (j < cnt)
      for (int i = j >= 2 ? j - 2 : 0; i < j; ++i)
        mbar_wait(landed + (i & 1), (i >> 1) & 1, nullptr, 0);
    return;
  }

  // -------------------------------------------------------------- consumers
  HaloRegs h;
  float hv[3] = {0.0f, 0.0f, 0.0f};
  auto load = [&](int p) {
    const int r = p & (kWsRing - 1);
    const LevelDev &L = BATCHED ? Ls[r] : L0;
    ws_halo_load((const float *)L.f_in, dstride, wide, grow[r], nbb[r], t, tabs, h);
    if (WALE) ws_vel_load(L, blk[r], nbb[r], t, hv);
  };
  // The prologue runs beside the first landing: the table, then item 0's
  // out-of-block loads as soon as it is described.  With both before or after
  // the landing a launch took 3 us more (8 steps of the 1024-block sphere 413
  // -> 381 us; per coarse step of cube_3lvl's 7 launches 758 -> 736 us).
  ws_load_table(tabs, tab, dstride, t);
  pdl_wait();
  consumer_sync_and(1);
  const bool described = mbar_wait(ready, 0, fault, kWsFaultConsumerWait);
  if (described) load(0);
  for (int j = 0; j < cnt; ++j) {
    const int r = j & (kWsRing - 1), bi = j & 1;
    unsigned char *const buf = ws_smem + bi * kWsBuf;
    float *const S = (float *)(buf + kWsS);
    float *const V = (float *)(buf + kWsV);
    const bool ok =
        described && mbar_wait(landed + bi, (j >> 1) & 1, fault, kWsFaultConsumerWait);
    const LevelDev &L = BATCHED ? Ls[r] : L0;
    const int *const nb = nbb[r];
    const int b = blk[r];
    CellAux aux;
    float spg = 0.0f;
    bool obs = false;
    if (ok) {
      ws_halo_store(S, nb, t, tabs, h, absent[r] && !grow[r], [&](int k, int x, int y, int z) {
        return pull_boundary<StoreF32>(L, k, b, x, y, z);
      });
      if (WALE && t < 256) {
#pragma unroll
        for (int c = 0; c < 3; ++c) V[c * kWsVPlane + BCELLS + t] = hv[c];
      }
      aux.wall_dist = ((const float *)(buf + kWsWD))[t];
      spg = ((const float *)(buf + kWsSP))[t];
      obs = buf[kWsOB + t] != 0;
    }
    if (!consumer_sync_and(ok)) break;  // the stage holds item j
    aux.nu_wale = WALE ? ws_wale(V, t, L.sp.c_wale) : 0.0f;
    float A[27];
#pragma unroll
    for (int k = 0; k < 27; ++k) A[k] = S[k * kSPlane + kSPad + t - cx_of(k)];
    // the buffer is read: order these shared-memory accesses before the bulk
    // copies of item j+2, then release it
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if ((t & 31) == 0) mbar_arrive(lfree + bi);
    // item j+1's out-of-block values, in flight while item j collides
    if (j + 1 < cnt) load(j + 1);
    collide_cell<OP, StoreF32, WALE, LOW, BATCHED ? pool_sums(OP, true) : kSumsShort>(
        L, nb, A, b, t, obs, spg, &aux);
  }
}

}  // namespace ol
