// sm_100a kernels of the NUFFT CG-SENSE operator pipeline.
//
// Data layouts in HBM (internal; the C ABI converts at its edges):
//   grid panel    [G*G][4C] f16, row q1*G + q0 (q1-major), per row hi(2C) | res(2C),
//                 complex interleaved per coil (re, im)
//   sample panel  [M][4C] f16, same row format
//   grid          [G*G][C] c64, row q1*G + q0
//   z1 / w1       [G][N][C] c64 (one FFT axis done)
//   CG vectors    [N][N] c64 FP32, scalars FP64 (CgState)
// The reference's equivalents are the N16 panels of nufft_integrated_bench.cu:339-359 and
// the coil-major grids of nufft_custom_fft_forward_bench.cu:538-747; here every stage
// reads and writes contiguous slabs and the panel row carries hi and res together so one
// gather feeds both sparse MMAs.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <vector>
#include <cmath>

#include "fft.cuh"
#include "kernels.cuh"

namespace tsn {

using namespace dev;

// Programmatic dependent launch (the next kernel's CTAs start while this one drains, and wait
// in pdl_wait before they touch its results; every kernel launched so calls pdl_wait).
//
// Inside the solver's graph only the interpolation is launched so: a plain graph edge costs
// 0.65 us, and FFT stages that start early wait beside a kernel that leaves room on the SMs
// (10-iteration solves, plain / programmatic FFT stages: 256^2 x 8 coils 616 / 636 us, 128^2 x
// 4 coils 302 / 309 us). The column stage ahead of a forward interpolation and the interpolation
// ahead of an adjoint one call pdl_trigger after their own wait; the others (split_samples among
// them, ahead of a plain adjoint's interpolation) leave it to their end. Batched cases, whose kernels run side by side on
// slices of the GPU, launch everything plainly: early CTAs would wait beside the other cases'
// kernels (the 48-case batch measured 1191 recons/s with it, 1325-1390 without it).
//
// Direct calls launch every kernel so: a plain launch behind a running kernel costs about 2 us
// and rounds the period up to the next 2 us (kernels of 2.5 us follow each other at 5.1 us),
// a programmatic one 0.7 us.
//
// TSN_PDL=0 in the environment launches everything plainly (the results are the same bit for
// bit).
static bool pdl_enabled() {
  static const bool on = [] {
    const char* e = std::getenv("TSN_PDL");
    return !(e && e[0] == '0');
  }();
  return on;
}

template <typename... KArgs, typename... Args>
static void launch_k(void (*kernel)(KArgs...), int grid, int block, size_t smem, cudaStream_t s, bool programmatic,
                     Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(grid));
  cfg.blockDim = dim3(static_cast<unsigned>(block));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = programmatic && pdl_enabled() ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// ------------------------------------------------------------------------------------------
// Sparse interpolation: one warp per 16-row group, 2:4 tiles through mma.sp m16n8k32.
// Per tile the 32 gathered panel rows (hi and res together) are brought to shared memory
// with 16-byte cp.async through a per-warp ring, swizzled so ldmatrix.trans is
// conflict-free; dead (padding) columns are zero-filled and never read.
// Reference: nufft_gt_spmma_complex_fused_f16_f32 (nufft_spmma_bench.cu:402-663), which
// gathers B with 2-byte loads and reduces 4 warps through shared memory.
// ------------------------------------------------------------------------------------------
template <int CH>
__device__ __forceinline__ int chunk_swizzle(int ch, int row) {
  if constexpr (CH == 2 || CH == 6) return ch ^ ((row >> 2) & 1);
  else if constexpr (CH == 4) return ch ^ ((row >> 1) & 3);
  else if constexpr (CH == 8) return ch ^ (row & 7);
  else return ch;
}

constexpr int kInterpWarps = 4;

// Output row s (0..15) of a record: 24-bit little-endian fields; -1 for a pad row (live bit
// 16 + s of the record flags clear), so every one of the 2^24 row indices is addressable.
__device__ __forceinline__ int32_t record_row(const uint8_t* rows24, int32_t flags, int s) {
  const uint32_t* w = reinterpret_cast<const uint32_t*>(rows24);
  const int bit = 24 * s, off = bit & 31;
  const uint32_t lo = w[bit >> 5];
  const uint32_t hi = off > 8 ? w[(bit >> 5) + 1] : 0u;  // stays inside the 48-byte field
  const uint32_t v = __funnelshift_r(lo, hi, off) & 0xFFFFFFu;
  return ((static_cast<uint32_t>(flags) >> (kRecLiveShift + s)) & 1u) ? static_cast<int32_t>(v) : -1;
}

// Per-warp shared-memory rings: kRingRecords tile records (offsets, A, meta, rows) and
// kRingGathers stages of 32 gathered panel rows. Records are fetched three tiles ahead,
// gathers one (the gather needs the record's offsets), so a warp waits only on cp.async
// groups, never on a register load.  Warps are persistent: each streams a contiguous,
// tile-balanced run of work items and the pipeline runs across item boundaries.
// Measured on 10-iteration solves (us): four records 594 / 1009 (256^2 with 8 / 16 coils)
// against three records 625 / 1016, three gather stages 625 / 1209 (fewer warps fit), and
// everything but the gathered rows in registers instead of shared memory 615 / 1112.
constexpr int kRingRecords = 4, kRingGathers = 2;
__host__ __device__ constexpr int interp_smem(int rowh, int ncomp) {
  return kInterpWarps * (kRingRecords * record_bytes(ncomp) + kRingGathers * 32 * rowh * 2);
}
// CTAs that an SM's shared memory (228 KB, 1 KB reserved per CTA) holds; registers follow
__host__ __device__ constexpr int interp_ctas(int rowh, int ncomp) {
  return 228 * 1024 / (interp_smem(rowh, ncomp) + 1024) < 10 ? 228 * 1024 / (interp_smem(rowh, ncomp) + 1024) : 10;
}
// Writes one finished item: split chunks publish their accumulators and the last chunk of
// the group reduces all chunks in chunk order; whole groups and finishing chunks apply the
// epilogue.
template <int ROWH, int NCOMP, int NA, int EPI, bool CONJ, bool SUMC>
__device__ __forceinline__ void interp_finish_item(float (&acc)[NCOMP][NA][4], const InterpView& v,
                                                   const InterpOut& o, const RecordInfo& info, int lane,
                                                   const int32_t (&rows)[2], const float (&wrow)[2], float scale) {
  const int t = lane & 3;
  if (info.split >= 0) {
    const int split = info.split;
    const int chunk = info.chunk & 0xFFFF, nchunks = info.chunk >> 16;
    // partial sums [chunk slot][component][coil block][lane] float4
    float4* slots = reinterpret_cast<float4*>(v.partials) + static_cast<size_t>(info.first_slot) * kPartialFloats * 8 + lane;
    float4* mine = slots + chunk * kPartialFloats * 8;
#pragma unroll
    for (int c = 0; c < NCOMP; ++c)
#pragma unroll
      for (int a2 = 0; a2 < NA; ++a2)
        mine[(c * NA + a2) * 32] = make_float4(acc[c][a2][0], acc[c][a2][1], acc[c][a2][2], acc[c][a2][3]);
    __threadfence();
    __syncwarp();
    int prior = 0;
    if (lane == 0) prior = atomicAdd(&v.counters[split], 1);
    prior = __shfl_sync(0xFFFFFFFFu, prior, 0);
    if (prior != nchunks - 1) return;
    __threadfence();
    // The last chunk to arrive is the launch's critical path (a central grid cell has tens of
    // chunks): kBatch loads travel together, the sums stay in chunk order.
    constexpr int kBatch = 8;
#pragma unroll
    for (int c = 0; c < NCOMP; ++c)
#pragma unroll
      for (int a2 = 0; a2 < NA; ++a2) {
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4* src = slots + (c * NA + a2) * 32;
        for (int k0 = 0; k0 < nchunks; k0 += kBatch) {
          float4 t[kBatch];
#pragma unroll
          for (int k = 0; k < kBatch; ++k)
            t[k] = k0 + k < nchunks ? __ldcg(src + (k0 + k) * kPartialFloats * 8) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int k = 0; k < kBatch; ++k) {
            sum.x += t[k].x;
            sum.y += t[k].y;
            sum.z += t[k].z;
            sum.w += t[k].w;
          }
        }
        acc[c][a2][0] = sum.x;
        acc[c][a2][1] = sum.y;
        acc[c][a2][2] = sum.z;
        acc[c][a2][3] = sum.w;
      }
    if (lane == 0) v.counters[split] = 0;  // ready for the next launch
  }
  if constexpr (EPI == EPI_RAW) {
#pragma unroll
    for (int hr = 0; hr < 2; ++hr) {
      if (rows[hr] < 0) continue;
#pragma unroll
      for (int a2 = 0; a2 < NA; ++a2) {
        float2 val = make_float2(acc[0][a2][2 * hr] * scale, acc[0][a2][2 * hr + 1] * scale);
        *reinterpret_cast<float2*>(o.raw + static_cast<size_t>(rows[hr]) * ROWH + 8 * a2 + 2 * t) = val;
      }
    }
  } else {
    const int C = o.coils;
#pragma unroll
    for (int hr = 0; hr < 2; ++hr) {
      const int32_t row = rows[hr];
      if (row < 0) continue;
      const float w = scale * wrow[hr];
#pragma unroll
      for (int a2 = 0; a2 < NA; ++a2) {
        const int coil = 4 * a2 + t;
        float re = acc[0][a2][2 * hr], im = acc[0][a2][2 * hr + 1];
        if constexpr (NCOMP == 2 && SUMC) {  // real coefficients split into FP16 high + low parts
          re += acc[1][a2][2 * hr];
          im += acc[1][a2][2 * hr + 1];
        } else if constexpr (NCOMP == 2) {
          const float qre = acc[1][a2][2 * hr], qim = acc[1][a2][2 * hr + 1];
          if (CONJ) {
            re = re + qim;
            im = im - qre;
          } else {
            re = re - qim;
            im = im + qre;
          }
        }
        re *= w;
        im *= w;
        if constexpr (EPI == EPI_SAMPLES) {
          o.c64[static_cast<size_t>(coil) * o.rows + row] = make_float2(re, im);
        } else if constexpr (EPI == EPI_GRID) {
          o.c64[static_cast<size_t>(row) * C + coil] = make_float2(re, im);
        } else {
          uint32_t hw, rw;
          split_hi_res2(re, im, hw, rw);
          uint32_t* rowp = reinterpret_cast<uint32_t*>(o.panel + static_cast<size_t>(row) * ROWH);
          rowp[coil] = hw;
          rowp[C + coil] = rw;
        }
      }
    }
  }
}

// What bounds it: instruction issue and the latency of the chain record -> gather -> MMA; with
// both data streams left out a launch still takes three quarters of its time. So the record
// holds what a lane needs as the lane needs it (the offsets of its gathers in one shared
// load, A as MMA fragments) instead of column ids that were passed around by shuffles and
// tested for every 16-byte copy (209 warp instructions per tile). 10-iteration solves: 256^2
// with 8 coils 615 -> 594 us, with 16 coils 1210 -> 1009 us, 128^2 with 4 coils 343 -> 322 us.
template <int ROWH, bool SPLIT, int NCOMP, int EPI, bool CONJ, bool SUMC = false>
__global__ void __launch_bounds__(kInterpWarps * 32, interp_ctas(ROWH, NCOMP)) interp_mmasp_kernel(InterpView v, const __half* __restrict__ panel,
                                                                         InterpOut o) {
  constexpr int NR = kRingRecords, NG = kRingGathers;
  constexpr int kRecAhead = NR - 1, kGatherAhead = NG - 1;
  constexpr int BYTES = ROWH * 2;
  constexpr int CH = BYTES / 16;
  constexpr int LPR = gather_lanes(ROWH);  // lanes sharing a row
  constexpr int NOFF = LPR;                // rows per lane: 32 / (32 / LPR)
  constexpr int NSUB = CH / LPR;           // chunks of each row per lane
  constexpr int NB = ROWH / 8;
  constexpr int NA = SPLIT ? NB / 2 : NB;
  constexpr int NACC = NCOMP * NA * 4;
  constexpr int INFO = 128 + 576 * NCOMP;         // RecordInfo offset in the record
  constexpr int REC = record_bytes(NCOMP);        // record bytes (all staged)
  constexpr int STAGE = 32 * BYTES;
  static_assert(NACC <= kPartialFloats, "partials slot too small");
  static_assert(REC % 16 == 0 && STAGE % 128 == 0, "16-byte records, aligned stages");
  static_assert(kGatherAhead >= 1 && kRecAhead > kGatherAhead, "ring arithmetic");
  extern __shared__ __align__(128) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wid = blockIdx.x * kInterpWarps + warp;
  if (wid >= v.n_warps) return;
  const int2 range = v.warp_ranges[wid];
  const int n = range.y - range.x;
  const uint8_t* rec_src = v.records + static_cast<size_t>(range.x) * REC + 16 * lane;
  const int g = lane >> 2;
  float scale = o.scale_mul;
  // records are plan data: their first copies stream in while the preceding kernel drains;
  // the panel, the scale and every output wait for it
  bool dep_ready = false;
  auto wait_dep = [&]() {
    if (dep_ready) return;
    pdl_wait();
    pdl_trigger();
    dep_ready = true;
    if (o.scale_ptr) {
      const float sp = *o.scale_ptr;
      scale *= o.scale_inv ? 1.0f / sp : sp;
    }
  };
  float wrow[2] = {1.f, 1.f};  // density of the open item's rows (EPI_PANEL)

  float acc[NCOMP][NA][4];
#pragma unroll
  for (int c = 0; c < NCOMP; ++c)
#pragma unroll
    for (int a = 0; a < NA; ++a)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[c][a][i] = 0.f;

  // gather stages of all warps first (128-byte aligned), then the records
  const uint8_t* rec_ring = smem + kInterpWarps * NG * STAGE + warp * NR * REC;
  const uint32_t gat_ring = smem_u32(smem + warp * NG * STAGE);
  // This lane's source chunk and its swizzled place in stage 0: row i of a lane lies
  // i * (32 / LPR) rows further with the same swizzle, but for 128-byte rows, where odd rows
  // flip chunk bit 2.
  const uint8_t* pb = reinterpret_cast<const uint8_t*>(panel) + (lane % LPR) * 16;
  const uint32_t dst0 =
      gat_ring + static_cast<uint32_t>((lane / LPR) * BYTES + chunk_swizzle<CH>(lane % LPR, lane / LPR) * 16);
  // this lane's ldmatrix row in stage 0; chunk nb flips address bits (the stages are aligned)
  const uint32_t ldm0 = gat_ring + static_cast<uint32_t>(lane * BYTES + chunk_swizzle<CH>(0, lane) * 16);
  auto ldm = [&](int nb) {
    return CH == 6 ? gat_ring + static_cast<uint32_t>(lane * BYTES + chunk_swizzle<CH>(nb, lane) * 16) : ldm0 ^ (nb * 16u);
  };
  // k-th record of this warp -> its ring slot
  auto issue_record = [&](int k, int slot) {
    if (k < n) {
      const uint32_t dst = smem_u32(rec_ring) + slot * REC + 16 * lane;
#pragma unroll
      for (int c0 = 0; c0 < REC / 16; c0 += 32)
        if (c0 + 32 <= REC / 16 || lane < REC / 16 - c0) cp_async16_u32(dst + 16 * c0, rec_src + 16 * c0);
      rec_src += REC;
    }
    cp_async_commit();  // empty groups keep the group arithmetic uniform
  };
  auto issue_gather = [&](int k, int slot, int stage) {
    if (k >= 0 && k < n) {
      wait_dep();
      const uint32_t* q = reinterpret_cast<const uint32_t*>(rec_ring + slot * REC) + (lane / LPR) * NOFF;
      uint32_t f[NOFF];
      if constexpr (NOFF == 2) {
        const uint2 t = *reinterpret_cast<const uint2*>(q);
        f[0] = t.x;
        f[1] = t.y;
      } else {
#pragma unroll
        for (int i = 0; i < NOFF; i += 4) {
          const uint4 t = *reinterpret_cast<const uint4*>(q + i);
          f[i] = t.x;
          f[i + 1] = t.y;
          f[i + 2] = t.z;
          f[i + 3] = t.w;
        }
      }
#pragma unroll
      for (int i = 0; i < NOFF; ++i) {
        const uint8_t* src = offset16(pb, f[i]);
#pragma unroll
        for (int u = 0; u < NSUB; ++u)
          cp_async16_or_zero((CH == 8 && (i & 1) ? dst0 ^ 64u : dst0) + stage * STAGE + i * (32 / LPR) * BYTES + u * LPR * 16,
                             src + u * LPR * 16, f[i] & kGatherDead);
      }
    }
    cp_async_commit();
  };
  auto compute = [&](int slot, int stage) {
    wait_dep();
    const uint8_t* st = rec_ring + slot * REC;
    const RecordInfo info = *reinterpret_cast<const RecordInfo*>(st + INFO);
    const uint8_t* trow = st + INFO + 16;
    if constexpr (EPI == EPI_PANEL) {  // density weights at the item's first tile
      if (o.density && (info.flags & kRecFirst)) {
        const int32_t r0 = record_row(trow, info.flags, g), r1 = record_row(trow, info.flags, g + 8);
        wrow[0] = r0 >= 0 ? __ldg(o.density + r0) : 1.f;
        wrow[1] = r1 >= 0 ? __ldg(o.density + r1) : 1.f;
      }
    }
    uint32_t a[NCOMP][4], meta[NCOMP];
#pragma unroll
    for (int c = 0; c < NCOMP; ++c) {
      const uint4 t = *reinterpret_cast<const uint4*>(st + 128 + 576 * c + 16 * lane);  // MMA fragment order
      a[c][0] = t.x;
      a[c][1] = t.y;
      a[c][2] = t.z;
      a[c][3] = t.w;
      meta[c] = reinterpret_cast<const uint32_t*>(st + 640 + 576 * c)[g * 2 + (lane & 1)];
    }
    // The tensor cores truncate as they add to an accumulator, so a tile starts from zero (low
    // parts of the panel before the high ones) and joins the item's sum in a rounding add:
    // over the thousands of samples of a central grid cell that halves the operator's noise.
#pragma unroll
    for (int na = 0; na < NA; ++na) {
      float t[NCOMP][4];
#pragma unroll
      for (int part = SPLIT ? 1 : 0; part >= 0; --part) {
        uint32_t b[4];
        ldmatrix_x4_trans_u32(b, ldm(na + part * NA) + stage * STAGE);
#pragma unroll
        for (int c = 0; c < NCOMP; ++c) {
          if (part == (SPLIT ? 1 : 0)) mma_sp_16832_zero(t[c], a[c], b, meta[c]);
          else mma_sp_16832(t[c], a[c], b, meta[c]);
        }
      }
#pragma unroll
      for (int c = 0; c < NCOMP; ++c)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[c][na][j] += t[c][j];
    }
    int32_t rows[2] = {-1, -1};
    if (info.flags & kRecLast) {
      rows[0] = record_row(trow, info.flags, g);
      rows[1] = record_row(trow, info.flags, g + 8);
    }
    __syncwarp();  // this slot and stage are refilled by the next iteration's copies
    if (info.flags & kRecLast) {  // last tile of its item
      interp_finish_item<ROWH, NCOMP, NA, EPI, CONJ, SUMC>(acc, v, o, info, lane, rows, wrow, scale);
#pragma unroll
      for (int c = 0; c < NCOMP; ++c)
#pragma unroll
        for (int a2 = 0; a2 < NA; ++a2)
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[c][a2][i] = 0.f;
    }
  };
  // Iterations k = -kRecAhead .. n-1, two commit groups each (empty when out of range):
  // rec(k + R) then gat(k + Ga), with R = kRecAhead, Ga = kGatherAhead.  Tile k lives in record
  // slot (k + R) % NR and gather stage (k + R) % NG; unrolling by a multiple of both makes
  // every address a constant.
  // After committing rec(k + R), the groups newer than rec(k + Ga) are gat(k + 2Ga - R)
  // and the 2(R - Ga) - 1 groups of the later iterations, so wait<2(R - Ga)> lands the
  // record the next gather reads; after committing gat(k + Ga), wait<2 Ga> lands gat(k).
  constexpr int UN = NR;
  static_assert(NR % NG == 0, "slots of both rings are constants");
  for (int k0 = -kRecAhead; k0 < n; k0 += UN) {
#pragma unroll
    for (int u = 0; u < UN; ++u) {
      const int k = k0 + u;
      if (k >= n) break;
      issue_record(k + kRecAhead, (u + kRecAhead) % NR);
      cp_async_wait<2 * (kRecAhead - kGatherAhead)>();
      __syncwarp();
      issue_gather(k + kGatherAhead, (u + kGatherAhead) % NR, (u + kGatherAhead) % NG);
      cp_async_wait<2 * kGatherAhead>();
      __syncwarp();
      if (k >= 0) compute(u % NR, u % NG);
    }
  }
  cp_async_wait<0>();
}

template <int ROWH, bool SPLIT, int NCOMP, int EPI, bool CONJ, bool SUMC = false>
static void launch_interp_t(const InterpView& v, const __half* panel, const InterpOut& o, cudaStream_t s) {
  const int blocks = (v.n_warps + kInterpWarps - 1) / kInterpWarps;
  constexpr size_t smem = interp_smem(ROWH, NCOMP);
  auto k = interp_mmasp_kernel<ROWH, SPLIT, NCOMP, EPI, CONJ, SUMC>;
  if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (blocks > 0) launch_k(k, blocks, kInterpWarps * 32, smem, s, v.programmatic != 0, v, panel, o);
}

template <int ROWH>
static void dispatch_epi(const InterpView& v, const __half* panel, int epi, bool conj, const InterpOut& o, cudaStream_t s) {
  if (v.sum_components) {  // FP16 high + low coefficient parts of a real pack
    if (epi == EPI_PANEL) launch_interp_t<ROWH, true, 2, EPI_PANEL, false, true>(v, panel, o, s);
    else if (epi == EPI_GRID) launch_interp_t<ROWH, true, 2, EPI_GRID, false, true>(v, panel, o, s);
    else launch_interp_t<ROWH, true, 2, EPI_SAMPLES, false, true>(v, panel, o, s);
    return;
  }
  if (v.ncomp == 2) {
    if (epi == EPI_SAMPLES) conj ? launch_interp_t<ROWH, true, 2, EPI_SAMPLES, true>(v, panel, o, s)
                                 : launch_interp_t<ROWH, true, 2, EPI_SAMPLES, false>(v, panel, o, s);
    else if (epi == EPI_PANEL) launch_interp_t<ROWH, true, 2, EPI_PANEL, false>(v, panel, o, s);
    else launch_interp_t<ROWH, true, 2, EPI_GRID, true>(v, panel, o, s);
  } else {
    if (epi == EPI_SAMPLES) launch_interp_t<ROWH, true, 1, EPI_SAMPLES, false>(v, panel, o, s);
    else if (epi == EPI_PANEL) launch_interp_t<ROWH, true, 1, EPI_PANEL, false>(v, panel, o, s);
    else launch_interp_t<ROWH, true, 1, EPI_GRID, false>(v, panel, o, s);
  }
}

static int sm_count();

template <int ROWH, int NCOMP>
static int resident_warps_t() {
  constexpr size_t smem = interp_smem(ROWH, NCOMP);
  auto k = interp_mmasp_kernel<ROWH, true, NCOMP, EPI_GRID, NCOMP == 2>;
  if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kInterpWarps * 32, smem);
  return std::max(1, per_sm) * kInterpWarps * sm_count();
}

int interp_resident_warps(int rowh, int ncomp) {
  switch (rowh * 4 + ncomp) {
    case 16 * 4 + 1: return resident_warps_t<16, 1>();
    case 16 * 4 + 2: return resident_warps_t<16, 2>();
    case 32 * 4 + 1: return resident_warps_t<32, 1>();
    case 32 * 4 + 2: return resident_warps_t<32, 2>();
    case 48 * 4 + 1: return resident_warps_t<48, 1>();
    case 48 * 4 + 2: return resident_warps_t<48, 2>();
    case 64 * 4 + 1: return resident_warps_t<64, 1>();
    default: return resident_warps_t<64, 2>();
  }
}

void launch_interp(const InterpView& v, const __half* panel, int rowh, bool split, int epi, bool conj,
                   const InterpOut& o, cudaStream_t s) {
  if (!split) {  // raw single-component product for the reference.bin gate (16 channels)
    launch_interp_t<16, false, 1, EPI_RAW, false>(v, panel, o, s);
    return;
  }
  switch (rowh) {
    case 16: dispatch_epi<16>(v, panel, epi, conj, o, s); break;
    case 32: dispatch_epi<32>(v, panel, epi, conj, o, s); break;
    case 48: dispatch_epi<48>(v, panel, epi, conj, o, s); break;
    case 64: dispatch_epi<64>(v, panel, epi, conj, o, s); break;
    default: break;
  }
}

// One warp per record, each lane an offset and 16-byte pieces of the rest. Bound by reading and
// writing the records once; a rebuild on the host cost the 256^2 x 8-coil view 11 ms a call.
__global__ void narrow_records_kernel(const uint8_t* __restrict__ records, int64_t tiles, int rowh, int ncomp,
                                      int component, uint8_t* __restrict__ out) {
  const int64_t t = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (t >= tiles) return;
  const uint8_t* src = records + t * record_bytes(ncomp);
  uint8_t* dst = out + t * record_bytes(1);
  // entry `lane` of 16-channel rows stands for tile column col, which lane group q of the view's
  // own rows holds as its entry j: col = q + j * (lane groups)
  const int col = gather_column(16, lane / gather_lanes(16), lane % gather_lanes(16));
  const int lanes = gather_lanes(rowh), groups = 32 / lanes;
  const uint32_t f = reinterpret_cast<const uint32_t*>(src)[col % groups * lanes + col / groups];
  reinterpret_cast<uint32_t*>(dst)[lane] =
      f == kGatherDead ? f : static_cast<uint32_t>(gather_offset(16, f / static_cast<uint32_t>(gather_offset(rowh, 1))));
  const uint4* comp = reinterpret_cast<const uint4*>(src + 128 + 576 * component);
  uint4* to = reinterpret_cast<uint4*>(dst + 128);
  to[lane] = comp[lane];                               // A
  if (lane < 4) to[32 + lane] = comp[32 + lane];       // metadata
  const uint4* info = reinterpret_cast<const uint4*>(src + 128 + 576 * ncomp);
  if (lane < kRecInfoBytes / 16) to[36 + lane] = info[lane];
}

void launch_narrow_records(const uint8_t* records, int64_t tiles, int rowh, int ncomp, int component, uint8_t* out,
                           cudaStream_t s) {
  if (tiles <= 0) return;
  narrow_records_kernel<<<static_cast<unsigned>((tiles + 7) / 8), 256, 0, s>>>(records, tiles, rowh, ncomp, component, out);
}

// ------------------------------------------------------------------------------------------
// Reductions
// ------------------------------------------------------------------------------------------
// n is even and v 16-byte aligned (images and coil k-space of 4 k coils)
__global__ void norm_partials_kernel(const float2* __restrict__ v, int64_t n, double* __restrict__ part) {
  __shared__ double scratch[32];
  pdl_wait();
  const float4* v4 = reinterpret_cast<const float4*>(v);
  double acc = 0.0;
#pragma unroll 4
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n / 2;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const float4 x = v4[i];
    acc += static_cast<double>(x.x) * x.x + static_cast<double>(x.y) * x.y + static_cast<double>(x.z) * x.z +
           static_cast<double>(x.w) * x.w;
  }
  const double t = block_sum(acc, scratch);
  if (threadIdx.x == 0) part[blockIdx.x] = t;
}

void launch_norm_partials(const float2* v, int64_t n, double* part, cudaStream_t s, bool pdl) {
  launch_k(norm_partials_kernel, kNormParts, 256, 0, s, pdl, v, n, part);
}

// Sum of nparts partials, identical (fixed tree) in every block. Call with all threads.
__device__ __forceinline__ double sum_partials(const double* part, int nparts, double* scratch) {
  double a = 0.0;
  for (int i = threadIdx.x; i < nparts; i += blockDim.x) a += part[i];
  return block_sum(a, scratch);
}

// Sums of four partial sections [nparts] spaced `stride` apart, in a fixed order. Each warp
// takes a strided piece of one section, so that a section's sum costs one tree of exchanges
// and not one per warp and section. `scratch` holds 32 doubles.
__device__ __forceinline__ double4 sum_partials4(const double* part, int nparts, int64_t stride, double* scratch) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int pieces = nw > 4 ? nw / 4 : 1;
  for (int t = warp; t < 4 * pieces; t += nw) {
    const double* sec = part + (t & 3) * stride;
    double a = 0.0;
#pragma unroll 4
    for (int i = (t >> 2) * 32 + lane; i < nparts; i += 32 * pieces) a += sec[i];
    a = warp_sum(a);
    if (lane == 0) scratch[t] = a;
  }
  __syncthreads();
  double4 r = make_double4(0.0, 0.0, 0.0, 0.0);
  for (int k = 0; k < pieces; ++k) {
    r.x += scratch[4 * k];
    r.y += scratch[4 * k + 1];
    r.z += scratch[4 * k + 2];
    r.w += scratch[4 * k + 3];
  }
  __syncthreads();
  return r;
}

// ------------------------------------------------------------------------------------------
// FFT endpoints: one CTA per line (image row, grid column) and coil group, see fft.cuh.
// ------------------------------------------------------------------------------------------
// Copy `bytes` (multiple of 16) from global to shared with 16-byte cp.async, all threads.
__device__ __forceinline__ void cp_async_bytes(void* dst, const void* src, int bytes) {
  uint8_t* d = static_cast<uint8_t*>(dst);
  const uint8_t* q = static_cast<const uint8_t*>(src);
  for (int i = threadIdx.x * 16; i < bytes; i += blockDim.x * 16) cp_async16(d + i, q + i);
}

// CTAs per SM that the register cap leaves room for: 1024 threads at 64 registers, and for the
// row stages, which hold a line's last butterflies and its epilogue, 768 at 80.
#define TSN_FFT_BOUNDS(T) __launch_bounds__((T), (1024 / (T)) > 0 ? 1024 / (T) : 1)
#define TSN_ROW_BOUNDS(T) __launch_bounds__((T), (T) <= 256 ? 768 / (T) : (T) <= 640 ? 2 : 1)

constexpr int kRowRed = 132;  // doubles of the row stages' static array (sums of partials)

// Lines of more than 256 threads (12 and 16 coils, large grids) leave the last inverse
// butterflies in shared memory instead of holding them in registers while the region changes
// hands: two CTAs of 480-640 threads then stay resident per SM, where one CTA per SM took three
// waves for 320 lines (320^2 x 12 coils normal operator 116 -> 109 us). The smaller lines hold
// them: their images are then read without bank conflicts.
template <class F>
__host__ __device__ constexpr bool rows_in_place() { return F::THREADS > 256; }

// Coils per CTA of the column and middle stages. 16 coils go in two CTAs of 8: a 64-byte run
// per row is still whole sectors, and the smaller CTA halves shared memory, so that several
// lines stay resident per SM at the largest grids. The row stages keep all coils of a line
// together (one image update, one coil combine).
__host__ __device__ constexpr int cols_coils(int C) { return C == 16 ? 8 : C; }

// k in [gap.x, gap.y)
__device__ __forceinline__ bool in_gap(int k, int2 gap) {
  return static_cast<unsigned>(k - gap.x) < static_cast<unsigned>(gap.y - gap.x);
}

// Row pitch (float2) of coil-map rows staged in shared memory for a coil-fastest reader:
// 16 bytes off a multiple of 128, so that 8 coils of two neighbouring pixels share no bank.
__host__ __device__ __forceinline__ int map_pitch(int N) { return (N + 15) / 16 * 16 + 2; }

// Forward rows (x-stage). Image row i0 -> z1[q1][i0][c] for all q1. Fuses the SENSE
// multiply, deapodization, power-of-two panel scaling, zero-padding and (CG) p = r + beta p.
//   mode 0 with smaps: the row of x; without: coil-image rows
//   mode 1 (CG): p = r + beta p, mode 2: p = r
//   mode 4 (CG, fused update): x += alpha p, r -= alpha A p, then p = r + beta p
// Mode 4 also finishes CG iteration iter-1, which then needs no cg_update launch: parts holds
// four sections [lines] of <p, Ap>, Re <r, Ap>, <Ap, Ap> and <r, r> from the inverse rows, so
// rho = <r, r> (a direct sum over the stored r, as the reference's rs_old), alpha = rho / pAp,
// and rho' = |r - alpha Ap|^2 = rho - 2 alpha Re <r, Ap> + alpha^2 <Ap, Ap> (FP64, a negative
// rounding residue clamped to 0).  The expansion restarts from the direct sum every
// iteration, so its rounding does not accumulate while rho falls.  Each row updates
// x += alpha p and r -= alpha Ap before p = r + beta p.
// Shared memory: FFT rows [G + R1][C] | the line's vectors [N]: row0 = x, r or (coil images)
// unused, later p times deapodization and panel scale; row1 = p; mode 4: row2 = A p, row3 = x |
// deapodization [N] float | (stage_maps) coil-map rows [C][pitch]. All are copied while the
// partial sums are reduced.
// Reference: fft512_rows4_shared16_pad_scale<true> (nufft_custom_fft_forward_bench.cu:1600-1844);
// the CG update of reference_sparse_solver.py:297-323.
template <int G, int C>
__global__ void TSN_ROW_BOUNDS((LineFft<G, C, false>::THREADS))
fwd_rows_kernel(FftArgs f, const float2* __restrict__ x, float2* __restrict__ z1, int mode, float2* __restrict__ p,
                float2* __restrict__ r, const double* __restrict__ parts, int nparts, CgState* __restrict__ st,
                int iter, float2* __restrict__ xs, const float2* __restrict__ ap, int stage_maps) {
  using F = LineFft<G, C, false>;
  extern __shared__ __align__(16) uint8_t sm[];
  const int N = f.N;
  const int lines = f.lines();
  const int64_t pix = f.pix();
  const bool has_beta = (mode == 1 && iter > 0) || mode == 4;
  float2* buf = reinterpret_cast<float2*>(sm);
  float2* row0 = buf + F::ROWS * C;
  float2* row1 = row0 + N;
  float2* row2 = row1 + (mode >= 1 ? N : 0);
  float2* row3 = row2 + (mode == 4 ? N : 0);
  float* srow = reinterpret_cast<float*>(row3 + (mode == 4 ? N : 0));
  float2* maps_s = reinterpret_cast<float2*>(srow + N);
  const int pitch = map_pitch(N);
  __shared__ double red[kRowRed];
  const int tid = threadIdx.x, c = tid % C;
  // part 1: rows no kernel of a solve writes (coil maps, deapodization); part 2: the rest
  const int i0 = blockIdx.x;
  const size_t off = static_cast<size_t>(i0) * N;
  auto issue = [&](int part) {
    if (part & 1) {
      cp_async_bytes(srow, f.scaling + off, N * 4);
      if (stage_maps)
        for (int cc = 0; cc < C; ++cc)
          cp_async_bytes(maps_s + cc * pitch, f.smaps + static_cast<size_t>(cc) * pix + off, N * 8);
    }
    if (part & 2) {
      if (mode >= 1) cp_async_bytes(row0, r + off, N * 8);
      else if (f.smaps) cp_async_bytes(row0, x + off, N * 8);
      if (has_beta) cp_async_bytes(row1, p + off, N * 8);
      if (mode == 4) {
        cp_async_bytes(row2, ap + off, N * 8);
        cp_async_bytes(row3, xs + off, N * 8);
      }
    }
    cp_async_commit();
  };
  if (f.maps_early) issue(1);
  pdl_wait();
  if (!f.maps_early) issue(1);
  issue(2);
  double total, alpha = 0.0, rho_prev = 0.0;
  if (mode == 4) {  // finish iteration iter-1 (the cg_update scalars)
    const double4 s3 = sum_partials4(parts, nparts, lines, red);
    const double rho = s3.w;  // |r_{iter-1}|^2 summed directly
    rho_prev = rho;
    const bool ok = isfinite(s3.x) && s3.x > 0.0;
    alpha = ok ? rho / s3.x : 0.0;
    const double rn = rho - 2.0 * alpha * s3.y + alpha * alpha * s3.z;
    total = rn < 0.0 ? 0.0 : rn;  // a negative rounding residue clamps to 0; NaN stays NaN
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      st->rho[iter - 1] = rho;  // the history keeps the direct sum
      st->pap[iter - 1] = s3.x;
      st->alpha[iter - 1] = alpha;
      // the iteration count stops at the first failing iteration, as the reference solver
      // stops there (reference_sparse_solver.py:281-293); the solve itself runs on with alpha 0
      const bool fin = isfinite(s3.x) && isfinite(rho) && isfinite(total);
      const bool prior_ok = st->curvature_ok && st->finite_ok;
      if (!ok) st->curvature_ok = 0;
      if (!fin) st->finite_ok = 0;
      if (prior_ok && ok && fin) st->completed = iter;
    }
  } else {
    total = sum_partials(parts, nparts, red);
  }
  float sigma;
  double beta = 0.0;
  if (mode == 0) {
    sigma = pow2_scale(total, static_cast<double>(pix) * (f.smaps ? 1 : C), kPanelTarget);
    if (blockIdx.x == 0 && threadIdx.x == 0) st->sigma_x = sigma;
  } else {
    sigma = pow2_scale(total, static_cast<double>(pix), kPanelTarget);
    // mode 4 divides by its own direct rho (block 0 rewrites st->rho[iter - 1] concurrently)
    const double rho_old = mode == 4 ? rho_prev : (iter > 0 ? st->rho[iter - 1] : 1.0);
    beta = (iter == 0 || mode == 2) ? 0.0 : total / fmax(rho_old, 1e-30);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      st->rho[iter] = total;
      st->beta[iter] = beta;
      st->sigma[iter] = sigma;
    }
  }
  const float scl = sigma / f.gs();
  const bool sense = f.smaps || mode >= 1;
  cp_async_wait<0>();
  __syncthreads();
  for (int i = tid; i < N; i += F::THREADS) {
    const float d = srow[i] * scl;
    if (!sense) {
      row0[i].x = d;
      continue;
    }
    float2 v = row0[i];
    if (has_beta) {
      const float2 pv = row1[i];
      if (mode == 4) {  // x += alpha p, r -= alpha Ap (the previous iteration's update)
        v = axpy64(-alpha, row2[i], v);
        r[off + i] = v;
        xs[off + i] = axpy64(alpha, pv, row3[i]);
      }
      v = axpy64(beta, pv, v);
    }
    if (mode >= 1) p[off + i] = v;
    row0[i] = cscale(v, d);
  }
  __syncthreads();
  const float2* msrc = stage_maps ? maps_s + c * pitch : (f.smaps ? f.smaps : x) + static_cast<size_t>(c) * pix + off;
  F::first(buf, f.tw, tid, [&](int n) {
    int i1 = n + f.shift;
    if (i1 >= G) i1 -= G;
    if (i1 >= N) return make_float2(0.f, 0.f);
    const float2 w = row0[i1];
    return sense ? cmul(w, msrc[i1]) : cscale(msrc[i1], w.x);
  });
  __syncthreads();
  if constexpr (F::R3 > 1) {
    F::middle(buf, f.tw, tid);
    __syncthreads();
  }
  // line i0 = (slab, row): z1 [slab][q][row][c] (one slab for images)
  float2* dst = z1 + (static_cast<size_t>(i0 / N) * G * N + i0 % N) * C + c;
  F::last(buf, tid, [&](int, int, int k, float2 v) {
    if (!in_gap(k, f.axis_gap)) dst[static_cast<size_t>(k) * N * C] = v;
  });
}

// Forward columns (y-stage): z1[q1][*][c] -> panel rows q1*G + q0, FP16 hi | res.
// Shared memory: FFT rows [G + R1][coils of the CTA].
// Reference: fft512_allcoils1_shared16_to_n16 (nufft_custom_fft_forward_bench.cu:538-747).
template <int G, int C>
__global__ void TSN_FFT_BOUNDS((LineFft<G, cols_coils(C), false>::THREADS))
fwd_cols_kernel(FftArgs f, const float2* __restrict__ z1, __half* __restrict__ panel) {
  constexpr int CC = cols_coils(C), GROUPS = C / CC;
  using F = LineFft<G, CC, false>;
  extern __shared__ __align__(16) uint8_t sm[];
  float2* buf = reinterpret_cast<float2*>(sm);
  const int N = f.N;
  pdl_wait();
  pdl_trigger();
  const int it = blockIdx.x;
  const int q1 = it / GROUPS, c = it % GROUPS * CC + threadIdx.x % CC;
  const int2 gap = f.cell_gap ? f.cell_gap[q1] : make_int2(0, 0);
  if (f.dims == 3 && gap.y - gap.x >= G) return;  // images: the loads do not wait for the gap's
  const float2* src = z1 + static_cast<size_t>(q1) * N * C + c;
  F::first(buf, f.tw, threadIdx.x, [&](int n) {
    int i0 = n + f.shift;
    if (i0 >= G) i0 -= G;
    return i0 < N ? src[i0 * C] : make_float2(0.f, 0.f);
  });
  __syncthreads();
  if constexpr (F::R3 > 1) {
    F::middle(buf, f.tw, threadIdx.x);
    __syncthreads();
  }
  uint32_t* dst = reinterpret_cast<uint32_t*>(panel + static_cast<size_t>(q1) * G * 4 * C) + c;
  F::last(buf, threadIdx.x, [&](int, int, int k, float2 v) {
    if (in_gap(k, gap)) return;
    uint32_t hw, rw;
    split_hi_res2(v.x, v.y, hw, rw);
    dst[k * 2 * C] = hw;
    dst[k * 2 * C + C] = rw;
  });
}

// Forward middle axis of a volume: z1[i0][q2][i1][c] -> z2[q2][q1][i0][c]. One item per line
// (q2, i0) with i0 fastest: neighbouring CTAs write neighbouring 8C-byte runs of z2.
// Shared memory: FFT rows [G + R1][coils of the CTA].
template <int G, int C>
__global__ void TSN_FFT_BOUNDS((LineFft<G, cols_coils(C), false>::THREADS))
fwd_mid_kernel(FftArgs f, const float2* __restrict__ z1, float2* __restrict__ z2) {
  constexpr int CC = cols_coils(C), GROUPS = C / CC;
  using F = LineFft<G, CC, false>;
  extern __shared__ __align__(16) uint8_t sm[];
  float2* buf = reinterpret_cast<float2*>(sm);
  const int N = f.N;
  pdl_wait();
  const int it = blockIdx.x;
  const int t = it / GROUPS, c = it % GROUPS * CC + threadIdx.x % CC;
  const int q2 = t / N, i0 = t - q2 * N;
  const int2 gap = f.line_gap ? f.line_gap[q2] : make_int2(0, 0);
  if (gap.y - gap.x >= G || in_gap(q2, f.axis_gap)) return;
  const float2* src = z1 + (static_cast<size_t>(i0) * G + q2) * N * C + c;
  F::first(buf, f.tw, threadIdx.x, [&](int n) {
    int i1 = n + f.shift;
    if (i1 >= G) i1 -= G;
    return i1 < N ? src[i1 * C] : make_float2(0.f, 0.f);
  });
  __syncthreads();
  if constexpr (F::R3 > 1) {
    F::middle(buf, f.tw, threadIdx.x);
    __syncthreads();
  }
  float2* dst = z2 + (static_cast<size_t>(q2) * G * N + i0) * C + c;
  F::last(buf, threadIdx.x, [&](int, int, int k, float2 v) {
    if (!in_gap(k, gap)) dst[static_cast<size_t>(k) * N * C] = v;
  });
}

// Measurement / adjoint input [C][M] -> sample panel [M][4C] with sigma_y and density.
// Reference: integrated_complex_to_split2_half_rows (nufft_integrated_bench.cu:339-359).
__global__ void split_samples_kernel(const float2* __restrict__ y, const float* __restrict__ density, int64_t m,
                                     int C, __half* __restrict__ panel, const double* __restrict__ parts, int nparts,
                                     CgState* __restrict__ st) {
  __shared__ double red[32];
  const int chunks = C / 4;
  const int64_t n = m * chunks, step = static_cast<int64_t>(gridDim.x) * blockDim.x;
  int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  float2 val[4];
  float w = 1.f;
  auto fetch = [&]() {
    const int64_t row = i / chunks;
    const int q = static_cast<int>(i - row * chunks);
#pragma unroll
    for (int k = 0; k < 4; ++k) val[k] = y[static_cast<size_t>(4 * q + k) * m + row];
    if (density) w = density[row];
  };
  pdl_wait();
  if (i < n) fetch();  // the first values travel while the scale is reduced
  const double total = sum_partials(parts, nparts, red);
  const float sigma = pow2_scale(total, static_cast<double>(m) * C, kPanelTarget);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->sigma_y = sigma;
    st->curvature_ok = 1;  // a solve starts here: reset the status words
    st->finite_ok = 1;
    st->completed = 0;
  }
  uint32_t* pu = reinterpret_cast<uint32_t*>(panel);
  while (i < n) {
    const int64_t row = i / chunks;
    const int q = static_cast<int>(i - row * chunks);
    const float ws = sigma * w;
    uint32_t hi[4], res[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) split_hi_res2(val[k].x * ws, val[k].y * ws, hi[k], res[k]);
    *reinterpret_cast<uint4*>(pu + row * 2 * C + 4 * q) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(pu + row * 2 * C + C + 4 * q) = make_uint4(res[0], res[1], res[2], res[3]);
    i += step;
    if (i < n) fetch();
  }
}

// Inverse columns: grid rows q1*G + [0,G) (all coils) -> w1[q1][i0][c], i0 < N (crop).
// Shared memory: FFT rows [G + R1][coils of the CTA].
// Reference: ifft512_rows8_regular_transposed (nufft_custom_fft_forward_bench.cu:1463-1515).
template <int G, int C>
__global__ void TSN_FFT_BOUNDS((LineFft<G, cols_coils(C), true>::THREADS))
inv_cols_kernel(FftArgs f, const float2* __restrict__ grid, float2* __restrict__ w1) {
  constexpr int CC = cols_coils(C), GROUPS = C / CC;
  using F = LineFft<G, CC, true>;
  extern __shared__ __align__(16) uint8_t sm[];
  float2* buf = reinterpret_cast<float2*>(sm);
  const int N = f.N;
  pdl_wait();
  const int it = blockIdx.x;
  const int q1 = it / GROUPS, c = it % GROUPS * CC + threadIdx.x % CC;
  // images read the unused cells' zeros: a load of the gap ahead of the line's own costs more
  const int2 gap = f.dims == 3 && f.cell_gap ? f.cell_gap[q1] : make_int2(0, 0);
  // a line that the next stage takes as zero (q1 = q2 G + q1 of volumes)
  if (f.dims == 3 ? (f.line_gap && in_gap(q1 % G, f.line_gap[q1 / G])) || in_gap(q1 / G, f.axis_gap)
                  : in_gap(q1, f.axis_gap))
    return;
  const float2* src = grid + static_cast<size_t>(q1) * G * C + c;
  F::first(buf, f.tw, threadIdx.x, [&](int n) { return in_gap(n, gap) ? make_float2(0.f, 0.f) : src[n * C]; });
  __syncthreads();
  if constexpr (F::R3 > 1) {
    F::middle(buf, f.tw, threadIdx.x);
    __syncthreads();
  }
  float2* dst = w1 + static_cast<size_t>(q1) * N * C + c;
  F::last(buf, threadIdx.x, [&](int, int, int k, float2 v) {
    int i0 = k + f.shift;
    if (i0 >= G) i0 -= G;
    if (i0 < N) dst[i0 * C] = v;
  });
}

// Inverse middle axis of a volume: z2[q2][q1][i0][c] -> z1[q2][i0][i1][c], i1 < N (crop).
// One item per line (q2, i0), i0 fastest: neighbouring CTAs read neighbouring 8C-byte runs.
// Shared memory: FFT rows [G + R1][coils of the CTA].
template <int G, int C>
__global__ void TSN_FFT_BOUNDS((LineFft<G, cols_coils(C), true>::THREADS))
inv_mid_kernel(FftArgs f, const float2* __restrict__ z2, float2* __restrict__ z1) {
  constexpr int CC = cols_coils(C), GROUPS = C / CC;
  using F = LineFft<G, CC, true>;
  extern __shared__ __align__(16) uint8_t sm[];
  float2* buf = reinterpret_cast<float2*>(sm);
  const int N = f.N;
  pdl_wait();
  const int it = blockIdx.x;
  const int t = it / GROUPS, c = it % GROUPS * CC + threadIdx.x % CC;
  const int q2 = t / N, i0 = t - q2 * N;
  if (in_gap(q2, f.axis_gap)) return;
  const int2 gap = f.line_gap ? f.line_gap[q2] : make_int2(0, 0);
  const float2* src = z2 + (static_cast<size_t>(q2) * G * N + i0) * C + c;
  F::first(buf, f.tw, threadIdx.x, [&](int n) {
    return in_gap(n, gap) ? make_float2(0.f, 0.f) : src[static_cast<size_t>(n) * N * C];
  });
  __syncthreads();
  if constexpr (F::R3 > 1) {
    F::middle(buf, f.tw, threadIdx.x);
    __syncthreads();
  }
  float2* dst = z1 + static_cast<size_t>(t) * N * C + c;
  F::last(buf, threadIdx.x, [&](int, int, int k, float2 v) {
    int i1 = k + f.shift;
    if (i1 >= G) i1 -= G;
    if (i1 < N) dst[i1 * C] = v;
  });
}

// Inverse rows + crop + deapodization + SENSE coil combine (+ CG epilogues).
// Shared memory: FFT rows [G + R1][C], then (rows_in_place: permuted) the coil images [N][C+1]
// in their place |
// (epi_smem) the epilogue inputs of the row, copied while the line is transformed: maps
// [C][N] (with smaps), p row [N] (modes 2, 3, 5), r or b row [N] (modes 2 with r, 3), scaling
// row [N] float. Without epi_smem the epilogue reads them from global memory.
// Mode 2 with r given also writes Re <r, Ap>, <Ap, Ap> and <r, r> per line into
// parts[lines + i0], parts[2 lines + i0] and parts[3 lines + i0], for the next forward rows to
// finish the CG update (mode 4 there).
// Reference: ifft512_rows8_regular_crop_scale (nufft_custom_fft_forward_bench.cu:1517-1552)
// followed by sense_combine_scaled (nufft_fp16x2_cg_bench.cu:27-54).
template <int G, int C>
__global__ void TSN_ROW_BOUNDS((LineFft<G, C, true>::THREADS))
inv_rows_kernel(FftArgs f, const float2* __restrict__ w1, float2* __restrict__ out, int mode, float2* __restrict__ x,
                float2* __restrict__ r, const float2* __restrict__ p, double* __restrict__ parts,
                CgState* __restrict__ st, int iter, float inv_scale2, float lambda_scaled, int region, int epi_smem) {
  using F = LineFft<G, C, true>;
  extern __shared__ __align__(16) uint8_t sm[];
  const int N = f.N;
  const int lines = f.lines();
  const int64_t pix_n = f.pix();
  float2* buf = reinterpret_cast<float2*>(sm);
  float2* emaps = reinterpret_cast<float2*>(sm + region);
  float2* eprow = emaps + (f.smaps ? C * N : 0);
  float2* errow = eprow + (mode >= 2 ? N : 0);
  const float2* rsrc = mode == 2 ? r : mode == 3 ? x : nullptr;  // r, or the right-hand side b
  float* escale = reinterpret_cast<float*>(errow + (rsrc ? N : 0));
  __shared__ double red[kRowRed];
  const int tid = threadIdx.x, c = tid % C;
  // part 1: rows no kernel of a solve writes (coil maps, deapodization); part 2: the rest
  const int i0 = blockIdx.x;
  const size_t off = static_cast<size_t>(i0) * N;
  auto issue = [&](int part) {
    if (epi_smem && (part & 1)) {
      if (f.smaps)
        for (int cc = 0; cc < C; ++cc)
          cp_async_bytes(emaps + cc * N, f.smaps + static_cast<size_t>(cc) * pix_n + off, N * 8);
      cp_async_bytes(escale, f.scaling + off, N * 4);
    }
    if (epi_smem && (part & 2)) {
      if (mode >= 2) cp_async_bytes(eprow, p + off, N * 8);
      if (rsrc) cp_async_bytes(errow, rsrc + off, N * 8);
    }
    cp_async_commit();
  };
  issue(1);
  pdl_wait();
  issue(2);
  float factor;
  if (mode == 2) factor = f.gs() / st->sigma[iter] * inv_scale2;
  else if (mode == 3 || mode == 5) factor = f.gs() / st->sigma_x * inv_scale2;
  else factor = inv_scale2 / st->sigma_y;
  const float2* src = w1 + static_cast<size_t>(i0) * C + c;
  F::first(buf, f.tw, tid, [&](int n) {
    return in_gap(n, f.axis_gap) ? make_float2(0.f, 0.f) : src[static_cast<size_t>(n) * lines * C];
  });
  __syncthreads();
  if constexpr (F::R3 > 1) {
    F::middle(buf, f.tw, tid);
    __syncthreads();
  }
  float2* img_s = buf;
  if constexpr (rows_in_place<F>()) {
    F::last_in_place(buf, tid);
    cp_async_wait<0>();
  } else {
    float2 v[F::ITL][F::RL];
    F::last(buf, tid, [&](int i, int j, int, float2 val) { v[i][j] = val; });
    cp_async_wait<0>();
    __syncthreads();  // the FFT rows are read: the region becomes the coil images [N][C+1]
#pragma unroll
    for (int i = 0; i < F::ITL; ++i) {
      const int b = F::last_base(tid, i);
      if (b < 0) continue;
#pragma unroll
      for (int j = 0; j < F::RL; ++j) {
        int i1 = b + F::NL * j + f.shift;
        if (i1 >= G) i1 -= G;
        if (i1 < N) img_s[i1 * (C + 1) + c] = v[i][j];
      }
    }
  }
  __syncthreads();
  double dot = 0.0, dot_r = 0.0, dot_a = 0.0, dot_rr = 0.0;
  for (int i1 = tid; i1 < N; i1 += blockDim.x) {
    const size_t pix = static_cast<size_t>(i0) * N + i1;
    const float d = (epi_smem ? escale[i1] : f.scaling[pix]) * factor;
    const int k = i1 >= f.shift ? i1 - f.shift : i1 - f.shift + G;  // the pixel's grid position
    const float2* img = img_s + (rows_in_place<F>() ? F::out_row(k) * C : i1 * (C + 1));
    if (!f.smaps) {  // coil images out [C][N][N]
#pragma unroll
      for (int cc = 0; cc < C; ++cc) out[static_cast<size_t>(cc) * pix_n + pix] = cscale(img[cc], d);
      continue;
    }
    if (mode == 5 && x) {  // the coil images before the combine, [C][N][N]
#pragma unroll
      for (int cc = 0; cc < C; ++cc) x[static_cast<size_t>(cc) * pix_n + pix] = cscale(img[cc], d);
    }
    float2 acc = make_float2(0.f, 0.f);
#pragma unroll
    for (int cc = 0; cc < C; ++cc) {
      const float2 s = epi_smem ? emaps[cc * N + i1] : f.smaps[static_cast<size_t>(cc) * pix_n + pix];
      acc = cadd(acc, cmulc(img[cc], s));
    }
    acc = cscale(acc, d);
    if (mode == 0) {
      out[pix] = acc;
    } else if (mode == 1) {
      r[pix] = acc;
      x[pix] = make_float2(0.f, 0.f);
      dot += static_cast<double>(acc.x) * acc.x + static_cast<double>(acc.y) * acc.y;
    } else {
      const float2 pv = epi_smem ? eprow[i1] : p[pix];
      acc.x += lambda_scaled * pv.x;
      acc.y += lambda_scaled * pv.y;
      if (mode == 2 || mode == 5) {
        out[pix] = acc;
        dot += static_cast<double>(pv.x) * acc.x + static_cast<double>(pv.y) * acc.y;
        if (mode == 2 && r) {
          const float2 rv = epi_smem ? errow[i1] : r[pix];
          dot_r += static_cast<double>(rv.x) * acc.x + static_cast<double>(rv.y) * acc.y;
          dot_a += static_cast<double>(acc.x) * acc.x + static_cast<double>(acc.y) * acc.y;
          dot_rr += static_cast<double>(rv.x) * rv.x + static_cast<double>(rv.y) * rv.y;
        }
      } else {  // reliable residual r = b - M v (b read through x)
        const float2 bv = epi_smem ? errow[i1] : x[pix];
        const float2 rv = make_float2(bv.x - acc.x, bv.y - acc.y);
        out[pix] = rv;
        dot += static_cast<double>(rv.x) * rv.x + static_cast<double>(rv.y) * rv.y;
      }
    }
  }
  if (mode == 2 && r) {
    const double t = warp_sum4(dot, dot_r, dot_a, dot_rr);
    if ((tid & 7) == 0) red[(tid >> 3 & 3) * 32 + (tid >> 5)] = t;
    __syncthreads();
    if (tid < 4) {
      double total = 0.0;
      for (int w = 0; w < F::THREADS / 32; ++w) total += red[tid * 32 + w];
      parts[tid * static_cast<int64_t>(lines) + i0] = total;
    }
  } else if (mode != 0) {
    const double t = block_sum(dot, red);
    if (tid == 0) parts[i0] = t;
  }
}

constexpr int kCgRowPix = 4;  // pixels per thread of cg_update: rows up to 1024 pixels at 256 threads

__global__ void cg_update_kernel(int N, int nparts, int lines, float2* __restrict__ x, float2* __restrict__ r,
                                 const float2* __restrict__ p, const float2* __restrict__ ap,
                                 const double* __restrict__ pap_parts, double* __restrict__ rr_parts,
                                 CgState* __restrict__ st, int iter) {
  __shared__ double red[33];
  // the row's vectors stream in while the pAp partials are reduced (N <= kCgRowPix * blockDim)
  const int i0 = blockIdx.x;
  float2 pv[kCgRowPix], av[kCgRowPix], xv[kCgRowPix], rv[kCgRowPix];
#pragma unroll
  for (int j = 0; j < kCgRowPix; ++j) {
    const int i1 = threadIdx.x + j * blockDim.x;
    if (i1 < N) {
      const size_t pix = static_cast<size_t>(i0) * N + i1;
      pv[j] = p[pix];
      av[j] = ap[pix];
      xv[j] = x[pix];
      rv[j] = r[pix];
    }
  }
  // <p, Ap> and the direct <r, r> of the r this iteration started from (sections 0 and 3 of
  // the inverse rows' partials)
  const double pap = sum_partials(pap_parts, nparts, red);
  const double rho = sum_partials(pap_parts + 3 * static_cast<int64_t>(lines), nparts, red);
  const bool ok = isfinite(pap) && pap > 0.0;
  const double alpha = ok ? rho / pap : 0.0;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->rho[iter] = rho;
    st->pap[iter] = pap;
    st->alpha[iter] = alpha;
    const bool prior_ok = st->curvature_ok && st->finite_ok;  // completed stops at a failure
    if (!ok) st->curvature_ok = 0;
    if (!isfinite(pap)) st->finite_ok = 0;
    if (prior_ok && ok) st->completed = iter + 1;
  }
  double acc = 0.0;
#pragma unroll
  for (int j = 0; j < kCgRowPix; ++j) {
    const int i1 = threadIdx.x + j * blockDim.x;
    if (i1 >= N) continue;
    const size_t pix = static_cast<size_t>(i0) * N + i1;
    xv[j] = axpy64(alpha, pv[j], xv[j]);
    rv[j] = axpy64(-alpha, av[j], rv[j]);
    x[pix] = xv[j];
    r[pix] = rv[j];
    acc += static_cast<double>(rv[j].x) * rv[j].x + static_cast<double>(rv[j].y) * rv[j].y;
  }
  const double t = block_sum(acc, red);
  if (threadIdx.x == 0) rr_parts[i0] = t;
}

__global__ void cg_finish_kernel(int nparts, const double* __restrict__ rr_parts, CgState* __restrict__ st,
                                 int iters) {
  __shared__ double red[33];
  const double rho = sum_partials(rr_parts, nparts, red);
  if (threadIdx.x == 0) {
    st->rho[iters] = rho;
    if (!isfinite(rho)) {  // a non-finite last update: the last iteration did not complete
      if (st->curvature_ok && st->finite_ok && st->completed == iters) st->completed = iters - 1;
      st->finite_ok = 0;
    }
  }
}

// ------------------------------------------------------------------------------------------
// Launchers
// ------------------------------------------------------------------------------------------
static size_t align16(size_t b) { return (b + 15) & ~static_cast<size_t>(15); }

// Shared memory of the FFT rows of a line of C coils
template <int G, int C>
static size_t fft_rows_bytes() {
  return sizeof(float2) * static_cast<size_t>(LineFft<G, C, false>::ROWS) * C;
}
// The row stages stage their coil-map rows (and other epilogue rows) in shared memory while
// two CTAs still fit on an SM with them (half of its 228 KB, less the 1 KB that each CTA reserves
// and the kernel's static array); larger lines read them from global memory. Lines of 112-114 KB
// staged, one CTA per SM, and not, two of them: adjoint of 256^2 x 16 coils on 640 points 66.9 and
// 65.0 us, 6-iteration solve of 488^2 x 8 coils on 1024 points 945 and 919 us.
constexpr size_t kFftStageSmem = 228 * 1024 / 2 - 1024 - kRowRed * sizeof(double);

// Dynamic shared memory beyond the default 48 KB, of which the kernels' static arrays take up
// to 2 KB, has to be asked for.
template <class K>
static void ensure_smem(K k, size_t bytes) {
  if (bytes > 46 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
}

static int sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

#define TSN_G_SWITCH(G_, ...)                                  \
  switch (G_) {                                                \
    case 128: { constexpr int GG = 128; __VA_ARGS__; } break;  \
    case 256: { constexpr int GG = 256; __VA_ARGS__; } break;  \
    case 384: { constexpr int GG = 384; __VA_ARGS__; } break;  \
    case 512: { constexpr int GG = 512; __VA_ARGS__; } break;  \
    case 640: { constexpr int GG = 640; __VA_ARGS__; } break;  \
    case 1024: { constexpr int GG = 1024; __VA_ARGS__; } break; \
    default: break;                                            \
  }
// FFT stage instantiation per coil count (4, 8, 12, 16): the index arithmetic folds to
// constants
#define TSN_FFT_C(C_, ...)                                  \
  switch (C_) {                                             \
    case 4: { constexpr int CC = 4; __VA_ARGS__; } break;   \
    case 8: { constexpr int CC = 8; __VA_ARGS__; } break;   \
    case 12: { constexpr int CC = 12; __VA_ARGS__; } break; \
    case 16: { constexpr int CC = 16; __VA_ARGS__; } break; \
    default: break;                                         \
  }

void launch_fwd_rows(const FftArgs& f, const float2* x, float2* z1, int mode, float2* p, float2* r,
                     const double* partials, int nparts, CgState* st, int iter, cudaStream_t s, float2* xs,
                     const float2* ap) {
  TSN_G_SWITCH(f.G, TSN_FFT_C(f.C, {
    const int rows = mode == 4 ? 4 : mode >= 1 ? 2 : 1;
    const size_t base = fft_rows_bytes<GG, CC>() + (sizeof(float2) * rows + sizeof(float)) * static_cast<size_t>(f.N);
    const size_t maps = sizeof(float2) * static_cast<size_t>(CC) * map_pitch(f.N);
    const int stage = f.smaps && base + maps <= kFftStageSmem ? 1 : 0;
    const size_t sm = base + (stage ? maps : 0);
    constexpr int T = LineFft<GG, CC, false>::THREADS;
    auto k = fwd_rows_kernel<GG, CC>;
    ensure_smem(k, sm);
    launch_k(k, f.lines(), T, sm, s, f.pdl, f, x, z1, mode, p, r, partials, nparts, st,
             iter, xs, ap, stage);
  }));
}

void launch_fwd_cols(const FftArgs& f, const float2* z1, __half* panel, cudaStream_t s) {
  TSN_G_SWITCH(f.G, TSN_FFT_C(f.C, {
    constexpr int W = cols_coils(CC), T = LineFft<GG, W, false>::THREADS;
    const size_t sm = fft_rows_bytes<GG, W>();
    auto k = fwd_cols_kernel<GG, CC>;
    ensure_smem(k, sm);
    launch_k(k, f.gcols() * (CC / W), T, sm, s, f.pdl, f, z1, panel);
  }));
}

void launch_fwd_mid(const FftArgs& f, const float2* z1, float2* z2, cudaStream_t s) {
  TSN_G_SWITCH(f.G, TSN_FFT_C(f.C, {
    constexpr int W = cols_coils(CC), T = LineFft<GG, W, false>::THREADS;
    const size_t sm = fft_rows_bytes<GG, W>();
    auto k = fwd_mid_kernel<GG, CC>;
    ensure_smem(k, sm);
    launch_k(k, f.N * f.G * (CC / W), T, sm, s, f.pdl, f, z1, z2);
  }));
}

void launch_inv_mid(const FftArgs& f, const float2* z2, float2* z1, cudaStream_t s) {
  TSN_G_SWITCH(f.G, TSN_FFT_C(f.C, {
    constexpr int W = cols_coils(CC), T = LineFft<GG, W, true>::THREADS;
    const size_t sm = fft_rows_bytes<GG, W>();
    auto k = inv_mid_kernel<GG, CC>;
    ensure_smem(k, sm);
    launch_k(k, f.N * f.G * (CC / W), T, sm, s, f.pdl, f, z2, z1);
  }));
}

void launch_split_samples(const float2* y, const float* density, int64_t m, int c, __half* panel,
                          const double* partials, int nparts, CgState* st, cudaStream_t s, bool pdl) {
  const int64_t blocks = std::min<int64_t>((m * (c / 4) + 255) / 256, 8 * 148);
  launch_k(split_samples_kernel, static_cast<int>(std::max<int64_t>(blocks, 1)), 256, 0, s, pdl, y, density, m, c, panel,
           partials, nparts, st);
}

void launch_inv_cols(const FftArgs& f, const float2* grid, float2* w1, cudaStream_t s) {
  TSN_G_SWITCH(f.G, TSN_FFT_C(f.C, {
    constexpr int W = cols_coils(CC), T = LineFft<GG, W, true>::THREADS;
    const size_t sm = fft_rows_bytes<GG, W>();
    auto k = inv_cols_kernel<GG, CC>;
    ensure_smem(k, sm);
    launch_k(k, f.gcols() * (CC / W), T, sm, s, f.pdl, f, grid, w1);
  }));
}

void launch_inv_rows(const FftArgs& f, const float2* w1, float2* out, int mode, float2* x, float2* r, const float2* p,
                     double* partials, CgState* st, int iter, float inv_scale2, float lambda_scaled, cudaStream_t s) {
  TSN_G_SWITCH(f.G, TSN_FFT_C(f.C, {
    const size_t img = sizeof(float2) * static_cast<size_t>(f.N) * (CC + 1);
    const size_t region =
        rows_in_place<LineFft<GG, CC, true>>() ? fft_rows_bytes<GG, CC>() : align16(std::max(fft_rows_bytes<GG, CC>(), img));
    const int rows = (f.smaps ? CC : 0) + (mode >= 2 ? 1 : 0) + ((mode == 2 && r) || mode == 3 ? 1 : 0);
    const size_t epi = (sizeof(float2) * rows + sizeof(float)) * static_cast<size_t>(f.N);
    const int epi_smem = region + epi <= kFftStageSmem ? 1 : 0;
    const size_t sm = region + (epi_smem ? epi : 0);
    constexpr int T = LineFft<GG, CC, true>::THREADS;
    auto k = inv_rows_kernel<GG, CC>;
    ensure_smem(k, sm);
    launch_k(k, f.lines(), T, sm, s, f.pdl, f, w1, out, mode, x, r, p, partials, st, iter,
             inv_scale2, lambda_scaled, static_cast<int>(region), epi_smem);
  }));
}

void launch_cg_update(int N, int lines, int nparts, float2* x, float2* r, const float2* p, const float2* ap,
                      const double* pap_parts, double* rr_parts, CgState* st, int iter, cudaStream_t s) {
  cg_update_kernel<<<lines, 256, 0, s>>>(N, nparts, lines, x, r, p, ap, pap_parts, rr_parts, st, iter);
}

void launch_cg_finish(int nparts, const double* rr_parts, CgState* st, int iters, cudaStream_t s) {
  cg_finish_kernel<<<1, 256, 0, s>>>(nparts, rr_parts, st, iters);
}

// Block b sums section b (part + b * stride, n values) into its first value.
__global__ void reduce_partials_kernel(double* part, int n, int64_t stride) {
  __shared__ double red[33];
  pdl_wait();
  double* sec = part + blockIdx.x * stride;
  const double t = sum_partials(sec, n, red);  // every read lands before block_sum's first barrier
  if (threadIdx.x == 0) sec[0] = t;
}

void launch_reduce_partials(double* part, int n, cudaStream_t s, int sections, int64_t stride, bool pdl) {
  launch_k(reduce_partials_kernel, sections, 1024, 0, s, pdl, part, n, stride);
}

// FP64 partials of Re <a, b> over n complex values (grid-stride, one per block).
__global__ void rdot_partials_kernel(const float2* __restrict__ a, const float2* __restrict__ b, int64_t n,
                                     double* __restrict__ part) {
  __shared__ double scratch[33];
  pdl_wait();
  double acc = 0.0;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const float2 u = a[i], v = b[i];
    acc += static_cast<double>(u.x) * v.x + static_cast<double>(u.y) * v.y;
  }
  const double t = block_sum(acc, scratch);
  if (threadIdx.x == 0) part[blockIdx.x] = t;
}

// out[0] = the sum of n partials, in a fixed order (one block).
__global__ void sum_partials_to_kernel(const double* __restrict__ part, int n, double* __restrict__ out) {
  __shared__ double red[33];
  pdl_wait();
  const double t = sum_partials(part, n, red);
  if (threadIdx.x == 0) out[0] = t;
}

void launch_rdot(const float2* a, const float2* b, int64_t n, double* parts, double* out, cudaStream_t s, bool pdl) {
  launch_k(rdot_partials_kernel, kNormParts, 256, 0, s, pdl, a, b, n, parts);
  launch_k(sum_partials_to_kernel, 1, 256, 0, s, pdl, parts, kNormParts, out);
}

void launch_sum_partials_to(const double* parts, int n, double* out, cudaStream_t s, bool pdl) {
  launch_k(sum_partials_to_kernel, 1, 256, 0, s, pdl, parts, n, out);
}

// ---- reverse-mode CG step (the adjoint recurrences of one CG iteration) -------------------
// Forward step k: alpha = rho / gamma (gamma = Re <p, q>, q = M p), x' = x + alpha p,
// r' = r - alpha q, rho' = |r'|^2, beta = rho' / rho, p' = r' + beta p. Given the cotangents
// xb (of x', constant over the solve), rb (of r'), pb (of p'), rhob (of rho'), the step makes
//   rb2   = rb + pb + 2 rhob_n r'                 rhob_n = rhob + <pb, p> / rho
//   alphab = <xb, p> - <rb2, q>                   gammab = -alphab rho / gamma^2
//   qb    = -alpha rb2 + gammab p
//   pbk   = beta pb + alpha xb + gammab q         (pb of step k = pbk + M qb, added later)
//   rhobk = -<pb, p> rho' / rho^2 + alphab / gamma
// with <rb2, q> = <rb, q> + <pb, q> + 2 rhob_n <r', q>, so the five FP64 inner products come
// from one pass over the vectors before any of them changes.
constexpr int kCgbBlocks = kCgStepParts;  // 2 x 148 SMs

__global__ void cgb_dots_kernel(int64_t n, const float2* __restrict__ rb, const float2* __restrict__ pb,
                                const float2* __restrict__ p, const float2* __restrict__ q,
                                const float2* __restrict__ rn, const float2* __restrict__ xb,
                                double* __restrict__ parts) {
  __shared__ double red[165];
  pdl_wait();
  double d[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const float2 vpb = pb[i], vp = p[i], vq = q[i], vrb = rb[i], vrn = rn[i], vxb = xb[i];
    d[0] += static_cast<double>(vpb.x) * vp.x + static_cast<double>(vpb.y) * vp.y;
    d[1] += static_cast<double>(vrb.x) * vq.x + static_cast<double>(vrb.y) * vq.y;
    d[2] += static_cast<double>(vpb.x) * vq.x + static_cast<double>(vpb.y) * vq.y;
    d[3] += static_cast<double>(vrn.x) * vq.x + static_cast<double>(vrn.y) * vq.y;
    d[4] += static_cast<double>(vxb.x) * vp.x + static_cast<double>(vxb.y) * vp.y;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const double v = warp_sum(d[k]);
    if (lane == 0) red[33 * k + warp] = v;
  }
  __syncthreads();
  if (threadIdx.x < 5) {
    const int nw = (blockDim.x + 31) >> 5;
    double t = 0.0;
    for (int w = 0; w < nw; ++w) t += red[33 * threadIdx.x + w];
    parts[static_cast<int64_t>(threadIdx.x) * gridDim.x + blockIdx.x] = t;
  }
}

// a x + b y (+ c z) in FP64, one rounding per component
__device__ __forceinline__ float2 lincomb64(double a, float2 x, double b, float2 y, double c = 0.0,
                                            float2 z = make_float2(0.f, 0.f)) {
  return make_float2(static_cast<float>(a * x.x + b * y.x + c * z.x), static_cast<float>(a * x.y + b * y.y + c * z.y));
}

// sc (device FP64): [0] rho, [1] rho', [2] gamma, [3] rhob in; [4] rhob of step k out.
__global__ void cgb_update_kernel(int64_t n, int nparts, const double* __restrict__ parts,
                                  const double* __restrict__ rho_p, const double* __restrict__ rhon_p,
                                  const double* __restrict__ gamma_p, const double* __restrict__ rhob_p,
                                  double* __restrict__ rhob_out, float2* __restrict__ rb, float2* __restrict__ pb,
                                  const float2* __restrict__ p, const float2* __restrict__ q,
                                  const float2* __restrict__ rn, const float2* __restrict__ xb,
                                  float2* __restrict__ qb, double* __restrict__ qnorm_parts) {
  __shared__ double red[132];
  __shared__ double dl[5];
  pdl_wait();
  const double4 s4 = sum_partials4(parts, nparts, nparts, red);
  if (threadIdx.x == 0) {
    dl[0] = s4.x;
    dl[1] = s4.y;
    dl[2] = s4.z;
    dl[3] = s4.w;
  }
  const double d5 = sum_partials(parts + 4 * static_cast<int64_t>(nparts), nparts, red);
  __syncthreads();
  const double rho = *rho_p, rho_n = *rhon_p, gamma = *gamma_p, rhob = *rhob_p;
  const double alpha = rho / gamma, beta = rho_n / rho;
  const double betab = dl[0];
  const double rhob_n = rhob + betab / rho;
  const double rb2q = dl[1] + dl[2] + 2.0 * rhob_n * dl[3];
  const double alphab = d5 - rb2q;
  const double gammab = -alphab * rho / (gamma * gamma);
  if (blockIdx.x == 0 && threadIdx.x == 0) *rhob_out = -betab * rho_n / (rho * rho) + alphab / gamma;
  const double h = 2.0 * rhob_n;
  double acc = 0.0;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const float2 vrb = rb[i], vpb = pb[i], vp = p[i], vq = q[i], vrn = rn[i], vxb = xb[i];
    const float2 r2 = axpy64(h, vrn, make_float2(vrb.x + vpb.x, vrb.y + vpb.y));
    rb[i] = r2;
    const float2 qv = lincomb64(-alpha, r2, gammab, vp);
    qb[i] = qv;
    acc += static_cast<double>(qv.x) * qv.x + static_cast<double>(qv.y) * qv.y;
    pb[i] = lincomb64(beta, vpb, alpha, vxb, gammab, vq);
  }
  if (qnorm_parts) {  // |qb|^2 partials: the panel scale of the M qb that follows
    const double t = block_sum(acc, red);
    if (threadIdx.x == 0) qnorm_parts[blockIdx.x] = t;
  }
}

// pb += M qb; with sb given, sb[c] += conj(qb) t[c] + tb[c] conj(p) over `coils` planes of n.
__global__ void cgb_finish_kernel(int64_t n, int coils, float2* __restrict__ pb, const float2* __restrict__ mqb,
                                  const float2* __restrict__ qb, const float2* __restrict__ t,
                                  const float2* __restrict__ tb, const float2* __restrict__ p,
                                  float2* __restrict__ sb) {
  pdl_wait();
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const float2 vm = mqb[i];
    float2 vpb = pb[i];
    vpb.x += vm.x;
    vpb.y += vm.y;
    pb[i] = vpb;
    if (!sb) continue;
    const float2 vq = qb[i], vp = p[i];
    for (int c = 0; c < coils; ++c) {
      const size_t j = static_cast<size_t>(c) * n + i;
      const float2 vt = t[j], vtb = tb[j];
      float2 acc = sb[j];
      // conj(qb) t + tb conj(p)
      acc.x += vq.x * vt.x + vq.y * vt.y + vtb.x * vp.x + vtb.y * vp.y;
      acc.y += vq.x * vt.y - vq.y * vt.x + vtb.y * vp.x - vtb.x * vp.y;
      sb[j] = acc;
    }
  }
}

// ---- one forward CG step on caller-owned vectors (differentiable solves) ------------------
// alpha = rho / gamma; x' = x + alpha p (when x is given); r' = r - alpha q; rho' = |r'|^2
// (FP64, fixed order); p' = r' + (rho' / rho) p. Outputs are separate arrays.
__global__ void cgf_update_kernel(int64_t n, const double* __restrict__ rho_p, const double* __restrict__ gamma_p,
                                  const float2* __restrict__ x, const float2* __restrict__ p,
                                  const float2* __restrict__ r, const float2* __restrict__ q,
                                  float2* __restrict__ x_out, float2* __restrict__ r_out, double* __restrict__ parts) {
  __shared__ double red[33];
  pdl_wait();
  const double a = *rho_p / *gamma_p;
  double acc = 0.0;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const float2 vp = p[i], vr = r[i], vq = q[i];
    if (x) {
      const float2 vx = x[i];
      x_out[i] = axpy64(a, vp, vx);
    }
    const float2 rn = axpy64(-a, vq, vr);
    r_out[i] = rn;
    acc += static_cast<double>(rn.x) * rn.x + static_cast<double>(rn.y) * rn.y;
  }
  const double t = block_sum(acc, red);
  if (threadIdx.x == 0) parts[blockIdx.x] = t;
}

// With pnorm_parts given, also one FP64 partial of |p'|^2 per block (the panel scale of the
// next normal-operator application, which then needs no norm pass of its own).
__global__ void cgf_direction_kernel(int64_t n, int nparts, const double* __restrict__ parts,
                                     const double* __restrict__ rho_p, double* __restrict__ rho_out,
                                     const float2* __restrict__ p, const float2* __restrict__ r_new,
                                     float2* __restrict__ p_out, double* __restrict__ pnorm_parts) {
  __shared__ double red[33];
  pdl_wait();
  const double rho_n = sum_partials(parts, nparts, red);
  if (blockIdx.x == 0 && threadIdx.x == 0) *rho_out = rho_n;
  const double b = rho_n / *rho_p;
  double acc = 0.0;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const float2 vp = p[i], vr = r_new[i];
    const float2 pn = axpy64(b, vp, vr);
    p_out[i] = pn;
    acc += static_cast<double>(pn.x) * pn.x + static_cast<double>(pn.y) * pn.y;
  }
  if (pnorm_parts) {
    const double t = block_sum(acc, red);
    if (threadIdx.x == 0) pnorm_parts[blockIdx.x] = t;
  }
}

void launch_cg_step(int64_t n, double* parts, const double* rho, const double* gamma, const float2* x, const float2* p,
                    const float2* r, const float2* q, float2* x_out, float2* r_out, float2* p_out, double* rho_out,
                    double* p_norm_parts, cudaStream_t s, bool pdl) {
  launch_k(cgf_update_kernel, kCgbBlocks, 256, 0, s, pdl, n, rho, gamma, x, p, r, q, x_out, r_out, parts);
  launch_k(cgf_direction_kernel, kCgbBlocks, 256, 0, s, pdl, n, kCgbBlocks, parts, rho, rho_out, p, r_out, p_out,
           p_norm_parts);
}

void launch_cg_adjoint_step(int64_t n, double* parts, const double* rho, const double* rho_n, const double* gamma,
                            const double* rhob, double* rhob_out, float2* rb, float2* pb, const float2* p,
                            const float2* q, const float2* rn, const float2* xb, float2* qb, double* qb_norm_parts,
                            cudaStream_t s, bool pdl) {
  launch_k(cgb_dots_kernel, kCgbBlocks, 256, 0, s, pdl, n, rb, pb, p, q, rn, xb, parts);
  launch_k(cgb_update_kernel, kCgbBlocks, 256, 0, s, pdl, n, kCgbBlocks, parts, rho, rho_n, gamma, rhob, rhob_out, rb, pb,
           p, q, rn, xb, qb, qb_norm_parts);
}

void launch_cg_adjoint_finish(int64_t n, int coils, float2* pb, const float2* mqb, const float2* qb, const float2* t,
                              const float2* tb, const float2* p, float2* sb, cudaStream_t s, bool pdl) {
  launch_k(cgb_finish_kernel, kCgbBlocks, 256, 0, s, pdl, n, coils, pb, mqb, qb, t, tb, p, sb);
}

template <class T>
__global__ void gather_rows_kernel(const T* __restrict__ src, const int32_t* __restrict__ map, int64_t rows, int width,
                                   T* __restrict__ dst) {
  const int64_t n = rows * width;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t row = i / width, col = i - row * width;
    dst[i] = src[static_cast<int64_t>(map[row]) * width + col];
  }
}

void launch_gather_rows_f16(const __half* src, const int32_t* map, int64_t rows, int width, __half* dst, cudaStream_t s) {
  gather_rows_kernel<__half><<<592, 256, 0, s>>>(src, map, rows, width, dst);
}
void launch_gather_rows_f32(const float* src, const int32_t* map, int64_t rows, int width, float* dst, cudaStream_t s) {
  gather_rows_kernel<float><<<592, 256, 0, s>>>(src, map, rows, width, dst);
}

}  // namespace tsn
