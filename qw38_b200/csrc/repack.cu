// One-time weight preparation: 144-byte llama.cpp-native Q4_K super-blocks -> the
// split-tile device layout every kernel of this library consumes.
//
// A 144-byte block is {fp16 d, fp16 dmin, 12 scale bytes, 128 quant bytes}; element
// 64c+l of the block is the low nibble of qs[32c+l], element 64c+32+l its high nibble
// (third_party/llama.cpp-q4k/reference.hpp:244-248,253-275).  A tile row keeps the 16
// metadata bytes as they are and stores element 2j in the low and 2j+1 in the high nibble
// of code byte j (src/format/pack.cpp:201-222).  Rows n..ceil8(n)-1 are written as zeros.
#include <cuda_bf16.h>

#include "common.cuh"
#include "launch.h"

namespace q4k {
namespace {

// One thread turns 32 quant bytes of a block (16 low-nibble, then 16 high-nibble pairs: 32 output bytes in place) at a time, two of
// them in flight, and every fourth thread copies the metadata, so a warp reads eight consecutive blocks of a row and writes eight
// whole 128-byte tile rows, 32 bytes per store.  Bound: HBM, 2 x 144 bytes per block.  Measured on 17408 x 5120 (50 MB): 19.1 us (one
// task per thread 19.6, four 20.3); repack and the decoding to bf16 behind it 58 us, 66 before, 229 with one byte per thread and
// one block per tile row.  Blocks that are not 16-byte aligned are gathered byte by byte (Wide = false).
template <bool Wide> __device__ __forceinline__ uint4 load_block16(const uint8_t* p) {
  if constexpr (Wide) {
    return __ldg(reinterpret_cast<const uint4*>(p));
  } else {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = p[4 * i] | (uint32_t(p[4 * i + 1]) << 8) | (uint32_t(p[4 * i + 2]) << 16) | (uint32_t(p[4 * i + 3]) << 24);
    return make_uint4(w[0], w[1], w[2], w[3]);
  }
}
// Nibble pairs of eight bytes whose low nibbles hold the values.
__device__ __forceinline__ uint32_t pair_nibbles(uint32_t a, uint32_t b) {
  a &= 0x0f0f0f0fu;
  b &= 0x0f0f0f0fu;
  return __byte_perm(a | (a >> 4), b | (b >> 4), 0x6420);
}

// 32 bytes in one store (the address is a multiple of 32).
__device__ __forceinline__ void store32(void* to, const uint32_t (&a)[4], const uint32_t (&b)[4]) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"l"(to), "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]) : "memory");
}

constexpr int kRepackTasks = 2;
template <bool Wide>
__global__ void __launch_bounds__(256) repack_blocks144_kernel(const uint8_t* __restrict__ blocks, uint32_t n, uint32_t padded_n,
                                                               uint32_t tiles_k, uint8_t* __restrict__ codes, uint8_t* __restrict__ meta,
                                                               bool codes32) {
  uint64_t const task0 = uint64_t(blockIdx.x) * (256 * kRepackTasks) + threadIdx.x, live = uint64_t(n) * tiles_k * 4,
                 tasks = uint64_t(padded_n) * tiles_k * 4;
  uint4 a[kRepackTasks], b[kRepackTasks], mv[kRepackTasks];
#pragma unroll
  for (int i = 0; i < kRepackTasks; ++i) {
    uint64_t const task = task0 + i * 256;
    uint32_t const c = uint32_t(task & 3);
    a[i] = b[i] = mv[i] = make_uint4(0u, 0u, 0u, 0u);
    if (task >= live) continue;
    const uint8_t* const src = blocks + (task >> 2) * 144;
    a[i] = load_block16<Wide>(src + 16 + 32 * c);
    b[i] = load_block16<Wide>(src + 32 + 32 * c);
    if (c == 0) mv[i] = load_block16<Wide>(src);
  }
#pragma unroll
  for (int i = 0; i < kRepackTasks; ++i) {
    uint64_t const task = task0 + i * 256, block = task >> 2;
    if (task >= tasks) break;
    uint32_t const row = uint32_t(block / tiles_k), kb = uint32_t(block % tiles_k), c = uint32_t(task & 3);
    uint32_t const lo[4] = {pair_nibbles(a[i].x, a[i].y), pair_nibbles(a[i].z, a[i].w), pair_nibbles(b[i].x, b[i].y), pair_nibbles(b[i].z, b[i].w)};
    uint32_t const hi[4] = {pair_nibbles(a[i].x >> 4, a[i].y >> 4), pair_nibbles(a[i].z >> 4, a[i].w >> 4),
                            pair_nibbles(b[i].x >> 4, b[i].y >> 4), pair_nibbles(b[i].z >> 4, b[i].w >> 4)};
    uint64_t const tr = tile_row(row, kb, tiles_k);
    uint8_t* const dst = codes + tr * 128 + 32 * c;
    if (codes32) store32(dst, lo, hi);
    else {
      reinterpret_cast<uint4*>(dst)[0] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
      reinterpret_cast<uint4*>(dst)[1] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    }
    if (c == 0) *reinterpret_cast<uint4*>(meta + tr * 16) = mv[i];
  }
}

// Admissibility of a resident split-tile weight, the Q4_K rows of format::validate_cuda_v0
// (src/format/unpack.cpp:156-226): a padded row (row >= n) holds zero codes and zero metadata; a live
// row's fp16 d and dmin are non-negative and finite.  The reference walks tile rows in index order,
// codes before metadata, and reports the first offence; here every tile row is checked by one thread
// and the smallest key (tile_row, stage, byte) wins an atomic minimum, which is the same offence.
// stage: 0 padded code byte, 1 padded metadata byte, 2 super-block scale.
__global__ void __launch_bounds__(256) validate_kernel(const uint8_t* __restrict__ codes, const uint8_t* __restrict__ meta,
                                                       uint32_t n, uint32_t tiles_k, uint64_t tile_rows,
                                                       unsigned long long* __restrict__ key) {
  uint64_t const tr = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (tr >= tile_rows) return;
  uint32_t const row = uint32_t((tr >> 3) / tiles_k) * 8 + uint32_t(tr & 7);
  uint4 const m = reinterpret_cast<const uint4*>(meta)[tr];
  unsigned long long found = ~0ull;
  if (row >= n) {
    uint32_t const mw[4] = {m.x, m.y, m.z, m.w};
    for (int w = 3; w >= 0; --w)
      if (mw[w]) found = (tr << 10) | (1u << 8) | uint32_t(4 * w + (__ffs(mw[w]) - 1) / 8);
    const uint4* c = reinterpret_cast<const uint4*>(codes) + tr * 8;
    for (int q = 7; q >= 0; --q) {
      uint4 const v = c[q];
      uint32_t const cw[4] = {v.x, v.y, v.z, v.w};
      for (int w = 3; w >= 0; --w)
        if (cw[w]) found = (tr << 10) | uint32_t(16 * q + 4 * w + (__ffs(cw[w]) - 1) / 8);
    }
  } else {
    uint32_t const d = m.x & 0xffffu, dmin = m.x >> 16;
    if ((dmin & 0x8000u) || (dmin & 0x7c00u) == 0x7c00u) found = (tr << 10) | (2u << 8) | 2u;
    if ((d & 0x8000u) || (d & 0x7c00u) == 0x7c00u) found = (tr << 10) | (2u << 8) | 0u;
  }
  if (found != ~0ull) atomicMin(key, found);
}

// Split tiles -> bf16 weights [n][k] row-major, the values of compiler::dequantize_to_bf16
// (src/compiler/quantization/reference.cpp:141-166): w = bf16_rne((d * sc) * q - dmin * mn) with three
// separately rounded fp32 operations.  A warp takes 2 * Pairs consecutive K tiles of one row: half a warp a tile, a lane eight
// code bytes and one 32-byte store, all loads issued before the first store, so that a row's output is written in runs of
// Pairs KiB.  The launch takes the Pairs that leaves the fewest idle tiles.
//
// Bound: HBM writes.  17408 x 5120 (50 MB in, 178 MB out; a memset of the latter alone takes 28.5 us): five pairs 42.2 us, two pairs
// 45, one pair, or one 16-byte store per code word as before, 47; through shared memory and bulk stores 41.4, but 1.7 slower behind a
// repack than with these evict-first stores.
template <int Pairs>
__global__ void __launch_bounds__(128) dequantize_bf16_kernel(const uint8_t* __restrict__ codes, const uint8_t* __restrict__ meta,
                                                              uint32_t n, uint32_t tiles_k, uint32_t chunks_k, bool wide,
                                                              uint16_t* __restrict__ out) {
  uint32_t const task = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  uint32_t const group = task / (8 * chunks_k), rem = task % (8 * chunks_k), r = rem & 7, kb0 = (rem >> 3) * (2 * Pairs) + (lane >> 4);
  uint32_t const c = lane & 15, g = c >> 1, row = group * 8 + r;
  if (row >= n) return;
  uint4 m[Pairs];
  uint2 w[Pairs];
#pragma unroll
  for (int t = 0; t < Pairs; ++t) {
    if (kb0 + 2 * t < tiles_k) {
      uint64_t const tr = (uint64_t(group) * tiles_k + kb0 + 2 * t) * 8 + r;
      m[t] = __ldg(reinterpret_cast<const uint4*>(meta) + tr);
      w[t] = __ldg(reinterpret_cast<const uint2*>(codes) + tr * 16 + c);
    }
  }
#pragma unroll
  for (int t = 0; t < Pairs; ++t) {
    if (kb0 + 2 * t >= tiles_k) break;
    ScaleMinWords const sm = decode_scale_min(m[t].y, m[t].z, m[t].w);
    uint32_t const sc = byte_of(g < 4 ? sm.sc_lo : sm.sc_hi, g & 3), mn = byte_of(g < 4 ? sm.mn_lo : sm.mn_hi, g & 3);
    float const step = __fmul_rn(fp16_bits_to_f32(m[t].x & 0xffffu), float(sc));
    float const offset = __fmul_rn(fp16_bits_to_f32(m[t].x >> 16), float(mn));
    uint32_t packed[2][4];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      // level -> float through the 2^23 bias (exact, and on the full-rate pipes); the pair is rounded
      // to bf16 by one conversion instruction (round to nearest even; values are finite)
      uint32_t const v = (i < 4 ? w[t].x : w[t].y) >> (8 * (i & 3));
      float const lo = __fsub_rn(__uint_as_float(0x4b000000u | (v & 15u)), 8388608.f);
      float const hi = __fsub_rn(__uint_as_float(0x4b000000u | ((v >> 4) & 15u)), 8388608.f);
      __nv_bfloat162 const pair = __floats2bfloat162_rn(__fsub_rn(__fmul_rn(step, lo), offset), __fsub_rn(__fmul_rn(step, hi), offset));
      packed[i >> 2][i & 3] = *reinterpret_cast<const uint32_t*>(&pair);
    }
    uint16_t* const to = out + (uint64_t(row) * tiles_k + kb0 + 2 * t) * 256 + 16 * c;
    uint32_t const(&a)[4] = packed[0];
    uint32_t const(&b)[4] = packed[1];
    if (wide)
      asm volatile("st.global.L1::no_allocate.L2::evict_first.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                   ::"l"(to), "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]) : "memory");
    else {
      __stcs(reinterpret_cast<uint4*>(to), make_uint4(a[0], a[1], a[2], a[3]));
      __stcs(reinterpret_cast<uint4*>(to) + 1, make_uint4(b[0], b[1], b[2], b[3]));
    }
  }
}

// Split tiles -> the logical form of format::unpack_cuda_v0 (src/format/unpack.cpp:262-380): int8 levels
// [n][k] and the 16 metadata bytes per super-block [n][k/256][16].  A block of eight warps takes one group of eight rows and
// kUnpackTiles consecutive K tiles; warp r owns row r.
constexpr int kUnpackTiles = 4;
__global__ void __launch_bounds__(256) unpack_logical_kernel(const uint8_t* __restrict__ codes, const uint8_t* __restrict__ meta,
                                                             uint32_t n, uint32_t tiles_k, uint32_t chunks_k,
                                                             int8_t* __restrict__ out_codes, uint8_t* __restrict__ out_meta) {
  uint32_t const group = blockIdx.x / chunks_k, kb0 = (blockIdx.x % chunks_k) * kUnpackTiles;
  uint32_t const r = threadIdx.x >> 5, c = threadIdx.x & 31;
  uint32_t const row = group * 8 + r;
  if (row >= n) return;
  auto spread = [](uint32_t n4) { return (n4 & 15u) | ((n4 & 0xf0u) << 4) | ((n4 & 0xf00u) << 8) | ((n4 & 0xf000u) << 12); };
#pragma unroll
  for (int t = 0; t < kUnpackTiles; ++t) {
    if (kb0 + t >= tiles_k) break;
    uint64_t const tr = (uint64_t(group) * tiles_k + kb0 + t) * 8 + r;
    uint32_t const w = __ldg(reinterpret_cast<const uint32_t*>(codes) + tr * 32 + c);
    uint64_t const block = uint64_t(row) * tiles_k + kb0 + t;
    *reinterpret_cast<uint2*>(out_codes + block * 256 + 8 * c) = make_uint2(spread(w & 0xffffu), spread(w >> 16));
    if (c < 4) reinterpret_cast<uint32_t*>(out_meta + block * 16)[c] = __ldg(reinterpret_cast<const uint32_t*>(meta + tr * 16) + c);
  }
}

// verdict[1] holds the winning key on entry; rewrites verdict as {kind, byte offset in its span}.
__global__ void validate_verdict_kernel(unsigned long long* verdict) {
  unsigned long long const key = verdict[1];
  if (key == ~0ull) {
    verdict[0] = 0;
    verdict[1] = 0;
    return;
  }
  unsigned long long const tr = key >> 10, stage = (key >> 8) & 3u, byte = key & 0xffu;
  verdict[0] = stage + 1;
  verdict[1] = stage == 0 ? tr * 128 + byte : tr * 16 + byte;
}

}  // namespace

cudaError_t launch_validate_weight(const uint8_t* codes, const uint8_t* meta, uint32_t n, uint32_t k, uint64_t* verdict,
                                   cudaStream_t stream) {
  uint32_t const tiles_k = k / 256;
  uint64_t const tile_rows = uint64_t((n + 7) / 8 * 8) * tiles_k;
  auto* v = reinterpret_cast<unsigned long long*>(verdict);
  cudaError_t st = cudaMemsetAsync(v, 0xff, 16, stream);
  if (st != cudaSuccess) return st;
  validate_kernel<<<unsigned((tile_rows + 255) / 256), 256, 0, stream>>>(codes, meta, n, tiles_k, tile_rows, v + 1);
  validate_verdict_kernel<<<1, 1, 0, stream>>>(v);
  return cudaGetLastError();
}

cudaError_t launch_dequantize_bf16(const uint8_t* codes, const uint8_t* meta, uint32_t n, uint32_t k, uint16_t* out,
                                   cudaStream_t stream) {
  uint32_t const tiles_k = k / 256;
  auto chunks = [&](uint32_t pairs) { return (tiles_k + 2 * pairs - 1) / (2 * pairs); };
  uint32_t pairs = 5;
  for (uint32_t p : {4u, 3u, 2u, 1u})
    if (chunks(p) * p < chunks(pairs) * pairs) pairs = p;
  uint64_t const blocks = uint64_t((n + 7) / 8) * 2 * chunks(pairs);
  if (blocks > 0x1fffffffull) return cudaErrorInvalidValue;  // task numbers are 32 bits wide
  auto const kernel = pairs == 5   ? dequantize_bf16_kernel<5>
                      : pairs == 4 ? dequantize_bf16_kernel<4>
                      : pairs == 3 ? dequantize_bf16_kernel<3>
                      : pairs == 2 ? dequantize_bf16_kernel<2>
                                   : dequantize_bf16_kernel<1>;
  kernel<<<unsigned(blocks), 128, 0, stream>>>(codes, meta, n, tiles_k, chunks(pairs), reinterpret_cast<uintptr_t>(out) % 32 == 0, out);
  return cudaGetLastError();
}

cudaError_t launch_unpack_logical(const uint8_t* codes, const uint8_t* meta, uint32_t n, uint32_t k, int8_t* out_codes,
                                  uint8_t* out_meta, cudaStream_t stream) {
  uint32_t const tiles_k = k / 256, chunks_k = (tiles_k + kUnpackTiles - 1) / kUnpackTiles;
  uint64_t const blocks = uint64_t((n + 7) / 8) * chunks_k;
  if (blocks > 0x7fffffffull) return cudaErrorInvalidValue;
  unpack_logical_kernel<<<unsigned(blocks), 256, 0, stream>>>(codes, meta, n, tiles_k, chunks_k, out_codes, out_meta);
  return cudaGetLastError();
}

cudaError_t launch_repack_blocks144(const uint8_t* blocks, uint32_t n, uint32_t k, uint8_t* codes,
                                    uint8_t* meta, cudaStream_t stream) {
  uint32_t const tiles_k = k / 256;
  uint32_t const padded_n = (n + 7) / 8 * 8;
  unsigned const grid = unsigned((uint64_t(padded_n) * tiles_k * 4 + 256 * kRepackTasks - 1) / (256 * kRepackTasks));
  bool const codes32 = reinterpret_cast<uintptr_t>(codes) % 32 == 0;
  if (reinterpret_cast<uintptr_t>(blocks) % 16 == 0)
    repack_blocks144_kernel<true><<<grid, 256, 0, stream>>>(blocks, n, padded_n, tiles_k, codes, meta, codes32);
  else
    repack_blocks144_kernel<false><<<grid, 256, 0, stream>>>(blocks, n, padded_n, tiles_k, codes, meta, codes32);
  return cudaGetLastError();
}

}  // namespace q4k
