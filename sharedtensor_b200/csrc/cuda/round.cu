// The sync-round kernel for sm_100a (see round.h for the protocol and ../core/codec.hpp for the arithmetic).
//
// A CTA holds two independent groups; a group is eight compute warps and one service warp and owns every n-th
// tile of the tensor.  The two kinds of warp talk through a few words of shared memory:
//
//   service warp  looks at several of the group's tiles at once, a lane per tile and ring: change mark, sequence flags of the
//                 in-rings, credits of the out-rings (all loads in flight together).  For every tile with something to
//                 do it writes a descriptor (tile, which frames arrived, which rings have room, what each link may
//                 hear) into a bank and arms the bank.  Tiles that all eight compute warps have finished are published
//                 together behind a fence (system scope, or device scope if all rings stay on this GPU): sequence flags
//                 to the receivers, credits to the senders.
//   compute warps walk through the bank, each on its own 512 elements of every tile.  A lane owns four 16-byte pieces
//                 128 elements apart, so that every access to values, mirrors and frames is a full, coalesced line:
//                 values and mirror are loaded straight into registers, the frames that arrived are decoded
//                 (reference 106-111, 124-127), what they say goes into the values as a reduction at the L2 (so an
//                 update another stream adds at the same moment is never overwritten) and into the mirror of its link,
//                 then values - mirror is quantised (reference 156-174), the mirror steps by what the codes say, and
//                 the codes go straight into the ring slots of the link's neighbours (peer stores over NVLink;
//                 reference src/sharedtensor.c:176-177, two socket writes).
//
// What bounds it.  Large tensors: HBM; a visit moves 12 to 18 bytes of values, mirror and frames per element.  Two groups
// keep 64 KB of loads in flight per SM and the next tile is on its way into the L2 meanwhile.  100 M elements on one link,
// each pass by itself with a wait for the GPU on both sides: 0.216 ms to send, 0.315 ms to receive and send, 0.295 ms to
// receive (0.324, 0.439 and 0.426 ms with tiles staged in shared memory by bulk copies for two groups of four warps, four
// windows instead of three and no overlap between them).
// Small tensors: latency.  A launch over one tile takes 6 us in the kernel, of which the look at the tile takes 2.3 and the
// tile 2; 811 tiles that are received and sent (sign frames) take 25 us when they are published at system scope and 17.5 at
// device scope (see the publication below).
//
// Nothing in here waits for another GPU.  The waits are on this group's own warps and copies, and every one is bounded.
// When one runs out, no visit is left half done: the warps go by the same answer, frames that are not in their stage are
// read from the ring, and a block whose maximum is not known is not spoken of while everything that arrived is taken in and
// acknowledged.  The group records an error in the status block, marks its tiles for another visit and leaves.
//
// Arithmetic is written with explicit round-to-nearest operations; block statistics are maxima (order does not
// matter), so codes, scales, mirrors and values are bit-identical to the host codec (../core/codec.cpp).
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "round.h"

#ifdef ST_ROUND_DEBUG
// progress marks in host memory, readable while a kernel is stuck (debug builds only)
#define ST_CRUMB(slot, code)                                                                  \
  do {                                                                                         \
    if (p.dbg != nullptr && lane == 0) {                                                       \
      *reinterpret_cast<volatile uint32_t*>(p.dbg + (blockIdx.x * 8 + (slot))) = uint32_t(code); \
    }                                                                                          \
  } while (0)
#else
#define ST_CRUMB(slot, code)
#endif

namespace st {

namespace {

constexpr int kComputeWarps = 8;                       // of a group
constexpr int kGroupThreads = (kComputeWarps + 1) * 32;  // and its service warp
constexpr int kBank = 32;                              // tiles a group has in hand at once
constexpr int kAhead = 6;                              // tiles in the compute warps' hands below which the service warp looks for more
constexpr int kPieces = 4;                             // 16-byte pieces of a lane
constexpr int kWarpElems = kPieces * 128;              // elements of a tile that one warp handles
static_assert(kComputeWarps * kWarpElems == kTile, "eight warps cover a tile");

// ----------------------------------------------------------------------------------------------
// small PTX wrappers
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t ld_acquire_sys(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_relaxed_sys(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_sys(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// this GPU's own bookkeeping words, written and read by different lanes and launches: always at the L2
__device__ __forceinline__ uint32_t ld_cg_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.global.cg.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_cg_u32(uint32_t* p, uint32_t v) { asm volatile("st.global.cg.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ uint32_t ld_shared_acquire(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.cta.shared.u32 %0, [%1];" : "=r"(v) : "r"(smem_u32(p)) : "memory");
  return v;
}
__device__ __forceinline__ void st_shared_release(uint32_t* p, uint32_t v) {
  asm volatile("st.release.cta.shared.u32 [%0], %1;" ::"r"(smem_u32(p)), "r"(v) : "memory");
}
__device__ __forceinline__ void red_shared_release_add(uint32_t* p, uint32_t v) {
  asm volatile("red.release.cta.shared.add.u32 [%0], %1;" ::"r"(smem_u32(p)), "r"(v) : "memory");
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {  // never blocks
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// global -> this CTA's shared memory, completion counted in bytes on `bar`.  Source is always this GPU's own memory; size
// and both addresses are multiples of 16.
__device__ __forceinline__ void bulk_g2s(void* dst_smem, const void* src_gmem, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst_smem)), "l"(src_gmem),
               "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// global -> L2, this GPU's own memory; size and address are multiples of 16
__device__ __forceinline__ void bulk_prefetch_l2(const void* src_gmem, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src_gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Bounded wait on one of this CTA's own barriers; false when `limit_ns` has passed.  The clock runs on while another process
// has the GPU, so the wait also takes a number of looks, the last of them after the clock was read.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, uint64_t limit_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  for (uint32_t it = 0; it < (1u << 26); it++) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 15) == 15 && it > 48 && globaltimer_ns() - t0 > limit_ns) break;
  }
  return mbar_test(bar, parity);
}

// ----------------------------------------------------------------------------------------------
// what the service warp tells the compute warps about a tile
// ----------------------------------------------------------------------------------------------
struct __align__(16) TileDesc {
  int32_t tile;
  uint32_t flags;
  uint16_t n_frames;  // entries of the tile's frame list
  uint16_t n_slots;   // entries of the tile's slot list
  uint32_t stage;     // two frames or more: the number of the tile among those whose frames are staged
};
constexpr uint32_t kDescNoValues = 2;       // the visit only receives: the values are not loaded, what arrived goes into them as a reduction
constexpr uint32_t kDescTxOk = 1u << 4;     // << link: every out-ring of the link has room
constexpr uint32_t kDescRxLink = 1u << 8;   // << link: at least one frame arrived on the link
constexpr uint32_t kDescTxWant = 1u << 12;  // << link: the link may have something to hear: the tile changed here, or frames arrived on another link
// what a compute warp adds to a tile's `done` word when it has finished its part
constexpr uint32_t kDoneWarp = 1, kDoneWarps = 0xff;
constexpr int kDoneNonsilentShift = 8;      // + 4 * link: warps that found something to say on the link
constexpr uint32_t kDoneFailed = 1u << 24;  // a wait ran out: what arrived has been taken in, links that were to hear something may not have

constexpr uint32_t kStop = 0x80000000u;     // a count of steps that has been closed, see claim_tile()

struct GroupShared {
  TileDesc desc[kBank];
  uint64_t frames[kBank][kMaxRings * kRxMax + 1];  // per tile: the frames that arrived (address | link), in ring and sequence order
  uint64_t slots[kBank][kMaxRings + 1];            // per tile: the ring slots a frame goes into (address | link)
  uint32_t done[kBank];
  uint64_t full[2], empty[2];  // of the two frame stages
  uint32_t armed;        // tiles armed so far in this launch (bank entry = number % kBank)
  uint32_t claim;        // tiles the compute warps have started so far | kStop: no new ones
  uint32_t exchanged;    // exchanges the compute warps have gone through so far | kStop: one ran out
  uint32_t pad;
  uint64_t gsync;        // the compute warps among themselves (blocks of more than 512 elements)
  float red[2][2][kComputeWarps];  // two buffers: a warp may be one step ahead of the slowest one
  alignas(16) uint32_t stage[kComputeWarps][kWarpElems / 4];  // the codes of a warp's part on their way into the ring slots
  // the service warp's own notes about the tiles in hand: the counters after the visit, what moved per ring (frames
  // taken | 4: a frame may go out), the change mark found
  uint32_t rx[kBank][kMaxRings], tx[kBank][kMaxRings];
  uint8_t moved[kBank][kMaxRings];
  uint32_t dirty[kBank];
};

// ----------------------------------------------------------------------------------------------
// per-lane arithmetic.  Piece i of lane `lane` of compute warp `w` is elements w*512 + i*128 + lane*4 .. +3 of the tile.
// A frame stores the codes of 32 consecutive elements t in an order of its own: their eight pieces c = 0..7 sit at
// positions c ^ (t & 7) (4 * Q bits each).  Four elements are held as two packed pairs: the packed fp32 instructions of
// sm_100 round like the scalar ones and halve the instruction count of decoding and quantising.
// ----------------------------------------------------------------------------------------------
struct Piece {
  uint64_t a, b;  // elements 0, 1 and 2, 3
};
__device__ __forceinline__ uint64_t pair(float lo, float hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ uint64_t pair(uint32_t lo, uint32_t hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
  return d;
}
__device__ __forceinline__ void unpair(uint64_t p, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p)); }
__device__ __forceinline__ uint64_t add2(uint64_t x, uint64_t y) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(x), "l"(y));
  return d;
}
__device__ __forceinline__ uint64_t sub2(uint64_t x, uint64_t y) {
  uint64_t d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(x), "l"(y));
  return d;
}
__device__ __forceinline__ uint64_t fma2(uint64_t x, uint64_t y, uint64_t z) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(x), "l"(y), "l"(z));
  return d;
}
__device__ __forceinline__ void add4(Piece& x, const Piece& y) {
  x.a = add2(x.a, y.a);
  x.b = add2(x.b, y.b);
}
// values, mirrors and frames have writers on other SMs and other GPUs: always at the L2
__device__ __forceinline__ Piece load_piece(const float* p) {
  Piece v;
  asm volatile("ld.global.cg.v2.b64 {%0, %1}, [%2];" : "=l"(v.a), "=l"(v.b) : "l"(p));
  return v;
}
__device__ __forceinline__ void store_piece(float* p, const Piece& v) {
  asm volatile("st.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(v.a), "l"(v.b) : "memory");
}
__device__ __forceinline__ void red_add_piece(float* p, const Piece& v) {
  float x, y, z, w;
  unpair(v.a, x, y);
  unpair(v.b, z, w);
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}
__device__ __forceinline__ float maxabs(const Piece& v) {
  float x, y, z, w;
  unpair(v.a, x, y);
  unpair(v.b, z, w);
  return fmaxf(fmaxf(fabsf(x), fabsf(y)), fmaxf(fabsf(z), fabsf(w)));
}

__device__ __forceinline__ int floor_log2_dev(float x) { return int((__float_as_uint(x) >> 23) & 0xff) - 127; }

// sign frames: step = 2^floor(log2(2/3 max|x|)), silent below the cut-off (block_code in ../core/codec.cpp)
__device__ __forceinline__ int block_code_sign(float xmax, uint32_t vmax_bits, int min_exp, int rel_bits) {
  const float scaled = __fmul_rn(xmax, 0.6666667f);
  if ((__float_as_uint(scaled) >> 23) == 0) return 0;
  int kx = floor_log2_dev(scaled);
  if (kx < min_exp) return 0;
  if ((vmax_bits >> 23) != 0) {
    int emax = int(vmax_bits >> 23) - 127;
    if (kx < emax - rel_bits) return 0;
  }
  if (kx < -126) return 0;
  if (kx > 127) kx = 127;
  return kx + 127;
}

// integer frames: the smallest step for which the largest residual still fits (block_code_int in ../core/codec.cpp)
template <int Q>
__device__ __forceinline__ int block_code_int_dev(float xmax, uint32_t vmax_bits, int min_exp, int rel_bits) {
  const uint32_t xb = __float_as_uint(xmax) & 0x7fffffffu;
  const int ef = int(xb >> 23);
  if (ef == 0 || ef == 255) return 0;
  const int ex = ef - 127;
  if (ex > 100) return 0;
  const uint32_t mant = xb & 0x7fffffu;
  int es = ex - (Q - 2);
  if (mant >= (1u << 23) - (1u << (24 - Q))) es += 1;
  es = max(es, min_exp);
  if ((vmax_bits >> 23) != 0) es = max(es, int((vmax_bits >> 23) & 0xffu) - 127 - rel_bits);
  es = max(es, -126);
  if (ex < es - 1 || (ex == es - 1 && mant == 0)) return 0;
  return es + 127;
}

template <int Q>
__device__ __forceinline__ int block_code_dev(float xmax, uint32_t vmax_bits, int min_exp, int rel_bits) {
  if constexpr (Q == 1) return block_code_sign(xmax, vmax_bits, min_exp, rel_bits);
  else return block_code_int_dev<Q>(xmax, vmax_bits, min_exp, rel_bits);
}

// Where piece i of a lane sits in its warp's part of a frame: the 32-element chunk (0..15) and the position in it.
__device__ __forceinline__ int piece_chunk(int i, int lane) { return i * 4 + (lane >> 3); }
__device__ __forceinline__ int piece_pos(int i, int lane) { return (lane & 7) ^ (((i & 1) << 2) + (lane >> 3)); }

// A lane's share of a frame: the codes of its four pieces (the low 4 * Q bits of each word) and their blocks' scale bytes.
// Frame words were written by a neighbour GPU: they are read from the L2, never from this SM's L1.
struct FrameRegs {
  uint32_t w[kPieces];
  uint32_t codes;
  __device__ __forceinline__ uint32_t code(int i) const { return (codes >> (8 * i)) & 0xffu; }
};
template <int Q>
__device__ __forceinline__ void load_frame(const uint8_t* fp, int warp, int lane, int log2_block, FrameRegs& f) {
  const uint8_t* mine = fp + warp * (kWarpElems * Q / 8);
#pragma unroll
  for (int i = 0; i < kPieces; i++) {
    const int unit = piece_chunk(i, lane) * 8 + piece_pos(i, lane);  // in pieces of 4 * Q bits
    if (Q == 8) asm volatile("ld.global.cg.u32 %0, [%1];" : "=r"(f.w[i]) : "l"(mine + unit * 4));
    else if (Q == 4) asm volatile("{\n\t.reg .u16 h;\n\tld.global.cg.u16 h, [%1];\n\tcvt.u32.u16 %0, h;\n\t}" : "=r"(f.w[i]) : "l"(mine + unit * 2));
    else if (Q == 2) asm volatile("ld.global.cg.u8 %0, [%1];" : "=r"(f.w[i]) : "l"(mine + unit));
    else {
      asm volatile("ld.global.cg.u32 %0, [%1];" : "=r"(f.w[i]) : "l"(mine + piece_chunk(i, lane) * 4));
      f.w[i] >>= 4 * piece_pos(i, lane);
    }
  }
  const uint8_t* scales = fp + 4 * Q * kWordsPerTile;
  if (log2_block == 5) {  // the warp's sixteen scale bytes at once
    uint4 c;
    asm volatile("ld.global.cg.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(c.x), "=r"(c.y), "=r"(c.z), "=r"(c.w) : "l"(scales + warp * 16));
    const uint32_t sel = uint32_t(lane >> 3) * 0x11u + 0x40u;
    f.codes = __byte_perm(__byte_perm(c.x, c.y, sel), __byte_perm(c.z, c.w, sel), 0x5410);
  } else {
    uint32_t b[kPieces];
#pragma unroll
    for (int i = 0; i < kPieces; i++)
      asm volatile("ld.global.cg.u8 %0, [%1];" : "=r"(b[i]) : "l"(scales + ((warp * kWarpElems + piece_chunk(i, lane) * 32) >> log2_block)));
    f.codes = b[0] | (b[1] << 8) | (b[2] << 16) | (b[3] << 24);
  }
}

// the same from a frame staged in shared memory
template <int Q>
__device__ __forceinline__ void load_staged(const uint8_t* fp, int warp, int lane, int log2_block, FrameRegs& f) {
  const uint8_t* mine = fp + warp * (kWarpElems * Q / 8);
  const uint8_t* scales = fp + 4 * Q * kWordsPerTile;
  f.codes = 0;
#pragma unroll
  for (int i = 0; i < kPieces; i++) {
    const int unit = piece_chunk(i, lane) * 8 + piece_pos(i, lane);
    if (Q == 8) f.w[i] = reinterpret_cast<const uint32_t*>(mine)[unit];
    else if (Q == 4) f.w[i] = reinterpret_cast<const uint16_t*>(mine)[unit];
    else if (Q == 2) f.w[i] = mine[unit];
    else f.w[i] = reinterpret_cast<const uint32_t*>(mine)[piece_chunk(i, lane)] >> (4 * piece_pos(i, lane));
    f.codes |= uint32_t(scales[(warp * kWarpElems + piece_chunk(i, lane) * 32) >> log2_block]) << (8 * i);
  }
}

// Which of the four elements of piece i exist (bits 0..3).  Only sign frames of the tensor's last tile need it: they have
// no code for "no step" (integer frames carry the code of zero beyond the tensor's end).
__device__ __forceinline__ uint32_t valid4(int left, int i) {
  const int m = left - i * 128;
  return m >= 4 ? 0xfu : (m <= 0 ? 0u : ((1u << m) - 1u));
}

// Four sign bits as steps of +-2^(c-127)
__device__ __forceinline__ Piece sign_steps(uint32_t w, uint32_t c, uint32_t valid) {
  const uint32_t sb = c << 23;
  uint32_t f0 = sb | ((w << 31) & 0x80000000u), f1 = sb | ((w << 30) & 0x80000000u);
  uint32_t f2 = sb | ((w << 29) & 0x80000000u), f3 = sb | ((w << 28) & 0x80000000u);
  if (valid != 0xfu) {
    f0 = valid & 1u ? f0 : 0u; f1 = valid & 2u ? f1 : 0u; f2 = valid & 4u ? f2 : 0u; f3 = valid & 8u ? f3 : 0u;
  }
  return {pair(f0, f1), pair(f2, f3)};
}

// The steps a frame gives the four elements of a piece.  Silent blocks (code 0) and the code no encoder emits (255) step
// by zero.
template <int Q>
__device__ __forceinline__ Piece frame_steps(uint32_t w, uint32_t code, uint32_t valid) {
  const uint32_t c = code == 255u ? 0u : code;
  if constexpr (Q == 1) {
    return sign_steps(w, c, valid);
  } else {
    // a code m stands for (m - 2^(Q-1)) steps; 2^23 + m as a float is 0x4B000000 | m
    const float s = __uint_as_float(c << 23), neg_ms = __fmul_rn(-(8388608.f + float(1 << (Q - 1))), s);
    uint32_t z0, z1, z2, z3;
    if (Q == 8) {
      z0 = __byte_perm(w, 0x4B000000u, 0x7650); z1 = __byte_perm(w, 0x4B000000u, 0x7651);
      z2 = __byte_perm(w, 0x4B000000u, 0x7652); z3 = __byte_perm(w, 0x4B000000u, 0x7653);
    } else {
      constexpr uint32_t m = (1u << Q) - 1u;
      z0 = (w & m) | 0x4B000000u; z1 = ((w >> Q) & m) | 0x4B000000u;
      z2 = ((w >> (2 * Q)) & m) | 0x4B000000u; z3 = ((w >> (3 * Q)) & m) | 0x4B000000u;
    }
    const uint64_t ss = pair(s, s), mm = pair(neg_ms, neg_ms);
    return {fma2(pair(z0, z1), ss, mm), fma2(pair(z2, z3), ss, mm)};
  }
}

// the codes of v - k (4 * Q bits) for a block with exponent code `code`, and the mirror's step (zero for code 0)
template <int Q>
__device__ __forceinline__ uint32_t quantise(const Piece& v, Piece& k, uint32_t code, uint32_t valid) {
  const Piece x = {sub2(v.a, k.a), sub2(v.b, k.b)};
  if constexpr (Q == 1) {
    float x0, x1, x2, x3;
    unpair(x.a, x0, x1);
    unpair(x.b, x2, x3);
    const uint32_t w = ((x0 > 0.f ? 0u : 1u) | (x1 > 0.f ? 0u : 2u) | (x2 > 0.f ? 0u : 4u) | (x3 > 0.f ? 0u : 8u)) & valid;
    add4(k, sign_steps(w, code, valid));
    return w;
  } else {
    const float s = __uint_as_float(code << 23), inv = code ? __uint_as_float((254u - code) << 23) : 0.f;
    const float big = 8388608.f + float(1 << (Q - 1)), neg_ms = __fmul_rn(-big, s);
    const uint64_t ii = pair(inv, inv), bb = pair(big, big), ss = pair(s, s), mm = pair(neg_ms, neg_ms);
    const uint64_t za = fma2(x.a, ii, bb), zb = fma2(x.b, ii, bb);
    k.a = add2(k.a, fma2(za, ss, mm));
    k.b = add2(k.b, fma2(zb, ss, mm));
    const uint32_t b0 = uint32_t(za), b1 = uint32_t(za >> 32), b2 = uint32_t(zb), b3 = uint32_t(zb >> 32);
    if (Q == 8) return __byte_perm(__byte_perm(b0, b1, 0x0040), __byte_perm(b2, b3, 0x0040), 0x5410);
    constexpr uint32_t m = (1u << Q) - 1u;
    return (b0 & m) | ((b1 & m) << Q) | ((b2 & m) << (2 * Q)) | ((b3 & m) << (3 * Q));
  }
}

// Reduces each of the four pieces' values over the eight lanes that share a 32-element chunk, in four shuffles instead of
// twelve: every step halves what a lane holds.  A lane ends up with the result of piece (lane & 3) of its chunk row.
template <class T, class Op>
__device__ __forceinline__ T reduce_pieces(const T (&a)[kPieces], int lane, Op op) {
  const bool b0 = lane & 1, b1 = lane & 2;
  const T s0 = b0 ? a[0] : a[1], k0 = b0 ? a[1] : a[0], s1 = b0 ? a[2] : a[3], k1 = b0 ? a[3] : a[2];
  const T r0 = op(k0, __shfl_xor_sync(0xffffffffu, s0, 1)), r1 = op(k1, __shfl_xor_sync(0xffffffffu, s1, 1));
  const T s = b1 ? r0 : r1, k = b1 ? r1 : r0;
  const T r = op(k, __shfl_xor_sync(0xffffffffu, s, 2));
  return op(r, __shfl_xor_sync(0xffffffffu, r, 4));
}

}  // namespace

// ----------------------------------------------------------------------------------------------
// the kernel
// ----------------------------------------------------------------------------------------------
namespace {

// The eight compute warps take the steps of a launch (tiles, exchanges) in order, and each step is taken by all of them or by
// none, so that no warp has stored its part of a visit that another gave up.  A count of the steps taken says which: the
// first warp to come by moves it past step c, or closes it (kStop) because its wait ran out; the others follow.

// Lane 0 of a compute warp: does the group work on its tile number c?  No when the service warp has closed the claim.  The
// wait covers a service warp that is looking for work; the limit only covers one that never comes back.
__device__ __forceinline__ bool claim_tile(GroupShared& sh, uint32_t c) {
  uint64_t t_start = 0;
  bool give_up = false;
#pragma unroll 1
  for (uint32_t it = 0; it < (1u << 28); it++) {
    const bool armed = int32_t(ld_shared_acquire(&sh.armed) - c) > 0;
    const uint32_t cl = *reinterpret_cast<volatile uint32_t*>(&sh.claim);
    if ((cl & ~kStop) > c) {
      if (armed) return true;  // (not armed: the word has been read before another warp saw it armed)
    } else if (cl & kStop) {
      return false;
    } else if (armed || give_up) {
      if (atomicCAS(&sh.claim, cl, armed ? c + 1u : cl | kStop) == cl) return armed;
      continue;
    }
    if ((it & 63) == 63) {
      const uint64_t now = globaltimer_ns();
      if (t_start == 0) t_start = now;
      give_up = now - t_start > 2000ull * 1000 * 1000;
    }
    if (!armed) __nanosleep(20);
  }
  return false;
}

// The frames of a tile, as the service warp listed them: address | link, in ring order and sequence order.
__device__ __forceinline__ const uint8_t* frame_at(uint64_t e) { return reinterpret_cast<const uint8_t*>(e & ~15ull); }

// Piece i of this lane's part of a link's plane of the group's stash: what arrived on the link.
__device__ __forceinline__ Piece get_part(const float* stash, int link, int i) {
  const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(stash + link * kTile + i * 128);
  return {y.x, y.y};
}
__device__ __forceinline__ void put_part(float* stash, int link, int i, const Piece& x) {
  *reinterpret_cast<ulonglong2*>(stash + link * kTile + i * 128) = make_ulonglong2(x.a, x.b);
}

// What kind of replica a kernel is for: a leaf of the tree (one link, one ring in), a member of a mesh group (one link,
// several rings in), an inner node (several links).
enum Kind { kLeaf, kMember, kInner };
// Frames of a tile that are staged in shared memory, and the room for one.  A member of a mesh of eight decodes seven frames
// per tile: out of shared memory, two tiles ahead, a pass over 4 Mi elements takes 42 us, with loads from the L2 48 us.  The
// other kinds fetch their frames themselves: a leaf seldom has more than one, an inner node no registers to spare (a pass of
// a hub and its leaves over 16 M elements takes 522 us so, 542 us with stages).
template <int Q>
constexpr int kFrameRoom = Q * 512 + 128;
template <int kKind>
constexpr int kStaged = kKind == kMember ? 8 : 0;
// Who asks the L2 for the lines of the next tile: the service warp, a lane per array, or a compute warp, whose own part of the
// tile in hand waits meanwhile.  With the service warp three rounds of 100 M elements on one link take 1144 us instead of 1159,
// a hub and two leaves over 30 M 632 instead of 644 (the pass of a hub with three links over 32 Mi alone 248 instead of 305).
// For a mesh member, whose service warp has copies to see to, it makes no difference (mesh of eight: 603 and 601).  In a leaf's
// short visits of sign frames the service warp comes late (3.3 M elements: 50.9 instead of 49.9).  That is no reason for an
// inner node with sign frames, which the rule takes along: with the service warp a hub and three leaves over 16 M elements
// would take 524 us instead of 531, a hub and two over 30 M 658 instead of 668 (3.3 M: 107 and 107).
template <int Q, int kKind>
constexpr bool kServiceAhead = kKind != kMember && Q > 1;

// total = the sum of the steps of the tile's frames, in list order; kStash: what came on each link is summed up besides, and
// left in this lane's part of the link's stash (shared memory; a frame is decoded once, however many links hear of it: a hub
// with three links and six frames per tile took 224 us per 16 M elements when it decoded them for the values and again for
// each mirror, 170 us so).  The loop stays rolled: the code of a tile's visit has to fit the instruction cache.
template <int Q, bool kStash, int kIn>
__device__ __forceinline__ void decode_frames(const uint64_t* list, const uint8_t* staged, bool in_stage, int count, uint32_t live, uint64_t* empty, int log2_block,
                                              int warp, int lane, int left, float* stash, Piece (&total)[kPieces]) {
  uint32_t seen = 0;
#pragma unroll
  for (int i = 0; i < kPieces; i++) total[i] = {0ull, 0ull};
#pragma unroll 1
  for (int j = 0; j < count; j++) {
    FrameRegs f{};
    if (live) {
      if (in_stage && j < kIn) load_staged<Q>(staged + j * kFrameRoom<Q>, warp, lane, log2_block, f);
      else load_frame<Q>(frame_at(list[j]), warp, lane, log2_block, f);
    }
    const int link = kStash && live ? int(list[j] & 15u) : 0;
    const bool again = (seen >> link) & 1u;
    seen |= 1u << link;
#pragma unroll
    for (int i = 0; i < kPieces; i++) {
      Piece st = frame_steps<Q>(f.w[i], f.code(i), Q == 1 ? valid4(left, i) : 0xfu);
      add4(total[i], st);
      if (kStash) {
        if (again) add4(st, get_part(stash, link, i));
        put_part(stash, link, i, st);
      }
    }
  }
  if (kIn == 0) return;
  __syncwarp();
  if (live && in_stage && lane == 0) mbar_arrive(empty);  // the stage may be filled again when all warps have read it
}

// One lane's codes of its four pieces into the ring slots of link l's neighbours.  They go through shared memory, so
// that a warp's part leaves as one contiguous run of 16-byte stores per ring.
template <int Q>
__device__ __forceinline__ void send_codes(const uint64_t* list, int count, int log2_block, int l, int warp, int lane,
                                           const uint32_t (&w)[kPieces], bool loud, uint32_t code, uint32_t* stage) {
  uint4 run = make_uint4(0u, 0u, 0u, 0u);
  if (loud) {
    if (Q == 1) {
      uint32_t word[kPieces];
#pragma unroll
      for (int i = 0; i < kPieces; i++) word[i] = w[i] << (4 * piece_pos(i, lane));
      const uint32_t chunk = reduce_pieces(word, lane, [](uint32_t a, uint32_t b) { return a | b; });
      if ((lane & 4) == 0) stage[piece_chunk(lane & 3, lane)] = chunk;
    } else {
#pragma unroll
      for (int i = 0; i < kPieces; i++) {
        const int unit = piece_chunk(i, lane) * 8 + piece_pos(i, lane);
        if (Q == 8) stage[unit] = w[i];
        else if (Q == 4) reinterpret_cast<uint16_t*>(stage)[unit] = uint16_t(w[i]);
        else reinterpret_cast<uint8_t*>(stage)[unit] = uint8_t(w[i]);
      }
    }
    __syncwarp();
    if (lane < 4 * Q) run = reinterpret_cast<const uint4*>(stage)[lane];
    __syncwarp();
  }
  // the scale byte of a block: the lane that holds the block's first chunk
  const int chunk = warp * 16 + piece_chunk(lane & 3, lane), per_block = log2_block - 5;
  const bool mine = (lane & 4) == 0 && (chunk & ((1 << per_block) - 1)) == 0;
  for (int j = 0; j < count; j++) {
    if (int(list[j] & 15u) != l) continue;
    uint8_t* pay = reinterpret_cast<uint8_t*>(list[j] & ~15ull);
    if (loud && lane < 4 * Q) *reinterpret_cast<uint4*>(pay + warp * (kWarpElems * Q / 8) + lane * 16) = run;
    if (mine) pay[4 * Q * kWordsPerTile + (chunk >> per_block)] = uint8_t(code);
  }
}

// Test hook: this warp's waits for the tile count as having run out.
__device__ __forceinline__ bool held(const RoundParams& p, int tile, int warp) {
  return tile == p.stall_tile && p.stall_warp >= 0 && (p.stall_warp & (kComputeWarps - 1)) == warp;
}

// The maxima of a block of 1024 elements and more, over the warps that share it: {-1, -1} if the eight did not come together
// in time for exchange number e.
__device__ __forceinline__ float2 exchange(const RoundParams& p, GroupShared& sh, uint32_t e, int tile, int warp, int lane, float xm, float vm) {
  const bool hold = held(p, tile, warp);
  float(*red)[kComputeWarps] = sh.red[e & 1u];
  __syncwarp();  // every lane has read the exchange before last, whose words are written again behind this one
  if (lane == 0 && !(hold && p.stall_warp < kComputeWarps)) {
    red[0][warp] = xm;
    red[1][warp] = vm;
    mbar_arrive(&sh.gsync);
  }
  const bool there = __all_sync(0xffffffffu, !hold && mbar_wait_bounded(&sh.gsync, e & 1u, p.wait_ns));
  bool go = false;
  if (lane == 0) {
    const uint32_t seen = atomicCAS(&sh.exchanged, e, there ? e + 1u : e | kStop);
    go = seen == e ? there : (seen & ~kStop) > e;
  }
  if (!__any_sync(0xffffffffu, go)) return make_float2(-1.f, -1.f);
  if (!there) (void)mbar_wait_bounded(&sh.gsync, e & 1u, p.wait_ns);  // (another warp has seen it complete)
  const int share = 1 << (p.log2_block - 9), w0 = warp & ~(share - 1);
  for (int j = 0; j < share; j++) {
    xm = fmaxf(xm, red[0][w0 + j]);
    vm = fmaxf(vm, red[1][w0 + j]);
  }
  return make_float2(xm, vm);
}
// (out of the way of smaller blocks where the visit has few registers to save around a call)
__device__ __noinline__ float2 exchange_apart(const RoundParams& p, GroupShared& sh, uint32_t e, int tile, int warp, int lane, float xm, float vm) {
  return exchange(p, sh, e, tile, warp, lane, xm, vm);
}

template <int Q, int kKind>
__device__ __forceinline__ void compute_warp(const RoundParams& p, GroupShared& sh, float* group_stash, const uint8_t* stages, int warp, int lane) {
  constexpr bool kOneLink = kKind != kInner;  // what arrived for the values is what arrived on the link
  constexpr int kIn = kStaged<kKind>;
  const int L = kOneLink ? 1 : p.n_links, lb = p.log2_block;
  float res_max0 = 0.f, res_max1 = 0.f, res_max2 = 0.f;
  uint32_t exchanges = 0;
  bool unstaged = false;  // the warp has stopped using the stages
  // While the service warp looks for work, the compute warps go once through the code of a visit with nothing in hand: the
  // instruction cache is cold at the start of a launch, and the first tile took 5 us longer than the others for that.
  uint32_t live = 0;
  asm volatile("" : "+r"(live));  // (the compiler is not to make a copy of the code for it)
#pragma unroll 1
  for (uint32_t c = 0;;) {
    TileDesc d{0, kDescTxOk | kDescRxLink | kDescTxWant, uint16_t(p.n_in > 1 ? 2 : 1), 0, 0};
    uint32_t entry = 0;
    if (live) {
      const uint32_t go = lane == 0 ? (claim_tile(sh, c) ? 1u : 0u) : 0u;
      if (!__shfl_sync(0xffffffffu, go, 0)) break;
      __syncwarp();  // a shuffle orders no memory: what lane 0 has acquired is there for all lanes from here on
      entry = c % kBank;
      d = sh.desc[entry];
      c++;
    }
    // Where the service warp does not do it: the next tile on its way into the L2.  A leaf and a mesh member ask once this
    // tile's loads are under way (ahead of them, a mesh of eight takes 643 us instead of 620, three sign rounds of 3.3 M elements
    // on one link 51 instead of 49), but ahead of them in a visit that only sends and has little else to wait for; an inner node
    // with sign frames, whose loads are spread over its visit, asks at the start.  One tile ahead is best: a window of 25 M
    // elements that receives and sends takes 92 us so, 115 us with two tiles ahead and 153 us with four; without, three rounds of
    // 100 M elements on one link take 1278 us instead of 1157.
    auto prefetch_next = [&]() {
      const uint32_t ahead = c;  // (c is the next tile's number by now)
      if (kServiceAhead<Q, kKind> || !live || warp != 0 || lane != 0 || int32_t(ld_shared_acquire(&sh.armed) - ahead) <= 0) return;
      const TileDesc& e = sh.desc[ahead % kBank];
      if (!(e.flags & kDescNoValues)) bulk_prefetch_l2(p.values + size_t(e.tile) * kTile, kTile * 4);
      for (int l = 0; l < L; l++) bulk_prefetch_l2(p.mirror[l] + size_t(e.tile) * kTile, kTile * 4);
      if (kIn == 0 || e.n_frames == 1)
        for (int j = 0; j < e.n_frames; j++) bulk_prefetch_l2(frame_at(sh.frames[ahead % kBank][j]), uint32_t(p.payload_bytes));
    };
    const int in_tile = warp * kWarpElems + lane * 4;
    const size_t off = size_t(d.tile) * kTile + in_tile;
    const int left = int(min(int64_t(kTile), p.n - int64_t(d.tile) * kTile)) - in_tile;  // (used by sign frames only)
    float* const vp = p.values + off;
    Piece v[kPieces], k[kPieces];
    const uint64_t* frames = sh.frames[entry];
    const bool load_v = live && (d.flags & kDescNoValues) == 0;
    float* const stash = group_stash + in_tile;
    if (!kOneLink) {
      // What arrived, then the values into it.  Nothing is held in registers beyond that and the mirror of the link in hand, and
      // the values' maxima are taken once for all links: the kernel spills nothing, and a hub with two leaves takes 638 us for
      // its rounds over 30 M elements instead of 657.  (While a compute warp asked for the next tile's lines, and held up the
      // group with it, more did not help: 72 registers and three groups gave 524 us against 511 for a hub and three leaves over
      // 16 M, the next link's mirror loaded ahead into registers 505 against 502.  Neither has been measured since.)
      prefetch_next();
      decode_frames<Q, true, 0>(frames, nullptr, false, d.n_frames, live, nullptr, lb, warp, lane, left, stash, v);
#pragma unroll
      for (int i = 0; i < kPieces; i++) k[i] = live ? load_piece(vp + i * 128) : Piece{0ull, 0ull};
#pragma unroll
      for (int i = 0; i < kPieces; i++) {
        if (live && (v[i].a | v[i].b)) red_add_piece(vp + i * 128, v[i]);
        add4(v[i], k[i]);
      }
    } else if (d.n_frames <= 1) {
      // the common case: everything is fetched at once, and the one frame's steps never have to be kept
      if (d.n_frames == 0) prefetch_next();
#pragma unroll
      for (int i = 0; i < kPieces; i++) v[i] = load_v ? load_piece(vp + i * 128) : Piece{0ull, 0ull};
#pragma unroll
      for (int i = 0; i < kPieces; i++) k[i] = live ? load_piece(p.mirror[0] + off + i * 128) : Piece{0ull, 0ull};
      if (d.n_frames == 1) {
        prefetch_next();
        FrameRegs f{};
        if (live) load_frame<Q>(frame_at(frames[0]), warp, lane, lb, f);
#pragma unroll
        for (int i = 0; i < kPieces; i++) {
          const Piece s = frame_steps<Q>(f.w[i], f.code(i), Q == 1 ? valid4(left, i) : 0xfu);
          if (f.code(i)) red_add_piece(vp + i * 128, s);
          add4(v[i], s);
          add4(k[i], s);
        }
      }
    } else {
      // (values and mirror on their way while the frames are decoded)
#pragma unroll
      for (int i = 0; i < kPieces; i++) {
        v[i] = load_v ? load_piece(vp + i * 128) : Piece{0ull, 0ull};
        k[i] = live ? load_piece(p.mirror[0] + off + i * 128) : Piece{0ull, 0ull};
      }
      prefetch_next();
      const uint32_t st = d.stage & 1u;
      if (kIn > 0 && live) {
        // A warp whose stage is not filled in time reads the frames from the ring, where they stay until the tile is
        // published.  It does not report the stage as read, so that neither stage is filled again under another warp's
        // hands once its turn has come, and uses no stage any more.
        if (!unstaged) unstaged = !__all_sync(0xffffffffu, !held(p, d.tile, warp) && mbar_wait_bounded(&sh.full[st], (d.stage >> 1) & 1u, 2ull * p.wait_ns));
      }
      Piece acc[kPieces];
      decode_frames<Q, false, kIn>(frames, stages + st * (kIn * kFrameRoom<Q>), !unstaged, d.n_frames, live, &sh.empty[st], lb, warp, lane, left, nullptr, acc);
#pragma unroll
      for (int i = 0; i < kPieces; i++) {
        if (live) red_add_piece(vp + i * 128, acc[i]);
        add4(v[i], acc[i]);
        add4(k[i], acc[i]);
      }
    }
    auto larger = [](float a, float b) { return fmaxf(a, b); };
    // over the chunks of a piece row and the piece rows: blocks of up to 512 elements
    auto over_block = [&](float m) {
      if (lb >= 6) {
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 8));
        if (lb >= 7) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16));
        if (lb >= 8) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
        if (lb >= 9) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
      }
      return m;
    };
    float vmax = 0.f;  // an inner node: the largest |value| of each block, the same for all links
    if (!kOneLink) {
      float vs[kPieces];
#pragma unroll
      for (int i = 0; i < kPieces; i++) {
        vs[i] = maxabs(v[i]);
      }
      vmax = over_block(reduce_pieces(vs, lane, larger));
    }
    const int n_links = live ? L : 1;  // (once through the code of a link is enough to fetch it)
    uint32_t finished = kDoneWarp;
    bool failed = false;
#pragma unroll 1
    for (int l = 0; l < n_links; l++) {
      float* const kp = p.mirror[l] + off;
      if (!kOneLink) {
#pragma unroll
        for (int i = 0; i < kPieces; i++) k[i] = live ? load_piece(kp + i * 128) : Piece{0ull, 0ull};
      }
      bool changed = false;
      if (d.flags & (kDescRxLink << l)) {
        if (!kOneLink) {
#pragma unroll
          for (int i = 0; i < kPieces; i++) add4(k[i], get_part(stash, l, i));
        }
        changed = true;
      }
      if (d.flags & (kDescTxWant << l)) {  // (a visit that only receives says nothing back, whatever rounding left)
        float xs[kPieces], vs[kPieces];
#pragma unroll
        for (int i = 0; i < kPieces; i++) {
          xs[i] = maxabs({sub2(v[i].a, k[i].a), sub2(v[i].b, k[i].b)});
          if (kOneLink) vs[i] = maxabs(v[i]);
        }
        float xm = reduce_pieces(xs, lane, larger), vm = kOneLink ? reduce_pieces(vs, lane, larger) : vmax;
        if (kOneLink || l == 0) res_max0 = fmaxf(res_max0, xm); else if (l == 1) res_max1 = fmaxf(res_max1, xm); else res_max2 = fmaxf(res_max2, xm);
        // blocks of more than 32 elements: over the chunks of a piece row, the piece rows, the warps
        if (lb >= 6) {
          xm = over_block(xm);
          if (kOneLink) vm = over_block(vm);
          if (lb >= 10 && live) {
            float2 m = make_float2(-1.f, -1.f);
            if (!failed) m = kOneLink ? exchange_apart(p, sh, exchanges, d.tile, warp, lane, xm, vm) : exchange(p, sh, exchanges, d.tile, warp, lane, xm, vm);
            if (__any_sync(0xffffffffu, m.x < 0.f)) {
              // Without the block's maximum nothing can be said on the link; what arrived is taken in all the same.  (From
              // here on no warp comes to the barrier any more: nobody is counted for an exchange it was late for.)
              failed = true;
              if (changed) {
#pragma unroll
                for (int i = 0; i < kPieces; i++) store_piece(kp + i * 128, k[i]);
              }
              continue;
            }
            exchanges++;
            xm = m.x;
            vm = m.y;
          }
        }
        const uint32_t code = uint32_t(block_code_dev<Q>(xm, __float_as_uint(vm), p.min_exp, p.rel_bits));
        const bool loud = __any_sync(0xffffffffu, code != 0 || !live);
        if (loud) finished += 1u << (kDoneNonsilentShift + 4 * l);
        if (d.flags & (kDescTxOk << l)) {
          uint32_t w[kPieces];
          if (loud) {
#pragma unroll
            for (int i = 0; i < kPieces; i++)
              w[i] = quantise<Q>(v[i], k[i], __shfl_sync(0xffffffffu, code, (lane & ~3) | i), Q == 1 ? valid4(left, i) : 0xfu);
            changed = true;
          }
          send_codes<Q>(sh.slots[entry], d.n_slots, lb, l, warp, lane, w, loud, code, sh.stage[warp]);
        }
      }
      if (changed && live) {
#pragma unroll
        for (int i = 0; i < kPieces; i++) store_piece(kp + i * 128, k[i]);
      }
    }
    if (failed || unstaged) finished |= kDoneFailed;
    __syncwarp();  // what the lanes stored comes before what lane 0 says about it
    if (lane == 0 && live) red_shared_release_add(&sh.done[entry], finished);
    // (A member's warps leave at the next claim, which the service warp closes; until then no exchange is agreed on.  How the
    // compiler lays the loop out hangs on this exit: with it the mesh of eight takes 663 us, without 633; a leaf's three sign
    // rounds of 3.3 M elements take 70 us without it and 61 with it.)
    if (kKind != kMember && failed) break;
    live = 1;
    asm volatile("" : "+r"(live));
  }
  // ---- statistics: the largest outstanding residual per link
  for (int o = 16; o > 0; o >>= 1) {
    res_max0 = fmaxf(res_max0, __shfl_xor_sync(0xffffffffu, res_max0, o));
    res_max1 = fmaxf(res_max1, __shfl_xor_sync(0xffffffffu, res_max1, o));
    res_max2 = fmaxf(res_max2, __shfl_xor_sync(0xffffffffu, res_max2, o));
  }
  if (lane == 0) {  // non-negative floats order like their bit patterns
    unsigned long long* rm = reinterpret_cast<unsigned long long*>(p.status + (p.parity ? kDsLaunch1 : kDsLaunch0) + kDlResMax);
    if (res_max0 != 0.f) atomicMax(rm + 0, (unsigned long long)__float_as_uint(res_max0));
    if (res_max1 != 0.f) atomicMax(rm + 1, (unsigned long long)__float_as_uint(res_max1));
    if (res_max2 != 0.f) atomicMax(rm + 2, (unsigned long long)__float_as_uint(res_max2));
  }
}

// The service warp.  A lane looks after one ring pair (in-ring r and out-ring r) of one tile: with R rings, rounded up to
// a power of two above one, 32 / R tiles are looked at together, and every look costs two round trips to the L2 whatever R is.
// All 32 lanes run the same control flow; decisions taken from words that change under the warp's feet are taken by one
// lane, or on a ballot.
// What it does before the first tile is armed and after the last one is finished is the fixed part of every launch, a chain of
// one warp's instructions.  It is compiled for each kind of replica, so that a leaf has no loops over links and rings and no
// ballots among its lanes, and divides nothing and reads no clock on that way: the first tile of a launch is armed after 2.1 us
// instead of 3.1 (a member's after 2.9 instead of 3.8), and three rounds over 811 tiles of sign frames take 49 us instead of 54.
template <int Q, int kKind>
__device__ __forceinline__ void service_warp(const RoundParams& p, GroupShared& sh, uint8_t* stages, int staged_frames, int frame_room, int g, int n_groups, int lane) {
  // The group's tiles: a run of `chunk` consecutive tiles, or (chunk == 0) every gstride-th tile of the launch's window.
  // The groups of a CTA are a grid apart, so that the odd tiles of the last turn fall on all SMs alike.
  const int gidx = p.chunk > 0 ? int(blockIdx.x) * n_groups + g : g * int(gridDim.x) + int(blockIdx.x);
  const int gid0 = p.chunk > 0 ? gidx * p.chunk : gidx;
  const int gstride = p.chunk > 0 ? 1 : int(gridDim.x) * n_groups;
  const int my_count = p.chunk > 0 ? max(0, min(p.chunk, p.tile_count - gid0)) : p.tiles_each + (gid0 < p.groups_more ? 1 : 0);
  const int gid = p.tile_begin + gid0;
  const uint32_t smask = uint32_t(p.ring_slots) - 1u;
  const uint64_t limit_ns = p.wait_ns;
  uint64_t* const launch_words = p.status + (p.parity ? kDsLaunch1 : kDsLaunch0);
  unsigned long long sent_before = 0;             // for the trace

  // ---- this lane's ring pair and its place among the tiles looked at together
  constexpr bool kLeafOnly = kKind == kLeaf, kOneLink = kKind != kInner;
  const int n_links = kOneLink ? 1 : p.n_links, rings = kLeafOnly ? 1 : max(p.n_in, p.n_out);
  const int log2_rings = rings > 4 ? 3 : (rings > 2 ? 2 : 1);  // (16 tiles at most, so that the next look fits into the bank in time)
  const int at_once = 32 >> log2_rings;           // tiles of one look
  const int r = lane >> (5 - log2_rings), t = lane & (at_once - 1);
  // the lanes of this lane's tile, one per ring, in ring order
  const uint32_t same_tile = kLeafOnly ? 1u << lane : (log2_rings == 3 ? 0x11111111u : (log2_rings == 2 ? 0x01010101u : 0x00010001u)) << t;
  const uint32_t below = (1u << lane) - 1u;
  const bool is_in = r < p.n_in && p.do_rx, is_out = r < p.n_out && p.do_tx;
  InRing in{};
  OutRing out{};
  if (r < p.n_in) in = p.in[r];
  if (r < p.n_out) out = p.out[r];

  bool handed_on = false;   // the next window's launch has been let in
  uint32_t n_done = 0, n_tx = 0, n_rx = 0, n_blocked = 0, n_pending = 0, n_sweeps = 0;  // per lane, added up at the end
  bool open = false;        // this lane has found frames that have not been acknowledged
  uint32_t armed = 0, finished = 0, published = 0;  // tiles armed, finished by the compute warps, published so far
  uint32_t handed = 0, staged = 0;                  // tiles the compute warps may start, and those of them whose frames have been seen to
  uint32_t stage_no = 0, stage_issued = 0;          // tiles with two frames or more found so far, and those staged
  uint32_t ahead = 0;                               // the last tile whose lines have been asked for ahead of time
  bool aborted = false, yielded = false;
  bool ran_out = false;                             // a wait of a compute warp did

  // Bookkeeping of the launch, done behind the first look's loads.
  auto begin_launch = [&]() {
    if (blockIdx.x != 0 || g != 0) return;
    uint64_t* other = p.status + (p.parity ? kDsLaunch0 : kDsLaunch1);  // the next cycle's half
    if (p.zero_other && lane < 8) other[lane] = 0;
    if (lane == 0) sent_before = p.status[kDsFramesSent];
  };
  if (my_count == 0) begin_launch();
  auto update_waiting = [&]() -> bool {
    const uint32_t y = p.yield_flag != nullptr && lane == 0 ? ld_cg_u32(p.yield_flag) : 0u;
    return __any_sync(0xffffffffu, y != 0);
  };

  for (int sweep = 0; sweep < p.sweeps && !aborted && !yielded && my_count > 0; sweep++) {
    const uint32_t armed_before = armed;
    int looked = 0;           // tiles of the group looked at in this sweep
    uint32_t idle = 0;
    uint64_t t_last = 0;      // (read when there has been nothing to do for some looks: reading the clock takes its time)
    while (true) {
      // ---- the frames of the next tiles that have several on their way into shared memory, as stages become free
      while (staged_frames > 0 && staged != handed && !ran_out) {
        const TileDesc d = sh.desc[staged % kBank];
        if (d.n_frames > 1) {
          const uint32_t u = stage_issued & 1u;
          uint32_t free = 1;
          if (stage_issued >= 2 && lane == 0) free = mbar_test(&sh.empty[u], (stage_issued / 2 - 1u) & 1u) ? 1u : 0u;
          if (!__shfl_sync(0xffffffffu, free, 0)) break;
          const int count = min(int(d.n_frames), staged_frames);
          if (lane == 0) mbar_expect_tx(&sh.full[u], uint32_t(count) * uint32_t(p.payload_bytes));
          __syncwarp();
          if (lane < count) {
            asm volatile("fence.proxy.async;" ::: "memory");  // the frames came by ordinary stores, their flags have been acquired
            bulk_g2s(stages + (int(u) * staged_frames + lane) * frame_room, frame_at(sh.frames[staged % kBank][lane]), uint32_t(p.payload_bytes), &sh.full[u]);
          }
          __syncwarp();
          stage_issued++;
        }
        staged++;
      }
      // ---- look at more tiles while the compute warps have less than kAhead in hand and the bank has room for them
      if (looked < my_count && !yielded && !aborted && !ran_out && armed - finished < uint32_t(kAhead) && armed - published + uint32_t(at_once) <= uint32_t(kBank)) {
        ST_CRUMB(g, 2);
        const uint32_t y = p.yield_flag != nullptr && lane == 0 ? ld_cg_u32(p.yield_flag) : 0u;
        const int j = looked + t;
        const bool valid = j < my_count && (!kLeafOnly || r == 0);
        const int tile = gid + j * gstride;
        looked += at_once;
        uint32_t dirty = 0, rx = 0, tx = 0, credit = 0, avail = 0;
        if (valid) {
          // The change mark is cleared before the tile's values are read (the tile is armed after this exchange has
          // returned), and whoever changes the values sets it after the change: a change that this visit does not see
          // leaves its mark for the next one.
          if (r == 0) dirty = atomicExch(p.tile_state + tile, 0u);
          // With four slots or fewer all their flags are fetched along with the counters, before it is known which come next.
          const bool few = smask < 4u;
          const uint32_t* fl = in.flags + tile;
          uint32_t f0 = 0, f1 = 0, f2 = 0, s0 = 0, s1 = 0, s2 = 0, s3 = 0;
          if (is_in) {
            rx = ld_cg_u32(in.rx_seq + tile);
            if (few) {
              s0 = ld_relaxed_sys(fl);
              s1 = ld_relaxed_sys(fl + p.n_tiles);
              s2 = ld_relaxed_sys(fl + size_t(2u & smask) * p.n_tiles);
              s3 = ld_relaxed_sys(fl + size_t(3u & smask) * p.n_tiles);
            }
          }
          if (is_out) {
            tx = ld_cg_u32(out.tx_seq + tile);
            credit = ld_relaxed_sys(out.credit + tile);  // (a slot is only stored to once its credit has been seen)
          }
          if (is_in) {
            if (few) {
              auto slot = [&](uint32_t i) { return i & 2u ? (i & 1u ? s3 : s2) : (i & 1u ? s1 : s0); };
              f0 = slot(rx & smask);
              f1 = slot((rx + 1u) & smask);
              f2 = slot((rx + 2u) & smask);
            } else {
              f0 = ld_relaxed_sys(fl + size_t(rx & smask) * p.n_tiles);
              f1 = ld_relaxed_sys(fl + size_t((rx + 1u) & smask) * p.n_tiles);
              f2 = ld_relaxed_sys(fl + size_t((rx + 2u) & smask) * p.n_tiles);
            }
            avail = f0 != rx + 1u ? 0u : (f1 != rx + 2u ? 1u : (f2 != rx + 3u ? 2u : 3u));
            // the flag of the last frame once more, as the acquire that the frames' contents are read behind (the looks
            // above went out together; an acquire holds up every access after it)
            if (avail) (void)ld_acquire_sys(fl + size_t((rx + avail - 1u) & smask) * p.n_tiles);
          }
        }
        if (looked == at_once && sweep == 0) begin_launch();
        open |= tx != credit;  // (the flush() of a replica asks the passes whether its frames have been taken in)
        const bool room = is_out && (tx - credit) < uint32_t(p.ring_slots);
        // (a leaf's lane has its tile to itself)
        uint32_t in1 = avail >= 1 ? same_tile : 0u, in2 = avail >= 2 ? same_tile : 0u, in3 = avail >= 3 ? same_tile : 0u;
        if (!kLeafOnly) {
          dirty = __shfl_sync(0xffffffffu, dirty, t);
          in1 = __ballot_sync(0xffffffffu, avail >= 1);
          in2 = __ballot_sync(0xffffffffu, avail >= 2);
          in3 = __ballot_sync(0xffffffffu, avail >= 3);
        }
        const bool any_in = (in1 & same_tile) != 0, work = valid && (dirty != 0 || any_in);
        if (__any_sync(0xffffffffu, y != 0)) {  // an update is waiting for SMs: hand out nothing more
          if (dirty && r == 0) st_cg_u32(p.tile_state + tile, 1u);
          yielded = true;
          continue;
        }
        const uint32_t work_tiles = __ballot_sync(0xffffffffu, work && r == 0);  // bit t: the t-th tile of this look
        if (work_tiles == 0) continue;
        // A frame that arrived on link l changes the values and l's mirror alike: it leaves nothing to say on l, and
        // what rounding makes of it (or a cut-off that moved with the values) is not worth a frame back.  The link
        // gets a frame when the tile changed here (its mark) or when another link brought something to pass on.
        uint32_t flags = 0;
        bool goes_out = false;
        for (int l = 0; l < n_links; l++) {
          uint32_t here, outs, full;
          if (kLeafOnly) {
            here = in1;
            outs = is_out ? same_tile : 0u;
            full = is_out && !room ? same_tile : 0u;
          } else if (kOneLink) {
            here = in1 & same_tile;
            outs = __ballot_sync(0xffffffffu, is_out) & same_tile;
            full = __ballot_sync(0xffffffffu, is_out && !room) & same_tile;
          } else {
            here = __ballot_sync(0xffffffffu, avail != 0 && in.link == l) & same_tile;
            outs = __ballot_sync(0xffffffffu, is_out && out.link == l) & same_tile;
            full = __ballot_sync(0xffffffffu, is_out && out.link == l && !room) & same_tile;
          }
          const bool want = dirty != 0 || (in1 & same_tile & ~here) != 0;
          const bool ok = want && outs != 0 && full == 0;
          flags |= (ok ? kDescTxOk << l : 0u) | (here ? kDescRxLink << l : 0u) | (want ? kDescTxWant << l : 0u);
          goes_out |= ok && is_out && (kOneLink || out.link == l);
        }
        // A tile of a one-link replica that carries no mark is here only to receive: nothing is said on the link, so
        // the values themselves are not needed.
        if (n_links == 1 && dirty == 0) flags |= kDescNoValues;
        const uint32_t sends = kLeafOnly ? (goes_out ? same_tile : 0u) : __ballot_sync(0xffffffffu, goes_out) & same_tile;
        const int n_frames = __popc(in1 & same_tile) + __popc(in2 & same_tile) + __popc(in3 & same_tile);
        const uint32_t several = staged_frames > 0 ? __ballot_sync(0xffffffffu, work && r == 0 && n_frames > 1) : 0u;
        const uint32_t pos = armed + __popc(work_tiles & ((1u << t) - 1u)), entry = pos % kBank;
        if (work) {
          if (r == 0) {
            sh.desc[entry] = TileDesc{tile, flags, uint16_t(n_frames), uint16_t(__popc(sends)), stage_no + __popc(several & ((1u << t) - 1u))};
            sh.done[entry] = 0;
            sh.dirty[entry] = dirty;
          }
          const uint32_t before = same_tile & below;
          uint64_t* list = &sh.frames[entry][__popc(in1 & before) + __popc(in2 & before) + __popc(in3 & before)];
          for (uint32_t f = 0; f < avail; f++)
            list[f] = reinterpret_cast<uint64_t>(in.payload + (size_t((rx + f) & smask) * p.n_tiles + tile) * p.payload_bytes) | uint32_t(in.link);
          if (goes_out)
            sh.slots[entry][__popc(sends & before)] =
                reinterpret_cast<uint64_t>(out.payload_remote + (size_t(tx & smask) * p.n_tiles + tile) * p.payload_bytes) | uint32_t(out.link);
          sh.rx[entry][r] = avail ? rx + avail : 0u;
          sh.tx[entry][r] = goes_out ? tx + 1u : 0u;
          sh.moved[entry][r] = uint8_t(avail | (goes_out ? 4u : 0u));
        }
        // test hook: this tile is never handed to the compute warps, so the wait for it below runs out
        const uint32_t stalled = __ballot_sync(0xffffffffu, work && tile == p.stall_tile && p.stall_warp < 0 && r == 0);
        handed = stalled ? armed + __popc(work_tiles & ((1u << (__ffs(stalled) - 1)) - 1u)) : armed + __popc(work_tiles);
        __syncwarp();
        if (lane == 0) st_shared_release(&sh.armed, handed);
        // The lines of a tile that is begun at once (for the later ones see kServiceAhead): all of them, while the warps are on
        // their way to asking for the first.  A hub and its leaves over 16 M elements take 517 us so, 522 without; a mesh of
        // eight, whose members begin with bulk copies of their frames, 603 without and 617 so.
        if (kKind != kMember && work && pos == finished) {
          if (r == 0) {
            if (!(flags & kDescNoValues)) bulk_prefetch_l2(p.values + size_t(tile) * kTile, kTile * 4);
            for (int l = 0; l < n_links; l++) bulk_prefetch_l2(p.mirror[l] + size_t(tile) * kTile, kTile * 4);
          }
          for (uint32_t f = 0; f < avail; f++)
            bulk_prefetch_l2(in.payload + (size_t((rx + f) & smask) * p.n_tiles + tile) * p.payload_bytes, uint32_t(p.payload_bytes));
        }
        armed += __popc(work_tiles);
        stage_no += __popc(several);
        if (stalled) looked = my_count;
        idle = 0;
        continue;
      }
      // ---- the next tile on its way into the L2, once the compute warps have started on the one before it
      if (kServiceAhead<Q, kKind> && int32_t(handed - finished) > 1 && ahead != finished + 1u) {
        const uint32_t begun = lane == 0 ? *reinterpret_cast<volatile uint32_t*>(&sh.claim) & ~kStop : 0u;
        if (__shfl_sync(0xffffffffu, begun, 0) > finished) {
          ahead = finished + 1u;
          const TileDesc e = sh.desc[ahead % kBank];
          if (lane == 0 && !(e.flags & kDescNoValues)) bulk_prefetch_l2(p.values + size_t(e.tile) * kTile, kTile * 4);
          if (lane >= 1 && lane <= n_links) bulk_prefetch_l2(p.mirror[lane - 1] + size_t(e.tile) * kTile, kTile * 4);
          if (lane >= 8 && lane - 8 < int(e.n_frames)) bulk_prefetch_l2(frame_at(sh.frames[ahead % kBank][lane - 8]), uint32_t(p.payload_bytes));
        }
      }
      // ---- the next window's launch may move in on SMs that run dry: its tiles are others than this launch's
      if (!handed_on && looked >= my_count && armed - finished <= 2u) {
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        handed_on = true;
      }
      // ---- watch the compute warps
      ST_CRUMB(g, 4);
      const uint32_t at = finished + uint32_t(lane);
      const uint32_t w = int32_t(armed - at) > 0 ? ld_shared_acquire(&sh.done[at % kBank]) : 0u;
      ran_out |= __any_sync(0xffffffffu, w >= kDoneFailed);
      const uint32_t ready = __ballot_sync(0xffffffffu, (w & kDoneWarps) == uint32_t(kComputeWarps));
      const uint32_t more = ready == 0xffffffffu ? 32u : uint32_t(__ffs(~ready) - 1);
      if (more) {
        __syncwarp();  // (nor does a ballot) what each lane has acquired of its tile comes before the fence and the flags of any lane
        finished += more;
        idle = 0;
      }
      const bool last = finished == armed && (looked >= my_count || yielded || aborted || ran_out);
      // ---- publish: when nothing is in hand, and earlier when half a bank has piled up, so that a neighbour does not
      // wait for the end of a long launch.  Not more often: a system-scope fence takes 1.5 us on a quiet GPU and 3.9 us as
      // soon as 37 or more SMs have one under way (measured: 2815 and 7400 cycles), and a fence that finds others under
      // way waits for those first: at the end of a launch of 296 groups it takes 1.5 to 10 us, 4.4 in the middle.  A fence
      // behind every tile made the last one of a launch take 8 us.
      // Where the far end of every ring is memory of this GPU, whoever reads the flags is within device scope, and a fence of
      // that scope takes 0.2 to 1.0 us there, 0.5 in the middle.
      if (finished != published && (finished == armed || finished - published >= uint32_t(kBank / 2))) {
        // the payloads are performed before the flags that announce them
        if (p.one_gpu) asm volatile("fence.acq_rel.gpu;" ::: "memory");
        else asm volatile("fence.acq_rel.sys;" ::: "memory");
        for (; published != finished; published += min(finished - published, uint32_t(at_once))) {
          if (int32_t(finished - published) <= t || (kLeafOnly && r != 0)) continue;
          const uint32_t entry = (published + uint32_t(t)) % kBank;
          const TileDesc d = sh.desc[entry];
          const uint32_t done = sh.done[entry], moved = sh.moved[entry][r];
          if ((moved & 4u) && ((done >> (kDoneNonsilentShift + (kOneLink ? 0 : 4 * out.link))) & 0xfu)) {
            const uint32_t seq = sh.tx[entry][r];
            st_relaxed_sys(out.flags_remote + size_t((seq - 1u) & smask) * p.n_tiles + d.tile, seq);
            st_cg_u32(out.tx_seq + d.tile, seq);
            n_tx++;
          }
          if (moved & 3u) {
            const uint32_t seq = sh.rx[entry][r];
            st_cg_u32(in.rx_seq + d.tile, seq);
            st_relaxed_sys(in.credit_remote + d.tile, seq);
            n_rx += moved & 3u;
          }
          if (r == 0) {
            bool left = done >= kDoneFailed;
            for (int l = 0; l < n_links; l++) {
              if (((done >> (kDoneNonsilentShift + 4 * l)) & 0xfu) == 0) continue;
              left = true;  // more may be left to say (or nothing could be said at all)
              if (!(d.flags & (kDescTxOk << l)) && p.do_tx) n_blocked++;
            }
            if (left) {
              st_cg_u32(p.tile_state + d.tile, 1u);
              n_pending++;
            }
            n_done++;
          }
        }
        __syncwarp();
        continue;
      }
      if (last) break;
      if (more) continue;
      if (++idle == 1024u) t_last = globaltimer_ns();
      // (The time by the clock and in looks, like the waits of the compute warps.  The second time it is longer than all the
      // waits of a compute warp in one tile: one on a stage, one per link on an exchange.)
      const bool late = __any_sync(0xffffffffu, idle > 2048u && globaltimer_ns() - t_last > (aborted ? 8 : 2) * limit_ns);
      if (late || (ran_out && !aborted)) {
        if (aborted) break;  // the tiles that had been started did not finish either
        aborted = true;
      } else if (yielded || aborted || (idle & 7u) != 0 || !update_waiting()) {
        __nanosleep(40);
        continue;
      } else {
        yielded = true;
      }
      // An update is waiting for the SMs this kernel holds, or a wait ran out: no more tiles are started.  Those that
      // were looked at but not started get their change marks back, everything else about them is untouched.
      uint32_t started = 0;
      if (lane == 0) started = atomicOr(&sh.claim, kStop) & ~kStop;
      started = __shfl_sync(0xffffffffu, started, 0);
      for (uint32_t c = started + uint32_t(lane); int32_t(armed - c) > 0; c += 32)
        if (sh.dirty[c % kBank]) st_cg_u32(p.tile_state + sh.desc[c % kBank].tile, 1u);
      armed = started;
      if (int32_t(handed - started) > 0) handed = started;
      if (int32_t(staged - handed) > 0) staged = handed;
      t_last = globaltimer_ns();
    }
    if (aborted || ran_out) break;
    n_sweeps++;
    if (armed == armed_before && sweep + 1 < p.sweeps) __nanosleep(1000);
  }
  if (lane == 0) atomicOr(&sh.claim, kStop);  // the compute warps leave
  // copies of tiles that nobody started get a bounded chance to land before the CTA's shared memory is released
  for (uint32_t q = stage_issued > 2 ? stage_issued - 2 : 0; q < stage_issued; q++)
    (void)__all_sync(0xffffffffu, mbar_wait_bounded(&sh.full[q & 1u], (q >> 1) & 1u, limit_ns));
  if (aborted || ran_out) {
    for (int j = lane; j < my_count; j += 32) st_cg_u32(p.tile_state + gid + j * gstride, 1u);
    if (lane == 0) {
      atomicOr(reinterpret_cast<unsigned long long*>(p.status + kDsErrors), (unsigned long long)kErrBarrierTimeout);
      atomicAdd(reinterpret_cast<unsigned long long*>(p.status + kDsWaitTimeouts), 1ull);
    }
  }
  // A launch that was let in early ends after the one before it, so that what follows in the stream finds both complete.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  n_done = __reduce_add_sync(0xffffffffu, n_done);
  n_tx = __reduce_add_sync(0xffffffffu, n_tx);
  n_rx = __reduce_add_sync(0xffffffffu, n_rx);
  n_blocked = __reduce_add_sync(0xffffffffu, n_blocked);
  n_pending = __reduce_add_sync(0xffffffffu, n_pending);
  open = __any_sync(0xffffffffu, open);
  if (lane == 0) {
    ST_CRUMB(g, 10);
    auto count = [&](uint64_t* w, unsigned long long by) {
      if (by) atomicAdd(reinterpret_cast<unsigned long long*>(w), by);
    };
    count(p.status + kDsYields, yielded ? 1 : 0);
    count(p.status + kDsTilesProcessed, n_done);
    count(p.status + kDsFramesSent, n_tx);
    count(p.status + kDsFramesRecv, n_rx);
    count(p.status + kDsBlockedNoCredit, n_blocked);
    count(p.status + kDsUnacknowledged, open ? 1 : 0);
    count(launch_words + kDlWork, n_done);
    count(launch_words + kDlPending, n_pending);
    if (blockIdx.x == 0 && g == 0) {
      count(p.status + kDsSweeps, n_sweeps);
      uint64_t* rec = p.status + kDsTrace + (uint64_t(p.round) % kTraceEntries) * kTraceWords;  // trace ring, read by stats()
      rec[0] = globaltimer_ns();
      rec[1] = uint64_t(p.round);
      rec[2] = n_done;
      rec[3] = sent_before + n_tx;
    }
  }
}

}  // namespace

template <int Q, int kKind>
__global__ void __launch_bounds__(kRoundGroups * kGroupThreads, 1) round_kernel(const __grid_constant__ RoundParams p) {
  __shared__ GroupShared shared[kRoundGroups];
  extern __shared__ __align__(128) uint8_t dynamic[];  // [group][two stages of frames], and for an inner node [group][link][element of the tile]
  constexpr int kIn = kStaged<kKind>, kStageBytes = 2 * kIn * kFrameRoom<Q>;
  const int g = int(threadIdx.x) / kGroupThreads, warp = (int(threadIdx.x) % kGroupThreads) >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x < kRoundGroups) {
    GroupShared& sh = shared[threadIdx.x];
    sh.armed = 0;
    sh.claim = 0;
    sh.exchanged = 0;
    mbar_init(&sh.gsync, kComputeWarps);
    for (int u = 0; u < 2; u++) {
      mbar_init(&sh.full[u], 1);
      mbar_init(&sh.empty[u], kComputeWarps);
    }
    if (kIn > 0) {  // (bulk copies will complete on them)
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
  }
  if (!p.follows_window) asm volatile("griddepcontrol.wait;" ::: "memory");
  __syncthreads();  // the only CTA-wide barrier: from here on the groups, and the two kinds of warp, run on their own
  uint8_t* const stages = dynamic + g * kStageBytes;
  float* const stash = reinterpret_cast<float*>(dynamic + kRoundGroups * kStageBytes) + (kKind == kInner ? g * kMaxLinks * kTile : 0);
  if (warp == kComputeWarps) service_warp<Q, kKind>(p, shared[g], stages, kIn, kFrameRoom<Q>, g, kRoundGroups, lane);
  else compute_warp<Q, kKind>(p, shared[g], stash, stages, warp, lane);
}

// ----------------------------------------------------------------------------------------------
// Taking frames back.  When a neighbour is lost, the frames it never acknowledged (sequence numbers from its last
// credit up to what was sent) are still in its ring, which stays mapped here; their steps come off the mirror again,
// so that what they said counts as not yet told (the TCP edges do the same with a frame whose write fails).
// One CTA per tile, warp w its 512 elements, the same lane layout as the round kernel.
// ----------------------------------------------------------------------------------------------
template <int Q>
__global__ void __launch_bounds__(kComputeWarps * 32) unsend_kernel(float* __restrict__ mirror, const uint8_t* __restrict__ payload,
                                                                    uint32_t* __restrict__ tx_seq, const uint32_t* __restrict__ credit,
                                                                    int n_tiles, int ring_slots, int pb, int log2_block, int64_t n,
                                                                    unsigned long long* __restrict__ taken_back) {
  const int tile = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t c = ld_acquire_sys(credit + tile), tx = ld_cg_u32(tx_seq + tile);
  const uint32_t count = tx - c;
  if (count == 0 || count > uint32_t(ring_slots)) return;
  const int in_tile = warp * kWarpElems + lane * 4, left = int(min(int64_t(kTile), n - int64_t(tile) * kTile)) - in_tile;
  Piece acc[kPieces];
#pragma unroll
  for (int i = 0; i < kPieces; i++) acc[i] = {0ull, 0ull};
  for (uint32_t f = 0; f < count; f++) {
    FrameRegs fr;
    load_frame<Q>(payload + (size_t((c + f) & uint32_t(ring_slots - 1)) * n_tiles + tile) * pb, warp, lane, log2_block, fr);
#pragma unroll
    for (int i = 0; i < kPieces; i++) add4(acc[i], frame_steps<Q>(fr.w[i], fr.code(i), Q == 1 ? valid4(left, i) : 0xfu));
  }
  float* const kp = mirror + size_t(tile) * kTile + in_tile;
#pragma unroll
  for (int i = 0; i < kPieces; i++) {
    const Piece k = load_piece(kp + i * 128);
    store_piece(kp + i * 128, {sub2(k.a, acc[i].a), sub2(k.b, acc[i].b)});
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    st_cg_u32(tx_seq + tile, c);
    atomicAdd(taken_back, (unsigned long long)count);
  }
}

int launch_unsend(float* mirror, const uint8_t* payload_remote, uint32_t* tx_seq, const uint32_t* credit, int n_tiles, int ring_slots,
                  int payload_bytes, int log2_block, int bits, int64_t n, uint64_t* taken_back, void* stream_v) {
  cudaStream_t s = static_cast<cudaStream_t>(stream_v);
  unsigned long long* tb = reinterpret_cast<unsigned long long*>(taken_back);
  switch (bits) {
    case 1: unsend_kernel<1><<<n_tiles, kComputeWarps * 32, 0, s>>>(mirror, payload_remote, tx_seq, credit, n_tiles, ring_slots, payload_bytes, log2_block, n, tb); break;
    case 2: unsend_kernel<2><<<n_tiles, kComputeWarps * 32, 0, s>>>(mirror, payload_remote, tx_seq, credit, n_tiles, ring_slots, payload_bytes, log2_block, n, tb); break;
    case 4: unsend_kernel<4><<<n_tiles, kComputeWarps * 32, 0, s>>>(mirror, payload_remote, tx_seq, credit, n_tiles, ring_slots, payload_bytes, log2_block, n, tb); break;
    case 8: unsend_kernel<8><<<n_tiles, kComputeWarps * 32, 0, s>>>(mirror, payload_remote, tx_seq, credit, n_tiles, ring_slots, payload_bytes, log2_block, n, tb); break;
    default: return int(cudaErrorInvalidValue);
  }
  return int(cudaGetLastError());
}

// ----------------------------------------------------------------------------------------------
// launcher
// ----------------------------------------------------------------------------------------------
template <int Q, int kKind>
constexpr int kDynamicBytes = kRoundGroups * (2 * kStaged<kKind> * kFrameRoom<Q> + (kKind == kInner ? kMaxLinks * kTile * 4 : 0));

// Loads the kernel and, once per device, gives it its shared memory.
template <int Q, int kKind>
static int load_round_l() {
  static std::atomic<uint64_t> loaded{0};
  int dev = 0;
  cudaGetDevice(&dev);
  if ((loaded.load(std::memory_order_relaxed) >> (dev & 63)) & 1u) return 0;
  const cudaError_t e = cudaFuncSetAttribute(round_kernel<Q, kKind>, cudaFuncAttributeMaxDynamicSharedMemorySize, kDynamicBytes<Q, kKind>);
  if (e == cudaSuccess) loaded.fetch_or(1ull << (dev & 63), std::memory_order_relaxed);
  return int(e);
}

template <int Q, int kKind>
static int launch_round_l(const RoundParams& p, int ctas, cudaStream_t stream) {
  if (const int e = load_round_l<Q, kKind>()) return e;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(kRoundGroups * kGroupThreads);
  cfg.dynamicSmemBytes = kDynamicBytes<Q, kKind>;
  cfg.stream = stream;
  // The launch may move in while the kernel before it in the stream is running out (and is cheaper to issue so: 2.4 instead
  // of 2.9 us).  A window that follows another of its cycle starts at once: the two have no tile in common.  Any other launch
  // waits for the stream first.  (A cycle's last window clears the counters of the cycle before, which was
  // complete when this cycle's first window began.)
  cudaLaunchAttribute early{};
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &early;
  cfg.numAttrs = 1;
  return int(cudaLaunchKernelEx(&cfg, round_kernel<Q, kKind>, p));
}

// `ctas` == 0: only loads the kernel
template <int Q>
static int launch_round_q(const RoundParams& p, int ctas, cudaStream_t stream) {
  if (p.n_links > 1) return ctas ? launch_round_l<Q, kInner>(p, ctas, stream) : load_round_l<Q, kInner>();
  if (p.n_in > 1) return ctas ? launch_round_l<Q, kMember>(p, ctas, stream) : load_round_l<Q, kMember>();
  return ctas ? launch_round_l<Q, kLeaf>(p, ctas, stream) : load_round_l<Q, kLeaf>();
}

static int launch_round_any(const RoundParams& p, int ctas, cudaStream_t stream) {
  switch (p.bits) {
    case 1: return launch_round_q<1>(p, ctas, stream);
    case 2: return launch_round_q<2>(p, ctas, stream);
    case 4: return launch_round_q<4>(p, ctas, stream);
    case 8: return launch_round_q<8>(p, ctas, stream);
    default: return int(cudaErrorInvalidValue);
  }
}

int load_round(const RoundParams& p) { return launch_round_any(p, 0, nullptr); }

int launch_round(const RoundParams& p, int ctas, void* stream_v) {
  if (p.n_links < 1 || p.n_links > kMaxLinks || p.sweeps < 1 || ctas < 1) return int(cudaErrorInvalidValue);
  if (p.ring_slots < 2 || p.ring_slots > 64 || (p.ring_slots & (p.ring_slots - 1))) return int(cudaErrorInvalidValue);
  return launch_round_any(p, ctas, static_cast<cudaStream_t>(stream_v));
}

}  // namespace st
