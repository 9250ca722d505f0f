// Building blocks of the kernels on the fifth-generation tensor cores (w4a16_tc.cu,
// w4a16_rows.cu): tensor-memory and MMA instructions, operand descriptors, the bounded
// wait, the int4 -> bf16 conversion in natural k order, and the cached tensor-map encoder.
#pragma once

#include <cuda.h>

#include "common.cuh"

namespace cb200 {

constexpr int kTcRowsPerTile = 128;  // weight rows of one MMA tile (its M dimension)
constexpr unsigned long long kTcWaitNs = 400000000ull;

// A 2-D tensor map: `inner` x `outer` elements with a row pitch of inner * esize bytes, box
// `box_inner` x `box_outer`.  kind 0: packed weights as uint32, 128-byte swizzle; 1:
// activations as bf16, 128-byte swizzle; 2: outputs as bf16, no swizzle.
int tc_encode(const void* base, int inner, int outer, int box_inner, int box_outer, int kind,
              CUtensorMap* out);
// Activations as bf16 [inner/64][outer][64], 128-byte swizzle, box `box_blocks` x `box_rows`
// x 64: one copy brings several blocks of 64 k, each in the MMA's operand layout.
int tc_encode_blocks(const void* base, int inner, int outer, int box_rows, int box_blocks, CUtensorMap* out);

// ---------------------------------------------------------------------------
// tcgen05 wrappers
// ---------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(std::uint32_t* smem_slot, std::uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_slot)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(std::uint32_t taddr, std::uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_commit(std::uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]; accumulate = 0 overwrites D.
__device__ __forceinline__ void tc_mma_ts(std::uint32_t d_tmem, std::uint32_t a_tmem,
                                          std::uint64_t b_desc, std::uint32_t idesc,
                                          std::uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
      :
      : "r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u)
      : "memory");
}
// The eight K=16 MMAs of one quantisation group in one go: D = A[:, 0:16) * B0 and
// then D += A[:, 16j:16j+16) * Bj.  A advances 8 columns per MMA; the B descriptor's
// start-address field (units of 16 bytes) advances 32 bytes per MMA inside an
// activation box and `box_step16` between the group's two boxes.  Issuing a
// tcgen05.mma costs the issuing thread on the order of a hundred cycles, so
// nothing else is computed between them.
__device__ __forceinline__ void tc_mma_group(std::uint32_t d_tmem, std::uint32_t a_tmem,
                                             std::uint32_t desc_lo, std::uint32_t desc_hi,
                                             std::uint32_t box_step16, std::uint32_t idesc) {
  asm volatile(
      "{\n\t"
      ".reg .pred pf, pt;\n\t"
      ".reg .b32 lo, aa;\n\t"
      ".reg .b64 bd;\n\t"
      "setp.ne.b32 pf, 0, 0;\n\t"
      "setp.eq.b32 pt, 0, 0;\n\t"
      "mov.b64 bd, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], bd, %5, pf;\n\t"
      "add.u32 lo, %2, 2;\n\t mov.b64 bd, {lo, %3};\n\t add.u32 aa, %1, 8;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [aa], bd, %5, pt;\n\t"
      "add.u32 lo, %2, 4;\n\t mov.b64 bd, {lo, %3};\n\t add.u32 aa, %1, 16;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [aa], bd, %5, pt;\n\t"
      "add.u32 lo, %2, 6;\n\t mov.b64 bd, {lo, %3};\n\t add.u32 aa, %1, 24;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [aa], bd, %5, pt;\n\t"
      "add.u32 lo, %2, %4;\n\t mov.b64 bd, {lo, %3};\n\t add.u32 aa, %1, 32;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [aa], bd, %5, pt;\n\t"
      "add.u32 lo, lo, 2;\n\t mov.b64 bd, {lo, %3};\n\t add.u32 aa, %1, 40;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [aa], bd, %5, pt;\n\t"
      "add.u32 lo, lo, 2;\n\t mov.b64 bd, {lo, %3};\n\t add.u32 aa, %1, 48;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [aa], bd, %5, pt;\n\t"
      "add.u32 lo, lo, 2;\n\t mov.b64 bd, {lo, %3};\n\t add.u32 aa, %1, 56;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [aa], bd, %5, pt;\n\t"
      "}"
      :
      : "r"(d_tmem), "r"(a_tmem), "r"(desc_lo), "r"(desc_hi), "r"(box_step16), "r"(idesc)
      : "memory");
}
// 16 consecutive 32-bit columns of this thread's lane
__device__ __forceinline__ void tmem_st16(std::uint32_t taddr, const std::uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_ld16_nowait(std::uint32_t taddr, std::uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld32_nowait(std::uint32_t taddr, std::uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld64_nowait(std::uint32_t taddr, std::uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x64.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47,%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63}, [%64];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]), "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]), "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]), "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]), "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// NCOL consecutive accumulator columns of this thread's lane, one instruction, one wait
template <int NCOL>
__device__ __forceinline__ void tmem_ld_cols(std::uint32_t taddr, std::uint32_t* r) {
  if (NCOL == 64) tmem_ld64_nowait(taddr, r);
  else if (NCOL == 32) tmem_ld32_nowait(taddr, r);
  else tmem_ld16_nowait(taddr, r);
  tmem_ld_wait();
}

// Shared-memory matrix descriptor of one K=16 slice of the B operand inside an
// activation box: K-major, 128-byte swizzle (rows of 128 bytes, eight rows per
// 1024-byte swizzle atom, so 1024 bytes between 8-row groups); the slice is
// selected by adding its byte offset (32 bytes per K=16) to the start address.
// Descriptor version 1.
__device__ __forceinline__ std::uint64_t tc_b_desc(std::uint32_t smem_addr) {
  std::uint64_t d = 0;
  d |= static_cast<std::uint64_t>((smem_addr & 0x3FFFFu) >> 4);
  d |= static_cast<std::uint64_t>(1u) << 16;            // leading byte offset: unused with a swizzle
  d |= static_cast<std::uint64_t>(1024u >> 4) << 32;    // stride byte offset
  d |= static_cast<std::uint64_t>(1u) << 46;            // version
  d |= static_cast<std::uint64_t>(2u) << 61;            // 128-byte swizzle
  return d;
}

// Instruction descriptor: D fp32, A and B bf16, both K-major, M = 128, N = ntok.
__host__ __device__ constexpr std::uint32_t tc_idesc(int ntok) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<std::uint32_t>(ntok >> 3) << 17) |
         (static_cast<std::uint32_t>(kTcRowsPerTile >> 4) << 24);
}

// Bounded, abort-aware wait.  Returns false when the wait ran out or another
// thread of the CTA already gave up.
__device__ __forceinline__ bool tc_wait(std::uint64_t* bar, std::uint32_t parity,
                                        volatile int* abort_flag) {
  if (mbar_try_wait(bar, parity)) return true;
  unsigned long long t0;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
  for (;;) {
    for (int i = 0; i < 64; ++i) {
      if (mbar_try_wait(bar, parity)) return true;
    }
    if (*abort_flag) return false;
    unsigned long long t1;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t1));
    if (t1 - t0 > kTcWaitNs) {
      *abort_flag = 1;
      return false;
    }
  }
}

// int4 word (k = 8w .. 8w+7, nibble i at bits 4i) -> four exact bf16 pairs
// {q(k), q(k + 1)}, k = 8w, 8w+2, 8w+4, 8w+6, in the natural order of k so that
// the activations need no rearrangement.  Byte b of the word holds nibbles 2b
// (low) and 2b+1 (high); in w >> 4 the same byte position holds nibble 2b+1 in
// its low four bits.  PRMT puts byte b of w into the low half of a register and
// byte b of w >> 4 into the high half; one LOP3 keeps the two low nibbles, flips
// their sign bits (two's complement n -> offset binary u = q + 8) and ORs in the
// bf16 pattern of 128, whose seven mantissa bits then hold u: {128 + u0,
// 128 + u1}, exact; subtracting {136, 136} leaves {q0, q1}, exact.
__device__ __forceinline__ void dequant_word_natural(std::uint32_t w, std::uint32_t* out) {
  const std::uint32_t w4 = w >> 4;
  constexpr std::uint32_t kMagic = 0x43084308u;  // {136, 136} = {128 + 8, 128 + 8}
  out[0] = sub_bf16x2(lop3_and_xor(__byte_perm(w, w4, 0x4400u), 0x000F000Fu, kMagic), kMagic);
  out[1] = sub_bf16x2(lop3_and_xor(__byte_perm(w, w4, 0x5511u), 0x000F000Fu, kMagic), kMagic);
  out[2] = sub_bf16x2(lop3_and_xor(__byte_perm(w, w4, 0x6622u), 0x000F000Fu, kMagic), kMagic);
  out[3] = sub_bf16x2(lop3_and_xor(__byte_perm(w, w4, 0x7733u), 0x000F000Fu, kMagic), kMagic);
}

// two floats rounded to nearest even into one word of bf16 values (lo in the low half)
__device__ __forceinline__ std::uint32_t pack_bf16x2(float lo, float hi) {
  std::uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

}  // namespace cb200
