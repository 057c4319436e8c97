// ewf_umma.h -- operand layout and descriptors of the surrogate's tcgen05 (UMMA) GEMM
// (host and device code; the host side is exercised by tests/test_umma_*_cpu.py).
//
// One CTA computes tiles of C = A . B^T, up to BM rows each, from bf16 operands that are stored K-major, A [M, K]
// and B [N, K], or transposed (below).  Of a K-major operand a k-stage of BK = 64 elements (128 bytes of every operand row) is brought into shared memory
// by one 2-D TMA copy with the 128-byte swizzle: row r of a stage tile occupies bytes
// [r * 128, r * 128 + 128) and its 16-byte chunk c sits at chunk c ^ (r % 8).  That is the
// tensor core's canonical K-major SWIZZLE_128B layout: 8-row atoms of 1024 bytes, one after the
// other (stride-dimension offset 1024 B), and the k-th MMA of a stage (K = 16, 32 bytes of each
// row) starts its descriptors 32 k bytes into the atom.  Stage tiles start on 1024-byte
// boundaries, so the descriptors' base offset is 0.
//
// Shared-memory matrix descriptor (64 bit): start address >> 4 in bits 0-13, leading-dimension
// byte offset >> 4 in bits 16-29 (not used by swizzled K-major layouts; 16 B), stride-dimension
// byte offset >> 4 in bits 32-45, descriptor version 1 in bits 46-47, base offset 0 (bits
// 49-51), layout type in bits 61-63 (2 = SWIZZLE_128B).
// Instruction descriptor (32 bit, kind::f16): D format F32 (1) in bits 4-5, A and B format BF16
// (1) in bits 7-9 and 10-12, both K-major (bits 15, 16 = 0), N >> 3 in bits 17-22, M >> 4 in
// bits 24-28; bits 15 and 16 are set for operands stored MN-major.
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define EWF_UHD __host__ __device__ __forceinline__
#else
#define EWF_UHD inline
#endif

namespace ewf_umma {

constexpr int BM = 128;          // rows of A per CTA tile (TMEM lanes of the accumulator)
constexpr int BK = 64;           // K per pipeline stage: 128 bytes per operand row
constexpr int STAGES = 4;        // slots of the ring of 128-row tiles 256 columns wide; narrower tiles have more
constexpr int ROW_BYTES = BK * 2;
constexpr int ATOM_BYTES = 8 * ROW_BYTES;  // 8 rows x 128 B: the swizzle atom, stride-dimension offset
constexpr int MMA_K = 16;
constexpr int THREADS = 192;     // warp 0: TMA producer of A; warp 1: MMA issuer; warps 2-5: epilogue
constexpr int MORE_EPILOGUE = 128;  // warps 6-9: a second epilogue warp per TMEM lane quarter (warp 10: the producer of B)
constexpr int LAYOUT_SW128 = 2;

// Per tile width BN (128 or 256): bytes of a stage and of the whole pipeline; TMEM columns = 2 BN
// (two accumulators).
EWF_UHD constexpr int a_bytes() { return BM * ROW_BYTES; }
EWF_UHD constexpr int b_bytes(int bn) { return bn * ROW_BYTES; }
EWF_UHD constexpr int stage_bytes(int bn) { return a_bytes() + b_bytes(bn); }
EWF_UHD constexpr int smem_bytes(int bn) { return STAGES * stage_bytes(bn) + 1024; }  // + alignment slack

EWF_UHD uint64_t smem_desc_sw128(uint32_t smem_addr)
{
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr >> 4) & 0x3FFFu);
    d |= (uint64_t)(16 >> 4) << 16;
    d |= (uint64_t)((ATOM_BYTES >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;  // version
    d |= (uint64_t)LAYOUT_SW128 << 61;
    return d;
}

// An operand stored transposed, [K, rows] with the rows contiguous ("MN-major"): a k-stage is one
// TMA box of 64 rows x BK per block of 64 rows (blocks BK * 128 = 8192 bytes apart), the box's row k
// being k's 64 values, 128 bytes, swizzled as above.  The canonical layout's 8-k groups are then 1024
// bytes apart (stride-dimension offset) and its 64-row atoms 8192 (leading-dimension offset); the
// k-th MMA of a stage starts 16 k rows, 2048 k bytes, into the block.
constexpr int MN_ATOM = 64;
constexpr int MN_BLOCK_BYTES = BK * ROW_BYTES;
constexpr int MN_K_STEP = MMA_K * ROW_BYTES;
EWF_UHD uint64_t smem_desc_sw128_mn(uint32_t smem_addr)
{
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr >> 4) & 0x3FFFu);
    d |= (uint64_t)((MN_BLOCK_BYTES >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((ATOM_BYTES >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;  // version
    d |= (uint64_t)LAYOUT_SW128 << 61;
    return d;
}
// where that layout has the 2-byte element (row mn, k) of an operand block, from the block's start
EWF_UHD uint32_t mn_offset(int mn, int k)
{
    const uint32_t b = (uint32_t)(mn / MN_ATOM) * MN_BLOCK_BYTES + (uint32_t)(k / 8) * ATOM_BYTES + (uint32_t)(k % 8) * ROW_BYTES +
                       (uint32_t)(mn % MN_ATOM) * 2;
    return b ^ (((b >> 7) & 7) << 4);
}

EWF_UHD uint32_t instr_desc_bf16_f32(int m, int n);
EWF_UHD uint32_t instr_desc_bf16_f32(int m, int n, bool a_mn, bool b_mn)
{
    return instr_desc_bf16_f32(m, n) | (a_mn ? 1u << 15 : 0u) | (b_mn ? 1u << 16 : 0u);
}

EWF_UHD uint32_t instr_desc_bf16_f32(int m, int n)
{
    uint32_t d = 0;
    d |= 1u << 4;   // D: F32
    d |= 1u << 7;   // A: BF16
    d |= 1u << 10;  // B: BF16
    d |= (uint32_t)((n >> 3) & 0x3F) << 17;
    d |= (uint32_t)((m >> 4) & 0x1F) << 24;
    return d;
}

// The end of the byte range an MMA of a stage reads from one operand tile of `rows` rows: every
// 8-row atom from the start address (32 k bytes into the first row) on, to the end of the last
// row's 32-byte K slice.
EWF_UHD uint32_t mma_read_end(uint32_t start, int rows)
{
    return start + (uint32_t)(rows / 8 - 1) * ATOM_BYTES + 7 * ROW_BYTES + 32;
}

// Phase bookkeeping of the GEMM's mbarriers.  An mbarrier wait with parity P returns once the
// barrier's current phase has a parity other than P, i.e. once the latest completed phase has
// parity P; a fresh barrier (phase 0 running) therefore lets a parity-1 wait through at once.
// Stage ring of `stages` slots: the g-th k-stage of a CTA (counted across its tiles) uses slot g % stages; its
// "full" completion is that slot's (g / stages)-th, its "empty" completion frees the slot for
// stage g + stages.  Accumulators: the i-th tile of a CTA uses buffer i % 2; "acc_full" completes
// once per tile in that buffer, "acc_empty" once per drained tile.
// The kernel's roles keep a slot and a parity and move on with ring_next; ring_slot and ring_full_parity serve its
// last waits, and ring_needs_free and ring_free_parity the host model of a single producer.
EWF_UHD int ring_slot(int g, int stages = STAGES) { return g % stages; }
EWF_UHD uint32_t ring_full_parity(int g, int stages = STAGES) { return (uint32_t)(g / stages) & 1u; }  // consumer of stage g
EWF_UHD bool ring_needs_free(int g, int stages = STAGES) { return g >= stages; }                       // producer of stage g waits?
EWF_UHD uint32_t ring_free_parity(int g, int stages = STAGES) { return (uint32_t)(g / stages - 1) & 1u; }  // ... for stage g - stages
// The slot after `s` in a ring of ns, and the parity of its wait (it toggles each time round).
EWF_UHD void ring_next(int s, uint32_t parity, int ns, int *s1, uint32_t *p1)
{
    *s1 = s + 1 == ns ? 0 : s + 1;
    *p1 = *s1 ? parity : parity ^ 1u;
}
EWF_UHD int acc_buf(int i) { return i & 1; }
EWF_UHD uint32_t acc_full_parity(int i) { return (uint32_t)(i >> 1) & 1u; }              // epilogue of tile i
EWF_UHD bool acc_needs_free(int i) { return i >= 2; }                                     // MMAs of tile i wait?
EWF_UHD uint32_t acc_free_parity(int i) { return (uint32_t)((i >> 1) - 1) & 1u; }        // ... for tile i - 2

// A warp's wait of at most `limit` polls.  Each lane polls for itself and nothing says that two lanes of a poll
// see the same, so the warp decides together -- vote(x): whether x holds in every lane.  Lanes that each went by their
// own poll could part as the limit ends, some leaving the role's loop and the others waiting for them there
// (elect.sync, __syncwarp) for good.
template <class Poll, class Failed, class Vote>
EWF_UHD bool warp_wait(int limit, Poll poll, Failed failed, Vote vote)
{
    for (int i = 0; i < limit; ++i) {
        if (vote(poll())) return true;
        if ((i & 1023) == 1023 && !vote(!failed())) return false;
    }
    return false;
}

// The last wait for copies or MMAs that a role issued itself, before the CTA's memory goes: they land within
// microseconds, and the polls (which do not suspend the thread) take milliseconds.  A copy's barrier need not complete:
// where the other operand's producer gave up first, its arrival never comes.
constexpr int DRAIN_POLLS = 1 << 18;
template <class Poll>
EWF_UHD void bounded_drain(Poll poll, int polls = DRAIN_POLLS)
{
    for (int i = 0; i < polls; ++i)
        if (poll()) return;
}

}  // namespace ewf_umma
