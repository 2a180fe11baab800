// Tiles with two cells per byte: rule sets with a block transition table of 4-bit keys.
//
// A row of the shared array is a row of 32-bit words of eight 4-bit ids.  One lane updates a
// chunk: the eight horizontally adjacent blocks (16 x 2 cells) that two words of a row and
// the words below them hold, read shifted by one cell on frames whose blocks start at odd
// columns.  A warp takes LX x LY chunks side by side, leaves them alone when all are one
// static material, and otherwise evaluates all of them at once.
//
// The reduced table holds a block's result for either outcome of the mirror test in a
// half-word each (a | b << 4 | c << 8 | d << 12: the low byte is the block's part of the
// upper row, the high byte that of the lower row), or 0xffff where the result also depends on
// another hash comparison.  Warps that meet such blocks (about one block in 30 in the
// twelve-material workload, fewer as it settles) look up their results for hash values above
// every constant they depend on, with the bound below which that does not hold, and hash that
// lane; the few blocks below their bound take the full table.  So a block costs one hash lane
// and one lookup, which does not wait for the hash.
//
// On the CPU the code runs with one thread per CTA and without the reduced tables, or, with
// SE_WHOLE_WARPS, with its real thread counts and tables.
#pragma once

#ifdef SE_NIB
// A block's four 4-bit ids in row order (a | b << 4 | c << 8 | d << 12) from column order
// (a | c << 4 | b << 8 | d << 12, the full table's keys and entries), and back.
__device__ __forceinline__ uint32_t se_nib_swap_order(uint32_t k) {
  return (k & 0xf00fu) | ((k & 0x00f0u) << 4) | ((k >> 4) & 0x00f0u);
}

// The two results of the block with row-order key `key`, for hash values above every constant
// it depends on (x), and the largest value of the other hash lane below the last of them, 0
// when there is none (y).  The lane is compared before its last mixing step, which leaves the
// top 16 bits alone, so the bound's low 16 bits are all ones.
__device__ __forceinline__ uint2 se_nib_bound(const uint16_t* __restrict__ lut, uint32_t key) {
  const uint32_t base = se_nib_swap_order(key) * SE_NIB_CLASSES;
  uint2 out = make_uint2(0u, 0u);
  for (uint32_t m = 0; m < 2u; ++m) {
    uint32_t val = 0;
    bool any = false;
    for (uint32_t q = SE_NIB_CLASSES; q-- > 0u;) {  // from the highest class down
      uint32_t a, b, c, d, h[4];
      se_gen::lut_decode(base + q, a, b, c, d, h[0], h[1], h[2], h[3]);
      if ((h[0] >= 0x7fffffc0u) != (m != 0u)) continue;
      const uint32_t o = lut[base + q];
      if (!any) {
        val = o;
        any = true;
      } else if (o != val) {
        uint32_t t = 0xffffffffu;
        if (SE_NIB_LANE) {  // class q + 1 of the lane is the lowest of those found equal
          se_gen::lut_decode(base + q + 1u, a, b, c, d, h[0], h[1], h[2], h[3]);
          t = (h[SE_NIB_LANE] - 1u) | 0xffffu;
        }
        if (t > out.y) out.y = t;
        break;
      }
    }
    out.x |= se_nib_swap_order(val) << (16 * m);
  }
  return out;
}
// The reduced table's entry.
__device__ __forceinline__ uint32_t se_nib_entry(const uint16_t* __restrict__ lut, uint32_t key) {
  const uint2 e = se_nib_bound(lut, key);
  return e.y ? 0xffffffffu : e.x;
}
// The static-material mask: bit m + 16 (m & 1) is set when the block of four m cells is
// static.  That is the bit that a word of eight m cells selects with its low 5 bits.
__device__ __forceinline__ uint32_t se_nib_static_mask(const uint16_t* __restrict__ lut) {
  const uint32_t* st = reinterpret_cast<const uint32_t*>(reinterpret_cast<const uint8_t*>(lut) + SE_LUT_STATIC_OFF);
  uint32_t mask = 0;
  for (uint32_t m = 0; m < SE_NMAT; ++m) {
    const uint32_t key = m * 0x1111u;
    mask |= ((st[key >> 5] >> (key & 31u)) & 1u) << (m + 16u * (m & 1u));
  }
  return mask;
}
// Fills the tables after se_build_lut and se_build_static.
extern "C" __global__ void __launch_bounds__(256) se_build_nib(uint16_t* __restrict__ lut) {
  uint32_t* out = reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(lut) + SE_NIB_OFF);
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < SE_NIB_ENTRIES) {
    const uint32_t n = SE_NMAT, a = i % n, b = i / n % n, c = i / (n * n) % n, d = i / (n * n * n);
    out[i] = se_nib_entry(lut, SE_NIB_SHARED ? a | (b << 4) | (c << 8) | (d << 12) : i);
  }
  if (SE_NIB_PROB && i < 65536u) {
    const uint2 e = se_nib_bound(lut, i);
    out[SE_NIB_BOUNDS + 2 * i] = e.x;
    out[SE_NIB_BOUNDS + 2 * i + 1] = e.y;
  }
  if (i == 0) out[SE_NIB_ENTRIES] = se_nib_static_mask(lut);
}

// Geometry of a tile's shared array: TW x TH cells and their halo, the width rounded up to
// whole chunks, the height to whole groups of LY block rows plus one row, so that every lane
// of every item has a chunk to read (the cells beyond start as WALL and only ever matter to
// the halo's outermost cells, which are inexact from the first frame on in any case).  The
// row stride is 2 mod 4 words with at least one word of padding: the 8-byte accesses of half
// a warp (LX = 2: two chunks of eight block rows) then touch 32 different banks.
template <int TW, int TH, int KMAX>
struct SeNib {
  static constexpr int HX = ((KMAX + 3) / 4) * 4, HY = KMAX;
  static constexpr int LX = 2, LY = 16;  // a warp takes LX chunks of LY block rows: 32 x 32 cells
  static constexpr int SW = ((TW + 2 * HX + 15) / 16) * 16, SH = TH + 2 * HY;
  static constexpr int CPR = (SW / 16 + LX - 1) / LX * LX, WPR = 2 * CPR;  // chunks, words a row
  static constexpr int STRIDE = WPR + 2;
  static_assert(WPR % 4 == 0, "a row's chunks come in pairs");
  static constexpr int NG = ((SH + 1) / 2 + LY - 1) / LY, ROWS = 2 * LY * NG + 1;
  static constexpr int TABLE = (STRIDE * ROWS + 3) & ~3;  // the reduced table's first word
  static constexpr int HIT = TABLE + (SE_NIB_SHARED ? (SE_NIB_ENTRIES + 3) & ~3 : 0);  // that of the edits' bits
};

// __byte_perm for selectors whose digits are at most 7.
__device__ __forceinline__ uint32_t se_prmt(uint32_t a, uint32_t b, uint32_t s) {
#if defined(__CUDA_ARCH__)
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(s));
  return r;
#else
  return __byte_perm(a, b, s);
#endif
}
__device__ __forceinline__ int se_max3(int a, int b, int c) {
#if defined(__CUDA_ARCH__)
  return __vimax3_s32(a, b, c);
#else
  return se_max(a, se_max(b, c));
#endif
}
__device__ __forceinline__ uint32_t se_max3u(uint32_t a, uint32_t b, uint32_t c) {
#if defined(__CUDA_ARCH__)
  return __vimax3_u32(a, b, c);
#else
  return se_max(a, se_max(b, c));
#endif
}
// 0x00ff where a is negative | 0xff00 where b is (as signed numbers).
__device__ __forceinline__ uint32_t se_signs(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, 0xfb;" : "=r"(r) : "r"(a), "r"(b));  // sign of byte 3, of byte 7
  return r & 0xffffu;
#else
  return ((a >> 31) * 0x00ffu) | ((b >> 31) * 0xff00u);
#endif
}

// Copies a shared reduced table into shared memory, 16 bytes a thread and step, asynchronously
// (both ends hold whole groups of four words); se_nib_table_ready before the barrier.
__device__ __forceinline__ void se_nib_copy_table(uint32_t* tab, const uint32_t* __restrict__ gtab, int nt) {
#if SE_NIB_SHARED && defined(SE_WHOLE_WARPS)
  for (int i = threadIdx.x; i < ((SE_NIB_ENTRIES + 3) & ~3); i += nt) tab[i] = gtab[i];
#elif SE_NIB_SHARED && defined(__CUDA_ARCH__)
  for (int i = threadIdx.x; i < (SE_NIB_ENTRIES + 3) / 4; i += nt)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(
                     (unsigned)__cvta_generic_to_shared(tab + 4 * i)),
                 "l"(gtab + 4 * i)
                 : "memory");
#endif
}
__device__ __forceinline__ void se_nib_table_ready() {
#if SE_NIB_SHARED && defined(__CUDA_ARCH__)
  asm volatile("cp.async.wait_all;" ::: "memory");
#endif
}

// The reduced table's entries of the four blocks of row words T and B.
template <int NT>
__device__ __forceinline__ void se_nib_lookup(uint32_t T, uint32_t B, uint32_t e[4], const uint32_t* tab,
                                              const uint32_t* __restrict__ gtab, const uint16_t* __restrict__ lut) {
  if (NT == 1) {  // emulated without the reduced table
    for (int j = 0; j < 4; ++j)
      e[j] = se_nib_entry(lut, ((T >> (8 * j)) & 0xffu) | (((B >> (8 * j)) & 0xffu) << 8));
  } else {
#if SE_NIB_SHARED
    // bytes a | b << 4 -> 4 (a + n b) (below 256), then the entries' byte offsets
    // 4 (pT + n^2 pB) (below 65536), two to a word
    constexpr uint32_t n = SE_NMAT;
    const uint32_t pT = T * 4u - ((T >> 4) & 0x0f0f0f0fu) * (4u * (16u - n)),
                   pB = B * 4u - ((B >> 4) & 0x0f0f0f0fu) * (4u * (16u - n));
    const uint32_t i01 = __byte_perm(pB, 0u, 0x4140) * (n * n) + __byte_perm(pT, 0u, 0x4140);
    const uint32_t i23 = __byte_perm(pB, 0u, 0x4342) * (n * n) + __byte_perm(pT, 0u, 0x4342);
    const uint32_t i[4] = {i01 & 0xffffu, i01 >> 16, i23 & 0xffffu, i23 >> 16};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      e[j] = *reinterpret_cast<const uint32_t*>(reinterpret_cast<const uint8_t*>(tab) +
                                                (se_check(i[j] < 4u * SE_NIB_ENTRIES, 1u) ? i[j] : 0u));
#else
    const uint32_t k01 = __byte_perm(T, B, 0x5140), k23 = __byte_perm(T, B, 0x7362);
    e[0] = __ldg(gtab + (k01 & 0xffffu));
    e[1] = __ldg(gtab + (k01 >> 16));
    e[2] = __ldg(gtab + (k23 & 0xffffu));
    e[3] = __ldg(gtab + (k23 >> 16));
#endif
  }
}

// A hash lane of a block up to its last step v ^= v >> 16, which leaves the top 16 bits
// alone; xm is the hash base times the lane's multiplier.
__device__ __forceinline__ uint32_t se_nib_mix(uint32_t xm) {
  xm ^= xm >> 16;
  xm *= 0x7feb352du;
  xm ^= xm >> 15;
  return xm * 0x846ca68bu;
}

// Selects the entries' half-words by the mirror selectors (s01, s23: two blocks each) and
// regroups the bytes into row words.
__device__ __forceinline__ void se_nib_rows(const uint32_t e[4], uint32_t s01, uint32_t s23, uint32_t& RT,
                                            uint32_t& RB) {
  const uint32_t P01 = se_prmt(e[0], e[1], s01), P23 = se_prmt(e[2], e[3], s23);
  RT = __byte_perm(P01, P23, 0x6420);
  RB = __byte_perm(P01, P23, 0x7531);
}

// The new rows of a chunk (16 x 2 cells, row words T[0], T[1] and B[0], B[1]) whose first
// block's hash base is x; tab, gtab: the reduced table in shared and in global memory.
template <int NT>
__device__ __forceinline__ void se_nib_eval(const uint32_t T[2], const uint32_t B[2], uint32_t x, uint32_t RT[2],
                                            uint32_t RB[2], const uint32_t* tab, const uint32_t* __restrict__ gtab,
                                            const uint16_t* __restrict__ lut) {
  uint32_t e[8];
  se_nib_lookup<NT>(T[0], B[0], e, tab, gtab, lut);
  se_nib_lookup<NT>(T[1], B[1], e + 4, tab, gtab, lut);
  // The blocks' origins are 2 cells apart, their hash bases 922.  The mirror test
  // h0 >= 2^31 - 64 is bit 31 of the lane before its last step, except when the top 16 bits
  // are 0x7fff.
  uint32_t v[8];
  int top = 0;
#pragma unroll
  for (int j = 0; j < 8; j += 2) {
    v[j] = se_nib_mix(x * 213u + (uint32_t)j * (922u * 213u));
    v[j + 1] = se_nib_mix(x * 213u + (uint32_t)(j + 1) * (922u * 213u));
    top = se_max3(top, (int)v[j], (int)v[j + 1]);
  }
  if (top >= 0x7fff0000) {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = (v[j] ^ (v[j] >> 16)) >= 0x7fffffc0u ? 0x80000000u : 0u;
  }
  uint32_t s[4];  // mirror selectors, two blocks each
#pragma unroll
  for (int j = 0; j < 4; ++j) s[j] = (se_signs(v[2 * j], v[2 * j + 1]) & 0x2222u) ^ 0x5410u;
#if SE_NIB_PROB
  // entries are 0xffffffff or, as ids are at most 14, at most 0xeeeeeeee
  uint32_t high = 0;
#pragma unroll
  for (int j = 0; j < 8; j += 2) high = se_max3u(high, e[j], e[j + 1]);
  uint32_t low = 0;  // bit j: block j takes the full table
  if (__ballot_sync(0xffffffffu, high == 0xffffffffu) != 0u) {
    uint32_t bound[8];
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      const uint32_t k01 = __byte_perm(T[w], B[w], 0x5140), k23 = __byte_perm(T[w], B[w], 0x7362);
      const uint32_t k[4] = {k01 & 0xffffu, k01 >> 16, k23 & 0xffffu, k23 >> 16};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint2 eb =
            NT == 1 ? se_nib_bound(lut, k[j]) : __ldg(reinterpret_cast<const uint2*>(gtab + SE_NIB_BOUNDS) + k[j]);
        e[4 * w + j] = eb.x;
        bound[4 * w + j] = eb.y;
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
#if SE_NIB_LANE
      if (se_nib_mix(x * SE_NIB_MUL + (uint32_t)j * (922u * SE_NIB_MUL)) <= bound[j]) low |= 1u << j;
#else
      if (bound[j]) low |= 1u << j;
#endif
    }
  }
#endif
  se_nib_rows(e, s[0], s[1], RT[0], RB[0]);
  se_nib_rows(e + 4, s[2], s[3], RT[1], RB[1]);
#if SE_NIB_PROB
  while (low) {
    const int j = __ffs(low) - 1, sh = 8 * (j & 3);
    low &= low - 1u;
    const uint32_t t = j & 4 ? T[1] : T[0], u = j & 4 ? B[1] : B[0];
    const uint32_t key = ((t >> sh) & 0xffu) | (((u >> sh) & 0xffu) << 8);
    const uint32_t idx = se_lut_key_index(se_nib_swap_order(key), x + (uint32_t)j * 922u);
    const uint32_t o = se_nib_swap_order(se_lut_fetch(lut, idx));
    const uint32_t mask = ~(0xffu << sh), ot = (o & 0xffu) << sh, ob = (o >> 8) << sh;
    if (j & 4) {
      RT[1] = (RT[1] & mask) | ot;
      RB[1] = (RB[1] & mask) | ob;
    } else {
      RT[0] = (RT[0] & mask) | ot;
      RB[0] = (RB[0] & mask) | ob;
    }
  }
#endif
}

// The bits of a row word whose cells lie outside columns [0, W), first column gx.
__device__ __forceinline__ uint32_t se_nib_outside(int gx, int W) {
  const int lo = se_min(se_max(-gx, 0), 8), hi = se_min(se_max(gx + 8 - W, 0), 8);
  const uint32_t ml = lo >= 8 ? 0xffffffffu : (1u << (4 * lo)) - 1u;
  const uint32_t mh = hi >= 8 ? 0xffffffffu : ~(0xffffffffu >> (4 * hi));
  return ml | mh;
}

// One chunk per lane: its upper row starts at word off (row stride `stride` words, a multiple
// of 2, off too), its first block's cell is world cell (gx, gy).  OX: the column parity of the
// blocks.  All lanes of a warp call it; those without `on` have some chunk to read and write
// nothing.  With `look`, the warp leaves its chunks alone when each is one static material,
// and returns true.
// With OX = 1 a chunk is read from three words a row; the first nibble of the first word
// belongs to the chunk on its left, and of the third only the first nibble to this one, so the
// changes to these two are added atomically (nibbles keep within [0, 15] whatever the order,
// so the differences of whole words add up).  With `edge`, cells outside the world stay WALL.
template <int NT, int OX>
__device__ __forceinline__ bool se_nib_chunk(uint32_t* sm, int off, int stride, bool on, bool look, int gx, int gy,
                                             uint32_t x, int W, int H, bool edge, uint32_t umask, const uint32_t* tab,
                                             const uint32_t* __restrict__ gtab, const uint16_t* __restrict__ lut) {
  uint32_t T[2], B[2], RT[2], RB[2];
  {
    const uint2 t = *reinterpret_cast<const uint2*>(sm + off);
    const uint2 b = *reinterpret_cast<const uint2*>(sm + off + stride);
    T[0] = t.x, T[1] = t.y, B[0] = b.x, B[1] = b.y;
  }
  if (OX) {
    const uint32_t t2 = sm[off + 2], b2 = sm[off + stride + 2];
    T[0] = __funnelshift_r(T[0], T[1], 4);
    T[1] = __funnelshift_r(T[1], t2, 4);
    B[0] = __funnelshift_r(B[0], B[1], 4);
    B[1] = __funnelshift_r(B[1], b2, 4);
  }
  if (look) {
    // the four words are equal and equal themselves turned by one cell
    const uint32_t diff = ((T[0] ^ B[0]) | (T[0] ^ __funnelshift_r(T[0], T[0], 4))) | ((T[1] ^ B[1]) | (T[1] ^ T[0]));
    if (__ballot_sync(0xffffffffu, diff != 0u || (__funnelshift_r(umask, 0u, T[0]) & 1u) == 0u) == 0u) return true;
  }
  se_nib_eval<NT>(T, B, x, RT, RB, tab, gtab, lut);
  if (edge) {
    const uint32_t above = gy >= 0 && gy < H ? 0u : 0xffffffffu, below = gy + 1 >= 0 && gy + 1 < H ? 0u : 0xffffffffu;
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      const uint32_t out = se_nib_outside(gx + 8 * w, W);
      RT[w] = (RT[w] & ~(out | above)) | (0x22222222u & (out | above));
      RB[w] = (RB[w] & ~(out | below)) | (0x22222222u & (out | below));
    }
  }
  if (!on) return false;
  if (OX == 0) {
    *reinterpret_cast<uint2*>(sm + off) = make_uint2(RT[0], RT[1]);
    *reinterpret_cast<uint2*>(sm + off + stride) = make_uint2(RB[0], RB[1]);
  } else {
    int* p = reinterpret_cast<int*>(sm + off);
    sm[off + 1] = __funnelshift_r(RT[0], RT[1], 28);
    sm[off + stride + 1] = __funnelshift_r(RB[0], RB[1], 28);
    atomicAdd(p, (int)((RT[0] - T[0]) << 4));
    atomicAdd(p + stride, (int)((RB[0] - B[0]) << 4));
    const int nt = (int)(RT[1] >> 28) - (int)(T[1] >> 28), nb = (int)(RB[1] >> 28) - (int)(B[1] >> 28);
    if (nt) atomicAdd(p + 2, nt);
    if (nb) atomicAdd(p + stride + 2, nb);
  }
  return false;
}

// One frame of a tile: the blocks of block rows ly0 + 2 j.  A warp stops looking for items at
// rest (`look`) once fewer than one in eight are.
template <class G, int NT, int OX>
__device__ __forceinline__ void se_nib_step(uint32_t* sm, bool& look, int ly0, int gx0, int gy0, int f, int W, int H,
                                            bool edge, uint32_t umask, const uint32_t* tab,
                                            const uint32_t* __restrict__ gtab, const uint16_t* __restrict__ lut) {
  constexpr int WS = NT == 1 ? 1 : 32, LX = NT == 1 ? 1 : G::LX, LY = WS / LX, NW = NT / WS;
  constexpr int NSUB = G::CPR / LX, ITEMS = NSUB * (G::NG * G::LY / LY);
  const int lane = threadIdx.x & (WS - 1), warp = threadIdx.x / WS;
  const int c0 = 16 * (lane % LX) + OX, r0 = ly0 + 2 * (lane / LX);  // the first item's cell
  const int off0 = r0 * G::STRIDE + c0 / 16 * 2;
  const uint32_t x0 = (uint32_t)(gx0 + c0) * 461u + (uint32_t)(gy0 + r0) * 2131u + (uint32_t)f * 4541161u;
  int still = 0, seen = 0;
  for (int it = warp; it < ITEMS; it += NW) {
    const int g = it / NSUB, q = it - g * NSUB;
    const int off = off0 + g * (2 * LY * G::STRIDE) + q * (2 * LX);
    // a lane whose check fails takes no chunk of its own, but the votes of its warp
    const bool ok = se_check(off >= 0 && off + G::STRIDE + 2 < G::STRIDE * G::ROWS, 8u);
    if (look) ++seen;
    if (se_nib_chunk<NT, OX>(sm, ok ? off : 0, G::STRIDE, ok, look, gx0 + c0 + 16 * LX * q, gy0 + r0 + 2 * LY * g,
                             x0 + (uint32_t)(g * LY) * 4262u + (uint32_t)(q * LX) * 7376u, W, H, edge, umask, tab,
                             gtab, lut))
      ++still;
  }
  look = 8 * still > seen;
}

// se_tile_edits (margolus.cuh) on the word-packed array, for the few mods of most lists.  A cell is written only by the last
// mod that hits it, so its nibble changes once; the other cells of its word may change at the
// same time, so the difference is added atomically.
template <class G, int NT>
__device__ __forceinline__ void se_nib_few_edits(uint32_t* sm, int gx0, int gy0, int W, int H, int ya, int yb,
                                                 const SeEditParams* __restrict__ p, int n) {
  const int rx0 = gx0 > 0 ? gx0 : 0, rx1 = (gx0 + G::SW < W ? gx0 + G::SW : W) - 1;
  const int ylo = ya > 0 ? ya : 0, yhi = yb < H ? yb : H;
  const int ry0 = gy0 > ylo ? gy0 : ylo, ry1 = (gy0 + G::SH < yhi ? gy0 + G::SH : yhi) - 1;
  for (int q = 0; q < n; ++q) {
    const int4 b = p->boxes[q];
    if (p->mods[q].mat == (int)SE_NULL) continue;  // its cells keep the simulated value
    const int x0 = b.x > rx0 ? b.x : rx0, x1 = b.z < rx1 ? b.z : rx1;
    const int y0 = b.y > ry0 ? b.y : ry0, y1 = b.w < ry1 ? b.w : ry1;
    if (x0 > x1 || y0 > y1) continue;
    const SeMod m = p->mods[q];
    const int w = x1 - x0 + 1, cnt = w * (y1 - y0 + 1);
    for (int t = threadIdx.x; t < cnt; t += NT) {
      const int y = y0 + t / w, x = x0 + t % w;
      if (!se_mod_hits(m, x, y)) continue;
      bool later = false;
      for (int r = q + 1; r < n && !later; ++r) {
        const int4 rb = p->boxes[r];
        later = x >= rb.x && x <= rb.z && y >= rb.y && y <= rb.w && se_mod_hits(p->mods[r], x, y);
      }
      const int i = (y - gy0) * G::STRIDE + (x - gx0) / 8, sh = 4 * ((x - gx0) & 7);
      if (later || !se_check(i >= 0 && i < G::STRIDE * G::ROWS, 32u)) continue;
      const int d = m.mat - (int)((sm[i] >> sh) & 15u);
      if (d) atomicAdd(reinterpret_cast<int*>(sm) + i, (int)((uint32_t)d << sh));
    }
  }
}

// Longer lists.  Eight words of bits (`hit`, zero before) say which mods' boxes meet the cells
// that can change: those of the world and of the buffer rows [ya, yb).  After them lie these boxes,
// clipped to those cells, as array coordinates (x0 | y0 << 16, x1 | y1 << 16).
template <class G, int NT>
__device__ __forceinline__ void se_nib_find_edits(uint32_t* hit, int gx0, int gy0, int W, int H, int ya, int yb,
                                                  const SeEditParams* __restrict__ p, int n) {
  const int rx0 = se_max(gx0, 0), rx1 = se_min(gx0 + G::SW, W) - 1;
  const int ry0 = se_max(gy0, se_max(ya, 0)), ry1 = se_min(gy0 + G::SH, se_min(yb, H)) - 1;
  for (int q = threadIdx.x; q < n; q += NT) {
    const int4 b = p->boxes[q];
    const int x0 = se_max(b.x, rx0), y0 = se_max(b.y, ry0), x1 = se_min(b.z, rx1), y1 = se_min(b.w, ry1);
    if (x0 > x1 || y0 > y1) continue;
    atomicOr(hit + (q >> 5), 1u << (q & 31));
    hit[8 + 2 * q] = (uint32_t)(x0 - gx0) | (uint32_t)(y0 - gy0) << 16;
    hit[9 + 2 * q] = (uint32_t)(x1 - gx0) | (uint32_t)(y1 - gy0) << 16;
  }
}

// A cell takes the material of the last mod that hits it unless that is NULL.  A warp takes 32 x 4 cells,
// a column of four to a lane, finds the mods whose boxes meet them by a vote and goes through these
// from the last to the first, until each cell has met its last one.  Mod by mod, with a look at all
// later mods for every cell, the time is that of the fullest tile, and a stroke puts many mods into one
// (us of a frame on 256 x 256, four materials, waited for, mod by mod / so: 8 circles at random 22.7 / 21.3,
// 32 58 / 31, 256 690 / 90, 64 circles over each other 636 / 119; columns of eight cells 203).
template <class G, int NT>
__device__ __forceinline__ void se_nib_edits(uint32_t* sm, const uint32_t* hit, int gx0, int gy0,
                                             const SeEditParams* __restrict__ p, int n) {
  constexpr int WS = NT == 1 ? 1 : 32, R = 4, PX = (G::SW + WS - 1) / WS, PY = (G::SH + R - 1) / R;
  const int lane = threadIdx.x & (WS - 1);
  uint32_t any = 0;
  for (int k = 0; k < (n + 31) >> 5; ++k) any |= hit[k];
  if (!any) return;
  for (int i = threadIdx.x / WS; i < PX * PY; i += NT / WS) {
    const int py = i / PX * R, px = (i - i / PX * PX) * WS, cx = px + lane;
    uint32_t open = (1u << R) - 1u;  // the lane's cells that no mod has hit yet
    for (int q0 = (n - 1) / WS * WS; q0 >= 0; q0 -= WS) {
      if (!(hit[q0 >> 5] >> (WS == 1 ? q0 & 31 : 0))) continue;
      const int l = q0 + WS - 1 - lane;  // the last mod in the vote's lowest bit
      bool meets = (hit[l >> 5] >> (l & 31)) & 1u;  // false beyond n
      if (meets) {
        const uint32_t lo = hit[8 + 2 * l], hi = hit[9 + 2 * l];
        meets = (int)(lo & 0xffffu) < px + WS && (int)(hi & 0xffffu) >= px && (int)(lo >> 16) < py + R &&
                (int)(hi >> 16) >= py;
      }
      for (uint32_t m = __ballot_sync(0xffffffffu, meets); m;) {
        const int q = q0 + WS - __ffs((int)m);
        m &= m - 1u;
        const uint32_t lo = hit[8 + 2 * q], hi = hit[9 + 2 * q];
        if (!open || cx < (int)(lo & 0xffffu) || cx > (int)(hi & 0xffffu)) continue;
        const SeMod mod = p->mods[q];
        uint32_t hits = 0;  // all rows at once: the roots in flight together
#pragma unroll
        for (int r = 0; r < R; ++r) hits |= se_mod_hits(mod, gx0 + cx, gy0 + py + r) ? 1u << r : 0u;
        hits &= open & (0xffu << se_max((int)(lo >> 16) - py, 0)) & (0xffu >> se_max(py + 7 - (int)(hi >> 16), 0));
        open &= ~hits;
        if (mod.mat == (int)SE_NULL) continue;  // its cells keep the simulated value
        for (; hits; hits &= hits - 1u) {
          const int w = (py + __ffs((int)hits) - 1) * G::STRIDE + cx / 8, sh = 4 * (cx & 7);
          if (!se_check(w >= 0 && w < G::STRIDE * G::ROWS, 32u)) continue;
          const int d = mod.mat - (int)((sm[w] >> sh) & 15u);
          if (d) atomicAdd(reinterpret_cast<int*>(sm) + w, (int)((uint32_t)d << sh));
        }
      }
    }
  }
}

// Four ids as a half-word of nibbles (unknown ids NULL).
__device__ __forceinline__ uint32_t se_nib_pack(uint4 v) {
  if (max(max(v.x, v.y), max(v.z, v.w)) >= (uint32_t)SE_NMAT)
    v = make_uint4(se_norm(v.x), se_norm(v.y), se_norm(v.z), se_norm(v.w));
  return (v.x + v.y * 16u) + (v.z + v.w * 16u) * 256u;
}

// se_tile_run (margolus.cuh) on the word-packed array: the same contract.  Bound by the ALU pipe
// (four materials: 78% of peak) or by the L1 data pipe that gathers a table too large for shared memory
// (twelve: 71%).  Against byte tiles with two hash lanes a block and lists of chunks, us of an
// 8-frame launch on 8192^2: twelve materials 320-337 -> 271, later frames 317-330 -> 232.  Two words a
// row per lane share the loop, the skip test and the checks over 8 blocks (one word: 333 -> 281).
template <int TW, int TH, int KMAX, int NT>
__device__ __forceinline__ void se_nib_run(const uint32_t* __restrict__ src, uint32_t* __restrict__ dst, int W,
                                           int H, int f0, int k, const uint16_t* __restrict__ lut, int X0, int Y0,
                                           int ya, int yb, const SeEditParams* __restrict__ edits, int nedits) {
  using G = SeNib<TW, TH, KMAX>;
  static_assert(TW % 4 == 0, "tile width must be a multiple of 4");
  static_assert(NT % 32 == 0 || NT == 1, "whole warps");
  extern __shared__ __align__(16) uint8_t se_smem[];
  uint32_t* sm = reinterpret_cast<uint32_t*>(se_smem);
  const uint32_t* gtab = reinterpret_cast<const uint32_t*>(reinterpret_cast<const uint8_t*>(lut) + SE_NIB_OFF);
  uint32_t* tab = sm + G::TABLE;
  const uint32_t umask = NT == 1 ? se_nib_static_mask(lut) : __ldg(gtab + SE_NIB_ENTRIES);
  se_nib_copy_table(tab, gtab, NT);
  const int gx0 = X0 - G::HX, gy0 = Y0 - G::HY;
  const bool many = nedits > SE_NIB_FEW_EDITS;
  if (many)
    for (int i = threadIdx.x; i < 8; i += NT) sm[G::HIT + i] = 0u;
  const bool vec = (W & 3) == 0;
  constexpr int HPR = G::SW / 4;  // half-words (four cells) per row
  uint16_t* sh = reinterpret_cast<uint16_t*>(se_smem);
  constexpr int PAD = G::STRIDE - G::SW / 8;
  for (int i = threadIdx.x; i < G::SH * PAD; i += NT) sm[i / PAD * G::STRIDE + G::SW / 8 + i % PAD] = 0x22222222u;
  for (int i = G::SH * G::STRIDE + threadIdx.x; i < G::ROWS * G::STRIDE; i += NT) sm[i] = 0x22222222u;
  if (vec && gx0 >= 0 && gy0 >= ya && gx0 + G::SW <= W && gy0 + G::SH <= yb) {
    // The region lies inside the world (and the buffer): four 16-byte loads per thread are
    // issued before any is converted, so they are in flight together.
    constexpr int NL = HPR * G::SH;
    const uint32_t* base = src + (size_t)(gy0 - ya) * W + gx0;
    for (int i0 = threadIdx.x; i0 < NL; i0 += 4 * NT) {
      uint4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = i0 + u * NT;
        if (i < NL) {
          const int r = i / HPR, c = i - r * HPR;
          if (!se_check(gy0 - ya + r < yb - ya && gx0 + 4 * c + 3 < W, 16u)) {
            v[u] = make_uint4(SE_WALL, SE_WALL, SE_WALL, SE_WALL);
            continue;
          }
          v[u] = __ldg(reinterpret_cast<const uint4*>(base + (size_t)r * W + 4 * c));
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = i0 + u * NT;
        if (i < NL) {
          const int r = i / HPR, c = i - r * HPR;
          sh[r * (2 * G::STRIDE) + c] = (uint16_t)se_nib_pack(v[u]);
        }
      }
    }
  } else {
    // As above, with a check of each group of four cells.
    constexpr int NL = HPR * G::SH;
    for (int i0 = threadIdx.x; i0 < NL; i0 += 4 * NT) {
      uint4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = i0 + u * NT, r = i / HPR, c = i - r * HPR;
        v[u] = se_load_quad(src, W, i < NL ? gx0 + 4 * c : W, gy0 + r, ya, yb, vec);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = i0 + u * NT, r = i / HPR, c = i - r * HPR;
        if (i < NL) sh[r * (2 * G::STRIDE) + c] = (uint16_t)se_nib_pack(v[u]);
      }
    }
  }
  se_nib_table_ready();
  __syncthreads();
  if (many)  // read after the first frame's barrier
    se_nib_find_edits<G, NT>(sm + G::HIT, gx0, gy0, W, H, ya, yb, edits, nedits);

  const bool edge = gx0 < 0 || gy0 < 0 || gx0 + G::SW > W || gy0 + G::SH > H;
  bool look = true;
  for (int s = 0; s < k; ++s) {
    const int f = f0 + s;
    const int ly0 = (se_off_y(f) + gy0) & 1;
    if (se_off_x(f) == 0)
      se_nib_step<G, NT, 0>(sm, look, ly0, gx0, gy0, f, W, H, edge, umask, tab, gtab, lut);
    else
      se_nib_step<G, NT, 1>(sm, look, ly0, gx0, gy0, f, W, H, edge, umask, tab, gtab, lut);
    __syncthreads();
    if (s == 0 && nedits > 0) {  // the first frame's edits (the host passes them only then)
      if (many)
        se_nib_edits<G, NT>(sm, sm + G::HIT, gx0, gy0, edits, nedits);
      else
        se_nib_few_edits<G, NT>(sm, gx0, gy0, W, H, ya, yb, edits, nedits);
      __syncthreads();
    }
  }

  constexpr int OWPR = TW / 4;
  const bool inside = vec && X0 + TW <= W && Y0 + TH <= yb && Y0 >= ya;
  for (int i = threadIdx.x; i < OWPR * TH; i += NT) {
    const int r = i / OWPR, c = i - r * OWPR;
    const int gy = Y0 + r, gx = X0 + 4 * c;
    if (!inside && (gy >= yb || gx >= W)) continue;
    if (!se_check(gy >= ya, 16u)) continue;
    const uint32_t h = sh[(r + G::HY) * (2 * G::STRIDE) + G::HX / 4 + c];
    uint32_t* out = dst + (size_t)(gy - ya) * W + gx;
    if (inside || (vec && gx + 3 < W)) {
      *reinterpret_cast<uint4*>(out) = make_uint4(h & 15u, (h >> 4) & 15u, (h >> 8) & 15u, h >> 12);
    } else {
      for (int e = 0; e < 4; ++e)
        if (gx + e < W) out[e] = (h >> (4 * e)) & 15u;
    }
  }
}

// One frame of a whole world (se_nib_resident's array): chunk i of cpr * nby, a lane each.
template <int OX>
__device__ __forceinline__ void se_nib_world_step(uint32_t* sm, int stride, int rows, int cpr, float inv_cpr, bool& look,
                                                  int ly0, int gx0, int gy0, int f, int W, int H, uint32_t umask,
                                                  const uint32_t* tab, const uint32_t* __restrict__ gtab,
                                                  const uint16_t* __restrict__ lut) {
#if defined(__CUDA_ARCH__) || defined(SE_WHOLE_WARPS)
  constexpr int NT = 32;
#else
  constexpr int NT = 1;  // emulated: one thread per CTA
#endif
  const int lane = threadIdx.x & (NT - 1), nc = cpr * ((rows - ly0) / 2);
  int still = 0, seen = 0;
  for (int base = threadIdx.x & ~(NT - 1); base < nc; base += blockDim.x) {  // warp-uniform trip count
    const bool on = base + lane < nc;
    int j, q;
    se_divmod_rt(on ? base + lane : base, cpr, inv_cpr, j, q);
    const int row = ly0 + 2 * j, off = row * stride + 2 * q, gx = gx0 + 16 * q + OX, gy = gy0 + row;
    const bool ok = se_check(off >= 0 && off + stride + 2 < stride * rows, 8u);  // as in se_nib_step
    if (look) ++seen;
    const uint32_t x = (uint32_t)gx * 461u + (uint32_t)gy * 2131u + (uint32_t)f * 4541161u;
    if (se_nib_chunk<NT, OX>(sm, ok ? off : 0, stride, on && ok, look, gx, gy, x, W, H, true, umask, tab, gtab, lut)) ++still;
  }
  look = 8 * still > seen;
}

// se_resident's body on a word-packed array: the whole world with a WALL border of 4 columns on
// the left, at least one on the right, and one row above and below; two words of padding per
// row (the stride is 0 mod 4 words where cpr is odd: some of its 8-byte accesses meet in a bank, unlike a
// tile's).  A world takes half a byte a cell, so worlds of up to about 450,000 cells fit a CTA.  Bound as
// the tiles are (4096 worlds, 100 frames, on byte arrays / so: 28.5 / 23.5 ms).
__device__ __forceinline__ void se_nib_resident(const SeWorldDesc& w, int frames, int out_flip,
                                                const uint16_t* __restrict__ lut) {
  extern __shared__ __align__(16) uint8_t se_smem[];
  const int W = w.W, H = w.H, cpr = (W + 5 + 15) / 16, stride = 2 * cpr + 2, rows = H + 2, nt = blockDim.x;
  uint32_t* sm = reinterpret_cast<uint32_t*>(se_smem);
  const uint32_t* gtab = reinterpret_cast<const uint32_t*>(reinterpret_cast<const uint8_t*>(lut) + SE_NIB_OFF);
  uint32_t* tab = sm + ((stride * rows + 3) & ~3);
#if defined(__CUDA_ARCH__) || defined(SE_WHOLE_WARPS)
  const uint32_t umask = __ldg(gtab + SE_NIB_ENTRIES);
  se_nib_copy_table(tab, gtab, nt);
#else
  const uint32_t umask = se_nib_static_mask(lut);
#endif
  for (int i = threadIdx.x; i < stride * rows; i += nt) sm[i] = 0x22222222u;
  se_nib_table_ready();
  __syncthreads();
  const uint32_t* src = w.cur ? w.buf1 : w.buf0;
  uint32_t* dst = (w.cur ^ out_flip) ? w.buf1 : w.buf0;
  uint16_t* sh = reinterpret_cast<uint16_t*>(se_smem);
  const int hpr = (W + 3) / 4;  // half-words (four cells) of world cells per row
  const float inv_hpr = 1.0f / (float)hpr, inv_cpr = 1.0f / (float)cpr;
  const bool vec = (W & 3) == 0;
  for (int i = threadIdx.x; i < hpr * H; i += nt) {
    int y, c;
    se_divmod_rt(i, hpr, inv_hpr, y, c);
    const uint32_t* p = src + (size_t)y * W + 4 * c;
    uint4 v;
    if (vec) {
      v = __ldg(reinterpret_cast<const uint4*>(p));
    } else {
      v.x = __ldg(p);
      v.y = 4 * c + 1 < W ? __ldg(p + 1) : SE_WALL;
      v.z = 4 * c + 2 < W ? __ldg(p + 2) : SE_WALL;
      v.w = 4 * c + 3 < W ? __ldg(p + 3) : SE_WALL;
    }
    const int k = (y + 1) * 2 * stride + 1 + c;
    if (se_check(k < 2 * stride * rows, 2u)) sh[k] = (uint16_t)se_nib_pack(v);
  }
  __syncthreads();
  bool look = true;
  for (int s = 0; s < frames; ++s) {
    const int f = w.frame + 1 + s, ly0 = (se_off_y(f) - 1) & 1;
    if (se_off_x(f) == 0)
      se_nib_world_step<0>(sm, stride, rows, cpr, inv_cpr, look, ly0, -4, -1, f, W, H, umask, tab, gtab, lut);
    else
      se_nib_world_step<1>(sm, stride, rows, cpr, inv_cpr, look, ly0, -4, -1, f, W, H, umask, tab, gtab, lut);
    if ((s & 63) == 63) look = true;  // the world may have come to rest
    __syncthreads();
  }
  for (int i = threadIdx.x; i < hpr * H; i += nt) {
    int y, c;
    se_divmod_rt(i, hpr, inv_hpr, y, c);
    const uint32_t h = sh[(y + 1) * 2 * stride + 1 + c];
    uint32_t* p = dst + (size_t)y * W + 4 * c;
    if (vec) {
      *reinterpret_cast<uint4*>(p) = make_uint4(h & 15u, (h >> 4) & 15u, (h >> 8) & 15u, h >> 12);
    } else {
      for (int e = 0; e < 4; ++e)
        if (4 * c + e < W) p[e] = (h >> (4 * e)) & 15u;
    }
  }
}
#endif  // SE_NIB
