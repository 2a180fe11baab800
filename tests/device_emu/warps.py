"""CPU emulation of the JIT device code with whole warps.  TEST INFRASTRUCTURE ONLY.

emu.py runs a CTA as one thread, whose warps have one lane.  Here each thread of a CTA is a
fiber: it runs until its next vote, shuffle or barrier, and goes on once the others it waits for
are there too.  So the kernels run with their real thread counts, lane layouts and reduced tables
(SE_WHOLE_WARPS), and a lane that leaves its warp before a vote is seen: the CTA cannot go on,
and the launch raises instead of hanging.  Lanes run one after the other between those points.
"""
import ctypes
import hashlib
import os
import subprocess

import numpy as np

from tests.device_emu.emu import HERE, OUT

# (tile width, tile height, frames, threads) of the 4-bit tile shapes, and three byte shapes
SHAPES = [(56, 30, 1, 128), (120, 120, 4, 128), (112, 112, 8, 256), (48, 48, 8, 128), (240, 176, 8, 256),
          (240, 240, 8, 256), (96, 96, 16, 256), (32, 32, 16, 128), (128, 128, 16, 256)]
BYTE_SHAPES = [(128, 64, 1, 256), (128, 64, 8, 256), (64, 64, 4, 256)]

PRELUDE = r'''
#include <ucontext.h>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <vector>
#define SE_WHOLE_WARPS 1
// emu.py's one-thread definitions give way to those below
#define __syncthreads shim_syncthreads
#define __ballot_sync shim_ballot_sync
#define __shfl_sync shim_shfl_sync
#define __shfl_up_sync shim_shfl_up_sync
#include "cuda_host_shim.hpp"
#undef __syncthreads
#undef __ballot_sync
#undef __shfl_sync
#undef __shfl_up_sync
namespace fibers {
enum Wait { kRun, kVote, kShuffle, kBarrier, kDone };
struct Fiber {
  ucontext_t ctx;
  Wait wait;
  unsigned long long value, result;
  int from;
};
constexpr size_t kStack = 128 << 10;
static ucontext_t g_main;
static std::vector<Fiber> g_fibers;
static std::vector<char> g_stacks;
static int g_cur = 0;
static const std::function<void()>* g_body = nullptr;
static void entry() {
  (*g_body)();
  g_fibers[g_cur].wait = kDone;
  swapcontext(&g_fibers[g_cur].ctx, &g_main);
}
inline unsigned long long wait(Wait w, unsigned long long value, int from) {
  Fiber& f = g_fibers[g_cur];
  f.wait = w, f.value = value, f.from = from;
  swapcontext(&f.ctx, &g_main);
  return f.result;
}
// Runs a CTA of nt threads; false when some of them wait for others that will not come.
static bool cta(int nt, const std::function<void()>& body) {
  g_body = &body;
  g_fibers.assign(nt, Fiber{});
  if (g_stacks.size() < nt * kStack) g_stacks.resize(nt * kStack);
  blockDim.x = nt;
  for (int i = 0; i < nt; ++i) {
    Fiber& f = g_fibers[i];
    getcontext(&f.ctx);
    f.ctx.uc_stack.ss_sp = g_stacks.data() + i * kStack;
    f.ctx.uc_stack.ss_size = kStack;
    f.ctx.uc_link = &g_main;
    makecontext(&f.ctx, entry, 0);
    f.wait = kRun;
  }
  for (;;) {
    bool ran = false;
    for (int i = 0; i < nt; ++i) {
      if (g_fibers[i].wait != kRun) continue;
      ran = true;
      g_cur = i;
      threadIdx.x = i;
      swapcontext(&g_main, &g_fibers[i].ctx);
    }
    int done = 0, barrier = 0;
    for (const Fiber& f : g_fibers) done += f.wait == kDone, barrier += f.wait == kBarrier;
    if (done == nt) return true;
    if (!ran) return false;
    if (done + barrier == nt) {
      for (Fiber& f : g_fibers)
        if (f.wait == kBarrier) f.wait = kRun;
      continue;
    }
    for (int w = 0; w < nt; w += 32) {  // whole warps only: every mask in the kernels is full
      const int lanes = nt - w < 32 ? nt - w : 32;
      const Wait kind = g_fibers[w].wait;
      bool all = kind == kVote || kind == kShuffle;
      unsigned long long votes = 0;
      for (int l = 0; l < lanes; ++l) {
        all = all && g_fibers[w + l].wait == kind;
        votes |= (g_fibers[w + l].value ? 1ull : 0ull) << l;
      }
      if (!all) continue;
      for (int l = 0; l < lanes; ++l) {
        Fiber& f = g_fibers[w + l];
        f.result = kind == kVote ? votes : g_fibers[w + f.from].value;
        f.wait = kRun;
      }
    }
  }
}
}  // namespace fibers
inline void __syncthreads() { fibers::wait(fibers::kBarrier, 0, 0); }
inline unsigned __ballot_sync(unsigned, bool p) { return (unsigned)fibers::wait(fibers::kVote, p, 0); }
template <class T>
inline T __shfl_sync(unsigned, T v, int lane) {
  return (T)fibers::wait(fibers::kShuffle, (unsigned long long)v, lane);
}
template <class T>
inline T __shfl_up_sync(unsigned, T v, unsigned d) {
  const int lane = threadIdx.x & 31;
  return (T)fibers::wait(fibers::kShuffle, (unsigned long long)v, lane < (int)d ? lane : lane - (int)d);
}
'''

DRIVER = r'''
alignas(16) uint8_t se_smem[1 << 20];
static uint16_t* g_lut = nullptr;
extern "C" unsigned emu_check_word() {
  const unsigned w = se_check_word;
  se_check_word = 0;
  return w;
}
static void one_thread(unsigned block, unsigned thread, unsigned threads) {
  blockIdx.x = block, threadIdx.x = thread, blockDim.x = threads;
}
extern "C" int emu_build_lut() {
#ifdef SE_LUT
  size_t bytes = SE_LUT_STATIC_OFF + 4u * SE_LUT_STATIC_WORDS;
#ifdef SE_NIB
  bytes = SE_NIB_OFF + 4u * (SE_NIB_BOUNDS + 2u * 65536u);
#endif
  g_lut = reinterpret_cast<uint16_t*>(aligned_alloc(256, (bytes + 255) & ~(size_t)255));
  memset(g_lut, 0xee, bytes);
  gridDim.x = gridDim.y = 1, blockIdx.x = blockIdx.y = 0;
  fibers::cta(1, [] { se_build_lut(g_lut); });  // the other builders have no barrier
  for (unsigned w = 0; w < SE_LUT_STATIC_WORDS; ++w) one_thread(w, 0, 1), se_build_static(g_lut);
#ifdef SE_NIB
  for (unsigned i = 0; i < 65536; ++i) one_thread(i / 256, i % 256, 256), se_build_nib(g_lut);
#endif
  one_thread(0, 0, 1);
  return 1;
#else
  return 0;
#endif
}
extern "C" int emu_nib_lane() {
#ifdef SE_NIB
  return SE_NIB_PROB ? SE_NIB_LANE : -1;
#else
  return -2;
#endif
}
static bool g_ok = true;
static void launch(unsigned gx, unsigned gy, int nt, const std::function<void()>& body) {
  gridDim.x = gx, gridDim.y = gy;
  for (unsigned y = 0; y < gy && g_ok; ++y)
    for (unsigned x = 0; x < gx && g_ok; ++x) {
      blockIdx.x = x, blockIdx.y = y;
      memset(se_smem, 0xee, sizeof se_smem);  // shared memory starts undefined
      g_ok = fibers::cta(nt, body);
    }
}
// 1 when a launch since the last call could not go on
extern "C" int emu_stuck() {
  const bool ok = g_ok;
  g_ok = true;
  return !ok;
}
#define EMU_SHAPE(TW, TH, K, NT) \
extern "C" void emu_tile_##TW##x##TH##_k##K(const uint32_t* src, uint32_t* dst, int W, int H, int f0, int k, \
                                           int ya, int yb, const void* edits, int nedits) { \
  launch((W + TW - 1) / TW, (yb - ya + TH - 1) / TH, NT, [=] { \
    se_tile_impl<TW, TH, K, NT>(src, dst, W, H, f0, k, g_lut, ya, yb, \
                                reinterpret_cast<const SeEditParams*>(edits), nedits); \
  }); \
} \
extern "C" void emu_mtile_##TW##x##TH##_k##K(const SeWorldDesc* worlds, const SeTileJob* jobs, int njobs, int pass, \
                                            int done, int k) { \
  launch(njobs, 1, NT, [=] { se_mtile_impl<TW, TH, K, NT>(worlds, jobs, pass, done, k, g_lut); }); \
} \
extern "C" void emu_stile_##TW##x##TH##_k##K(const SeWorldDesc* descs, const int* prefix, int n) { \
  launch(prefix[n], 1, NT, [=] { se_stile_impl<TW, TH, K, NT>(descs, prefix, n, g_lut); }); \
}
@SHAPES@
extern "C" void emu_resident(const SeWorldDesc* worlds, const int* ids, int nids, int frames, int flip, int nt) {
  launch(nids, 1, nt, [=] { se_resident(worlds, ids, frames, flip, g_lut); });
}
#ifdef SE_NIB
// One frame on the array `words` of a 48 x 48 tile of 8 frames.  CUT: the rows that count as the
// array's, so that the chunks below them fail their check.
template <int CUT>
struct CutTile : SeNib<48, 48, 8> {
  static constexpr int ROWS = SeNib<48, 48, 8>::ROWS - CUT;
};
template <int CUT>
static void cut_step(uint32_t* words, int f) {
  using G = CutTile<CUT>;
  launch(1, 1, 128, [=] {
    uint32_t* sm = reinterpret_cast<uint32_t*>(se_smem);
    constexpr int N = G::STRIDE * SeNib<48, 48, 8>::ROWS;
    const uint32_t* gtab =
        reinterpret_cast<const uint32_t*>(reinterpret_cast<const uint8_t*>(g_lut) + SE_NIB_OFF);
    uint32_t* tab = sm + ((N + 3) & ~3);
    se_nib_copy_table(tab, gtab, 128);
    for (int i = threadIdx.x; i < N; i += 128) sm[i] = words[i];
    __syncthreads();
    bool look = true;
    const int ly0 = (se_off_y(f) + 100) & 1;
    if (se_off_x(f) == 0)
      se_nib_step<G, 128, 0>(sm, look, ly0, 100, 100, f, 1000, 1000, false, gtab[SE_NIB_ENTRIES], tab, gtab, g_lut);
    else
      se_nib_step<G, 128, 1>(sm, look, ly0, 100, 100, f, 1000, 1000, false, gtab[SE_NIB_ENTRIES], tab, gtab, g_lut);
    __syncthreads();
    for (int i = threadIdx.x; i < N; i += 128) words[i] = sm[i];
  });
}
extern "C" void emu_cut_step(uint32_t* words, int f, int cut) { cut ? cut_step<6>(words, f) : cut_step<0>(words, f); }
extern "C" int emu_cut_stride() { return SeNib<48, 48, 8>::STRIDE; }
extern "C" int emu_cut_rows() { return SeNib<48, 48, 8>::ROWS; }
// One frame of a whole world's array (`rows` rows of 2 cpr + 2 words) from block row ly0 on: chunks
// above row 0 fail their check.
extern "C" void emu_world_step(uint32_t* words, int rows, int cpr, int ly0, int f) {
  launch(1, 1, 64, [=] {
    uint32_t* sm = reinterpret_cast<uint32_t*>(se_smem);
    const int stride = 2 * cpr + 2, n = stride * rows;
    const uint32_t* gtab =
        reinterpret_cast<const uint32_t*>(reinterpret_cast<const uint8_t*>(g_lut) + SE_NIB_OFF);
    uint32_t* tab = sm + ((n + 3) & ~3);
    se_nib_copy_table(tab, gtab, 64);
    for (int i = threadIdx.x; i < n; i += 64) sm[i] = words[i];
    __syncthreads();
    bool look = true;
    if (se_off_x(f) == 0)
      se_nib_world_step<0>(sm, stride, rows, cpr, 1.0f / cpr, look, ly0, 100, 100, f, 1000, 1000, gtab[SE_NIB_ENTRIES],
                           tab, gtab, g_lut);
    else
      se_nib_world_step<1>(sm, stride, rows, cpr, 1.0f / cpr, look, ly0, 100, 100, f, 1000, 1000, gtab[SE_NIB_ENTRIES],
                           tab, gtab, g_lut);
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += 64) words[i] = sm[i];
  });
}
#endif
'''

WORLD = [("b0", "<u8"), ("b1", "<u8"), ("W", "<i4"), ("H", "<i4"), ("frame", "<i4"), ("cur", "<i4"), ("k", "<i4"),
         ("p1", "<i4")]


class WarpEmu:
    def __init__(self, ruleset, shapes=None):
        src = "#define SE_CHECKED 1\n" + ruleset.kernel_source
        shapes = shapes or SHAPES + BYTE_SHAPES
        defs = "\n".join(f"EMU_SHAPE({a}, {b}, {c}, {d})" for a, b, c, d in shapes)
        code = PRELUDE + src + DRIVER.replace("@SHAPES@", defs)
        with open(os.path.join(HERE, "cuda_host_shim.hpp")) as f:
            key = hashlib.sha256((code + f.read()).encode()).hexdigest()[:16]
        d = os.path.join(OUT, "warps_" + key)
        so = os.path.join(d, "warps.so")
        if not os.path.exists(so):
            os.makedirs(d, exist_ok=True)
            cpp = os.path.join(d, "warps.cpp")
            with open(cpp, "w") as f:
                f.write(code)
            tmp = so + f".tmp{os.getpid()}"
            r = subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-ffp-contract=off",
                                "-fno-strict-aliasing", "-w", f"-I{HERE}", cpp, "-o", tmp], capture_output=True, text=True)
            if r.returncode:
                raise RuntimeError(r.stderr[-4000:])
            os.replace(tmp, so)
        self.lib = ctypes.CDLL(so)
        self.lib.emu_check_word.restype = ctypes.c_uint
        self.has_lut = bool(self.lib.emu_build_lut())
        self.nib_lane = self.lib.emu_nib_lane()  # the extra hash lane; 0 several, -1 none, -2 byte tiles
        self.checked()

    def checked(self, word=0):
        stuck, w = self.lib.emu_stuck(), self.lib.emu_check_word()
        assert not stuck, "some threads of a CTA wait for others that will not come"
        assert w == word, f"check word {w:#x}"

    def tiles(self, src, f0, k, shape, band=None, edits=None, nedits=0):
        """k frames (counters f0 ..) with one launch; ``band = (world height, first row)``."""
        fn = getattr(self.lib, "emu_tile_%dx%d_k%d" % shape[:3])
        vp, ci = ctypes.c_void_p, ctypes.c_int
        fn.argtypes = [vp, vp] + [ci] * 6 + [vp, ci]
        rows, W = src.shape
        H, ya = band if band else (rows, 0)
        dst = np.full_like(src, 0xEE)
        fn(src.ctypes.data, dst.ctypes.data, W, H, f0, k, ya, ya + rows,
           edits.ctypes.data if edits is not None else None, nedits)
        self.checked()
        return dst

    def _worlds(self, grids, frames, ks):
        desc, bufs = np.zeros(len(grids), dtype=WORLD), []
        for i, g in enumerate(grids):
            a, b = np.ascontiguousarray(g, dtype=np.uint32).copy(), np.full(g.shape, 0xEE, dtype=np.uint32)
            bufs.append((a, b))
            desc[i] = (a.ctypes.data, b.ctypes.data, g.shape[1], g.shape[0], frames[i], 0, ks[i], 0)
        return desc, bufs

    def tile_jobs(self, grids, frames, k, shape):
        """One pass of a batch's tiled worlds."""
        desc, bufs = self._worlds(grids, frames, [0] * len(grids))
        jobs = np.array([(w, x, y, 0) for w, g in enumerate(grids) for y in range(0, g.shape[0], shape[1])
                         for x in range(0, g.shape[1], shape[0])], dtype=np.int32)
        getattr(self.lib, "emu_mtile_%dx%d_k%d" % shape[:3])(
            ctypes.c_void_p(desc.ctypes.data), ctypes.c_void_p(jobs.ctypes.data), len(jobs), 0, 0, k)
        self.checked()
        return [b for _, b in bufs]

    def serve(self, grids, frames, ks, shape):
        """One serving iteration: world a advances ks[a] frames."""
        desc, bufs = self._worlds(grids, frames, ks)
        pre = np.cumsum([0] + [-(-g.shape[1] // shape[0]) * -(-g.shape[0] // shape[1]) for g in grids]).astype(np.int32)
        getattr(self.lib, "emu_stile_%dx%d_k%d" % shape[:3])(
            ctypes.c_void_p(desc.ctypes.data), ctypes.c_void_p(pre.ctypes.data), len(grids))
        self.checked()
        return [b for _, b in bufs]

    def resident(self, grids, frames, F, threads):
        """Whole worlds in shared memory for F frames, from buffer 0 to buffer 1."""
        desc, bufs = self._worlds(grids, frames, [0] * len(grids))
        ids = np.arange(len(grids), dtype=np.int32)
        self.lib.emu_resident(ctypes.c_void_p(desc.ctypes.data), ctypes.c_void_p(ids.ctypes.data), len(ids), F, 1,
                              threads)
        self.checked()
        return [b for _, b in bufs]
