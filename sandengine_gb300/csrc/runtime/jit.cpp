#include "jit.hpp"

#include <nvrtc.h>
#include <sys/stat.h>
#include <unistd.h>

#include <cstdio>
#include <cstdlib>
#include <fstream>
#include <functional>
#include <mutex>
#include <sstream>

#include "../../../include/sandengine.h"
#include "kernel_src.inc"  // SE_PRELUDE_SRC, SE_MARGOLUS_SRC, SE_NIBBLE_SRC (generated from csrc/kernels)

namespace se::rt {

std::string TileVariant::name() const {
  return "se_tile_" + std::to_string(tw) + "x" + std::to_string(th) + "_k" + std::to_string(kmax);
}

std::string TileVariant::edit_name() const {
  return "se_tile_edit_" + std::to_string(tw) + "x" + std::to_string(th) + "_k" + std::to_string(kmax);
}

// Tile shapes and fusion depths compiled into every rule-set module; the launcher and the
// autotuner choose among those marked for the rule set's kind of tile.  Larger tiles
// recompute a smaller share of halo cells per fused step (128x64 at k=8: 1.41x the tile's
// cells; 256x128 at k=8: 1.20x; 240x240: 1.14x).  Byte tiles must stay under 65,536 cells
// (16-bit offsets in the chunk list).  The arrays of 4-bit tiles take whole warp items of
// 32 x 32 cells, tile and halo together, so their shapes are 32 n - 2 halo.
const std::vector<TileVariant>& tile_variants() {
  constexpr int B = TileVariant::kByte | TileVariant::kByteTuned, N = TileVariant::kNibble,
                NT = TileVariant::kNibble | TileVariant::kNibbleTuned;
  static const std::vector<TileVariant> v = {
      // one frame of a small world is the latency of a few CTAs: 4-bit tiles of 64 x 32 cells with
      // their halo (us a launch, four materials, 56x30 / 128x64 bytes: 64^2 to 512^2 4.2 / 8.2, 1024^2
      // 6.2 / 8.3, 2048^2 8.3 / 11.4; twelve 4.1 / 7.6, 6.2 / 8.3, 10.3 / 12.3)
      {56, 30, 1, 128, NT, 0, 1 << 22},
      {128, 64, 1, 256, B | NT}, {256, 32, 1, 256, B | NT}, {128, 32, 1, 256, B | NT}, {128, 64, 2, 256, B},
      {128, 64, 4, 256, B},      {128, 64, 8, 256, B},      {128, 128, 8, 256, B},
      {256, 64, 4, 256, B},      {64, 64, 4, 256, B},       {256, 128, 8, 512, B},     {192, 128, 8, 256, B},
      {256, 128, 4, 512, B},     {256, 64, 8, 256, B},
      // 32x32 and 48x48 for the latency of small worlds, the large ones for the rate of large ones,
      // 96x96 between (us a frame, four materials, 32x32_k16 / 48x48_k8 / 96x96_k16 / 112x112_k8 /
      // 240x176_k8: 256^2 0.66 / 1.07 / 1.18 / 1.60 / 3.64, 1024^2 1.31 / 1.34 / 1.18 / 1.61 / 3.41, 4096^2 14.4
      // / 8.7 / 7.2 / 7.0 / 6.5; three 4096^2 worlds at once, 60 frames of one: 852 / 489 / 387 / 362 / 313 us).
      // The autotuner tries those whose range holds the world; 120x120 is for 2 to 4 frames of large worlds,
      // asked for or left at the end of a call, where the smaller halo pays for its few threads (us of 2 and 4
      // frames, twelve, 120x120_k4 / 240x176_k8 / 112x112_k8: 8192^2 119 154 / 135 184 / 130 177; 3001x2003 33 38 /
      // 36 44 / 31 39; 1000x700 25 32 / 30 39 / 20 24).
      {120, 120, 4, 128, N, 1 << 23},
      {112, 112, 8, 256, NT, 1 << 18},
      {48, 48, 8, 128, NT, 0, 1 << 23},
      {240, 176, 8, 256, NT, 1 << 22},
      {240, 240, 8, 256, NT, 1 << 23},
      {96, 96, 16, 256, NT, 0, 1 << 22},
      {32, 32, 16, 128, NT, 0, 1 << 20},
      // on 4-bit cells for callers that ask for 16 frames a launch on large worlds (us of 48 frames, four
      // materials, 128x128_k16 / 96x96_k16: 8192^2 1171 / 1262, 4096^2 352 / 363, 2500^2 182 / 163; twelve
      // 1679 / 1892, 513 / 554, 259 / 277)
      {128, 128, 16, 256, B | N, 1 << 24},
  };
  return v;
}

const TileVariant* pick_variant(int k, const LutShape& lut, long long cells) {
  const TileVariant* best = nullptr;
  for (bool ranged : {true, false}) {
    if (best) break;
    for (const TileVariant& t : tile_variants())
      if (t.kmax >= k && t.fits(lut) && (!ranged || t.holds(lut, cells)) && (!best || t.kmax < best->kmax))
        best = &t;
  }
  return best;
}

int fusion_depth(int k) {
  int depth = 0;
  for (const TileVariant& t : tile_variants())
    if (t.kmax >= k && (!depth || t.kmax < depth)) depth = t.kmax;
  return depth;
}

std::string kernel_source(const std::string& generated_rules) {
  std::ostringstream o;
  o << "#define SE_NIB_FEW_EDITS " << kFewEdits << "\n";
  o << SE_PRELUDE_SRC << "\n" << generated_rules << "\n" << SE_MARGOLUS_SRC << "\n"
    << SE_NIBBLE_SRC << "\n";
  for (const TileVariant& t : tile_variants()) {
    if (!(t.use & TileVariant::kByte)) o << "#ifdef SE_NIB\n";
    const std::string bounds = (t.kmax > 1 || t.small() ? "SE_TILE_BOUNDS(" : "__launch_bounds__(") + std::to_string(t.nt) + ") ";
    o << "extern \"C\" __global__ void " << bounds << t.name()
      << "(const uint32_t* __restrict__ src, uint32_t* __restrict__ dst, int W, int H, int f0, int k,"
         " const uint16_t* __restrict__ lut, int ya, int yb) {\n"
      << "  se_tile_impl<" << t.tw << ", " << t.th << ", " << t.kmax << ", " << t.nt
      << ">(src, dst, W, H, f0, k, lut, ya, yb);\n}\n";
    // the edit list travels in the parameter space, read in place (__grid_constant__)
    o << "extern \"C\" __global__ void " << bounds << t.edit_name()
      << "(const uint32_t* __restrict__ src, uint32_t* __restrict__ dst, int W, int H, int f0, int k,"
         " const uint16_t* __restrict__ lut, int ya, int yb, const __grid_constant__ SeEditParams edits,"
         " int nedits) {\n"
      << "  se_tile_impl<" << t.tw << ", " << t.th << ", " << t.kmax << ", " << t.nt
      << ">(src, dst, W, H, f0, k, lut, ya, yb, &edits, nedits);\n}\n";
    // batches and servers take the shapes chosen for the rule set's tiles; a world any, by set_tile
    if (!(t.use & TileVariant::kNibble)) o << "#ifndef SE_NIB\n";
    o << "extern \"C\" __global__ void " << bounds << t.multi_name()
      << "(const SeWorldDesc* __restrict__ worlds, const SeTileJob* __restrict__ jobs, int pass,"
         " int frames_done, int k, const uint16_t* __restrict__ lut) {\n"
      << "  se_mtile_impl<" << t.tw << ", " << t.th << ", " << t.kmax << ", " << t.nt
      << ">(worlds, jobs, pass, frames_done, k, lut);\n}\n";
    o << "extern \"C\" __global__ void " << bounds << t.serve_name()
      << "(const SeWorldDesc* __restrict__ descs, const int* __restrict__ prefix, int nactive,"
         " const uint16_t* __restrict__ lut) {\n"
      << "  se_stile_impl<" << t.tw << ", " << t.th << ", " << t.kmax << ", " << t.nt
      << ">(descs, prefix, nactive, lut);\n}\n";
    if (!(t.use & TileVariant::kByte) || !(t.use & TileVariant::kNibble)) o << "#endif\n";
  }
  return o.str();
}

std::string TileVariant::serve_name() const {
  return "se_stile_" + std::to_string(tw) + "x" + std::to_string(th) + "_k" + std::to_string(kmax);
}

std::string TileVariant::multi_name() const {
  return "se_mtile_" + std::to_string(tw) + "x" + std::to_string(th) + "_k" + std::to_string(kmax);
}

namespace {

std::string cache_dir() {
  if (const char* d = getenv("SE_CACHE_DIR")) return d;
  if (const char* x = getenv("XDG_CACHE_HOME")) return std::string(x) + "/sandengine_gb300";
  if (const char* h = getenv("HOME")) return std::string(h) + "/.cache/sandengine_gb300";
  return "";
}

std::string hex_digest(const std::string& s) {
  // FNV-1a 64 twice with different offsets: a cache key, not a security boundary.
  uint64_t a = 1469598103934665603ull, b = 1099511628211ull * 7ull + 13ull;
  for (unsigned char c : s) {
    a = (a ^ c) * 1099511628211ull;
    b = (b ^ c) * 0x100000001b3ull + 0x9e3779b97f4a7c15ull;
  }
  char buf[40];
  snprintf(buf, sizeof buf, "%016llx%016llx", (unsigned long long)a, (unsigned long long)b);
  return buf;
}

// parallel: the kernels of the 4-bit tiles are optimised on all cores (a rule set's first compilation
// on 8 cores: byte tiles alone 23 s, with these 33 s, in parallel 14 s; the 16384^2 world 5.59 ->
// 5.43 ms, 4096^2 313 -> 315 us).  Other rule sets' kernels came out 4% slower that way.
std::vector<std::string> nvrtc_options(bool parallel) {
  std::vector<std::string> o = {"-arch=sm_103a", "--std=c++17", "--fmad=false", "-lineinfo",
                                "--extra-device-vectorization"};
  if (parallel) o.push_back("--split-compile=0");
  return o;
}

std::mutex g_cache_mu;

}  // namespace

bool compile_cubin(const std::string& src, bool parallel, std::string* cubin, std::string* log) {
  const std::vector<std::string> options = nvrtc_options(parallel);
  int maj = 0, min = 0;
  nvrtcVersion(&maj, &min);
  std::string key_src = src + "\n//nvrtc " + std::to_string(maj) + "." + std::to_string(min);
  for (auto& o : options) key_src += "\n//" + o;
  const std::string key = hex_digest(key_src);
  const std::string dir = cache_dir();
  const std::string path = dir.empty() ? "" : dir + "/" + key + ".cubin";
  {
    std::lock_guard<std::mutex> g(g_cache_mu);
    if (!path.empty()) {
      std::ifstream f(path, std::ios::binary);
      if (f) {
        std::stringstream ss;
        ss << f.rdbuf();
        *cubin = ss.str();
        if (!cubin->empty()) return true;
      }
    }
  }
  nvrtcProgram prog;
  if (nvrtcCreateProgram(&prog, src.c_str(), "sandengine_rules.cu", 0, nullptr, nullptr) != NVRTC_SUCCESS) {
    *log = "nvrtcCreateProgram failed";
    return false;
  }
  std::vector<const char*> opts;
  for (auto& o : options) opts.push_back(o.c_str());
  nvrtcResult rc = nvrtcCompileProgram(prog, (int)opts.size(), opts.data());
  size_t lsz = 0;
  nvrtcGetProgramLogSize(prog, &lsz);
  std::string lg(lsz, '\0');
  if (lsz) nvrtcGetProgramLog(prog, lg.data());
  if (rc != NVRTC_SUCCESS) {
    *log = std::string(nvrtcGetErrorString(rc)) + "\n" + lg;
    nvrtcDestroyProgram(&prog);
    return false;
  }
  size_t csz = 0;
  nvrtcGetCUBINSize(prog, &csz);
  cubin->assign(csz, '\0');
  nvrtcGetCUBIN(prog, cubin->data());
  nvrtcDestroyProgram(&prog);
  if (!path.empty()) {
    std::lock_guard<std::mutex> g(g_cache_mu);
    std::string cmd_dir = dir;
    // mkdir -p
    for (size_t i = 1; i <= cmd_dir.size(); ++i)
      if (i == cmd_dir.size() || cmd_dir[i] == '/') mkdir(cmd_dir.substr(0, i).c_str(), 0755);
    std::string tmp = path + ".tmp" + std::to_string(getpid());
    std::ofstream f(tmp, std::ios::binary);
    if (f) {
      f.write(cubin->data(), (std::streamsize)cubin->size());
      f.close();
      rename(tmp.c_str(), path.c_str());
    }
  }
  return true;
}

Module::~Module() {
  if (lib) cudaLibraryUnload(lib);
}

size_t tile_smem_bytes(const TileVariant& t, const LutShape& lut, int nedits) {
  if (lut.nib_entries && (t.kmax > 1 || t.small())) {
    // SeNib's array (nibble.cuh), the reduced table when small, the bits and boxes of the edits
    const size_t sw16 = (size_t)(t.sw() + 15) / 16, wpr = 2 * ((sw16 + 1) / 2 * 2);
    const size_t stride = wpr + 2;
    const size_t rows = 32 * (((size_t)(t.sh() + 1) / 2 + 15) / 16) + 1;
    return (((stride * rows + 3) & ~(size_t)3) + (lut.nib_shared ? (lut.nib_entries + 3) & ~3ull : 0) +
            (nedits > kFewEdits ? 8 + 2 * SE_MAX_MODIFICATIONS : 0)) * 4;
  }
  size_t b = (t.smem_bytes() + 15) & ~(size_t)15;
  // 48-byte header (slack, list counters, uniform-material flags), then the per-step list
  // of chunks (4 blocks) to evaluate, one u16 offset each
  b += 48 + ((2 * (size_t)(t.sw() / 8) * (size_t)(t.sh() / 2) + 15) & ~(size_t)15);
  return b;
}

bool Module::load(const std::string& cubin, const LutShape& lut, std::string* err) {
  cudaError_t e = cudaLibraryLoadData(&lib, cubin.data(), nullptr, nullptr, 0, nullptr, nullptr, 0);
  if (e != cudaSuccess) {
    *err = std::string("cudaLibraryLoadData: ") + cudaGetErrorString(e);
    lib = nullptr;
    return false;
  }
  std::vector<std::string> names = {"se_edit", "se_resident", "se_batch_finalize"};
  if (lut.entries) {
    names.push_back("se_build_lut");
    names.push_back("se_build_static");
  }
  if (lut.nib_entries) names.push_back("se_build_nib");
  for (auto& t : tile_variants()) {
    if (!t.compiled(lut)) continue;
    names.push_back(t.name());
    names.push_back(t.edit_name());
    if (!t.fits(lut)) continue;
    names.push_back(t.multi_name());
    names.push_back(t.serve_name());
  }
  for (auto& n : names) {
    cudaKernel_t k;
    e = cudaLibraryGetKernel(&k, lib, n.c_str());
    if (e != cudaSuccess) {
      *err = "cudaLibraryGetKernel(" + n + "): " + cudaGetErrorString(e);
      return false;
    }
    kernels[n] = k;
  }
  for (auto& t : tile_variants()) {
    tiles.push_back(t.compiled(lut) ? kernels[t.name()] : nullptr);
    tiles.push_back(t.compiled(lut) ? kernels[t.edit_name()] : nullptr);
    if (!t.compiled(lut)) continue;
    for (const std::string& n : {t.name(), t.edit_name(), t.multi_name(), t.serve_name()}) {
      if (!kernels.count(n)) continue;
      e = cudaFuncSetAttribute((const void*)kernels[n], cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)tile_smem_bytes(t, lut, n == t.edit_name() ? SE_MAX_MODIFICATIONS : 0));
      if (e != cudaSuccess) {
        *err = std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e);
        return false;
      }
    }
  }
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  cudaFuncAttributes fa{};
  e = cudaFuncGetAttributes(&fa, (const void*)kernels["se_resident"]);
  if (e != cudaSuccess) {
    *err = std::string("cudaFuncGetAttributes(se_resident): ") + cudaGetErrorString(e);
    return false;
  }
  // static shared memory (the rule set's property tables) counts against the same limit
  max_dyn_smem = (size_t)optin - fa.sharedSizeBytes;
  e = cudaFuncSetAttribute((const void*)kernels["se_resident"], cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)max_dyn_smem);
  if (e != cudaSuccess) {
    *err = std::string("cudaFuncSetAttribute(se_resident): ") + cudaGetErrorString(e);
    return false;
  }
  return true;
}

cudaKernel_t Module::get(const std::string& name) const {
  auto it = kernels.find(name);
  return it == kernels.end() ? nullptr : it->second;
}

}  // namespace se::rt
