// NVRTC compilation of a rule set's kernels for sm_103a, with an on-disk cubin cache, and
// loading through the CUDA runtime's library API (no link-time dependency on libcuda).
#pragma once

#include <cuda_runtime.h>

#include <map>
#include <string>
#include <vector>

namespace se::rt {

// Size of a rule set's block transition table: its u16 entries and the 32-bit words of the
// bitset of static keys that follows it (both 0 without a table).
struct LutShape {
  unsigned long long entries = 0, static_words = 0;
  // Rule sets whose tiles pack two cells a byte (nibble.cuh): the entries of the reduced table
  // (0: byte tiles), whether each CTA copies it into shared memory, and the 32-bit words of
  // all that follows the static bits.
  unsigned long long nib_entries = 0, nib_words = 0;
  bool nib_shared = false;
};

// A tile-kernel instantiation: TW x TH output cells, up to KMAX frames per launch.
struct TileVariant {
  int tw, th, kmax, nt;
  enum { kByte = 1, kNibble = 2, kByteTuned = 4, kNibbleTuned = 8 };
  int use;  // the kinds of tile it is chosen for, and tried for by the autotuner (set_tile may ask for any)
  long long min_cells = 0, max_cells = 1ll << 62;  // as a 4-bit tile, for worlds of so many cells
  // Whether the rule set's module holds it: shapes for 4-bit tiles only where there are such.
  bool compiled(const LutShape& lut) const { return (use & kByte) || lut.nib_entries; }
  bool fits(const LutShape& lut) const { return use & (lut.nib_entries ? kNibble : kByte); }
  // Whether the autotuner tries it on `cells` cells (of one world, or of a batch's tiled worlds).
  bool tuned(const LutShape& lut, long long cells) const {
    return (use & (lut.nib_entries ? kNibbleTuned : kByteTuned)) && holds(lut, cells);
  }
  bool holds(const LutShape& lut, long long cells) const {
    return !lut.nib_entries || (cells >= min_cells && cells <= max_cells);
  }
  bool small() const { return tw * th <= 2048; }  // one-frame tiles on 4-bit cells (se_tile_run)
  std::string name() const;        // single-world kernel
  std::string edit_name() const;   // single-world kernel with the first frame's edit pass
  std::string multi_name() const;  // many-world (tile job list) kernel
  std::string serve_name() const;  // serving iteration kernel (per-world frame counts)
  int halo_x() const { return ((kmax + 3) / 4) * 4; }
  int halo_y() const { return kmax; }
  int sw() const { return tw + 2 * halo_x(); }  // shared array: tile plus halo
  int sh() const { return th + 2 * halo_y(); }
  size_t smem_bytes() const { return (size_t)sw() * (size_t)sh(); }
};
const std::vector<TileVariant>& tile_variants();
// The variant for k frames per launch: of those chosen for the rule set's tiles and for `cells` cells
// (of one world, or of all that a launch advances) the first with the fewest frames >= k.
const TileVariant* pick_variant(int k, const LutShape& lut, long long cells);
// The frames that a launch advances where k are asked for, whichever shape takes it: the fewest
// >= k of any shape, 0 beyond them all.
int fusion_depth(int k);

// Edit lists up to this long are applied mod by mod in 4-bit tiles (se_nib_few_edits; us of a frame on
// 256 x 256, four materials, waited for, so / the longer lists' way: 1 circle 14.9 / 16.7, 2 15.5 / 17.2, 4
// 23.4 / 21.8).
constexpr int kFewEdits = 4;
// Dynamic shared memory of a tile launch: the u8 tile, then the per-step list of chunks to
// evaluate; or the 4-bit tile and a small reduced table.  The block transition table and its
// static-key bitset stay in global memory (read through the read-only cache).
// nedits: the mods of an edit launch; the bits and boxes of a long list take 2 KB, which shorter ones leave
// to L1 (frame, light and image of 1920 x 1080, twelve materials, two mods: 51.2 us with them, 50.8 without).
size_t tile_smem_bytes(const TileVariant& t, const LutShape& lut, int nedits = 0);

// Full device source: prelude + generated rules + kernel template + instantiations.
std::string kernel_source(const std::string& generated_rules);

// Compiles `src` to an sm_103a cubin (cached by content hash).  No GPU needed.
bool compile_cubin(const std::string& src, bool parallel, std::string* cubin, std::string* log);

struct Module {
  cudaLibrary_t lib = nullptr;
  std::map<std::string, cudaKernel_t> kernels;
  std::vector<cudaKernel_t> tiles;  // of each variant: the plain kernel, the one with edits
  size_t max_dyn_smem = 0;  // opt-in dynamic shared memory per CTA on this device
  ~Module();
  bool load(const std::string& cubin, const LutShape& lut, std::string* err);
  cudaKernel_t get(const std::string& name) const;
  // The variant's kernel (t: an element of tile_variants()), without building its name.
  cudaKernel_t tile(const TileVariant& t, bool edits) const {
    return tiles[2 * (size_t)(&t - tile_variants().data()) + (edits ? 1 : 0)];
  }
};

}  // namespace se::rt
