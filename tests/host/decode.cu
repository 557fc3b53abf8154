// The arguments of the library's kernels, for cuda_stub.cpp.  The Reyes arguments are
// declared in the kernels' own file, which is therefore compiled here.
#include "../../piko-public_b200/csrc/reyes_kernels.cu"

#include "cuda_stub.h"

unsigned stub_frontier = 0, stub_leaves = 0;

std::string stub_kernel_name(const char* mangled)
{
  for (const char* n : {"raster_setup", "raster_large_count", "scan_tiles", "raster_scatter", "raster_frag8", "raster_bins",
                        "reyes_split", "reyes_dice", "reyes_big", "reyes_ties", "reyes_pixels"})
    if (strstr(mangled, n)) return n;
  return mangled;
}

StubLaunch stub_decode(const char* name, void** args)
{
  StubLaunch l;
  if (!strncmp(name, "reyes_wait", 10)) return l;
  if (!strncmp(name, "reyes", 5)) {
    const ReyesArgs a = *static_cast<const ReyesArgs*>(args[0]);
    l.objects = {a.ctr, a.samp};
    l.null_argument = !a.in_patches || !a.lvl[0] || !a.lvl[1] || !a.stack || !a.leaves || !a.up || !a.id_color || !a.id_key ||
                      !a.ties || !a.ctr || !a.host_ctr || !a.fb || !a.depth || !a.samp || !a.first0;
    if (!strcmp(name, "reyes_pixels"))
      l.counts = [a](bool) {
        ReyesCounters c = {};
        if (stub_frontier || stub_leaves) c.fc.status = kStatusPatchOverflow;
        c.level_count[1] = stub_frontier;
        c.leaf_meta = (unsigned long long)stub_leaves << 40;
        stub_frontier = stub_leaves = 0;
        *a.host_ctr = c;
      };
    if (!strcmp(name, "reyes_split")) l.cameras = [a] { return std::vector<float>{(float)a.lvl_cap, (float)a.leaf_cap}; };
    if (!strcmp(name, "reyes_pixels")) l.cameras = [a] { return std::vector<float>{a.vp[12]}; };
    return l;
  }
  const RasterFrameArgs a = *static_cast<const RasterFrameArgs*>(args[0]);
  l.objects = {a.work};
  const bool noalloc = !a.chunk_desc;
  l.null_argument = !a.setup || !a.tile_cnt || !a.tile_span || !a.tile_list || !a.pair_tl || !a.pair_g || !a.large_seg ||
                    !a.large_walk || !a.work || !a.ctr ||
                    (noalloc ? !a.heavy : !a.hdone || !a.chunk_keys || !a.host_bin) || (a.n_scenes > 1 && !a.scenes);
  if (!strcmp(name, "raster_frag8") || !strcmp(name, "raster_bins")) {
    if (a.host_bin)
      l.counts = [a](bool overflow) {
        a.host_bin->status = overflow ? kStatusListOverflow : 0u;
        a.host_bin->list_total = overflow ? a.list_cap + 1u : 0u;
        static unsigned frames = 0;
        a.ctr->covered = ++frames;
      };
    l.cameras = [a] {
      std::vector<float> c;
      for (int i = 0; i < a.n_scenes; ++i) c.push_back((a.scenes ? a.scenes[i] : a.one).vp[12]);
      return c;
    };
  }
  return l;
}

extern "C" uint32_t stub_next_patches(uint32_t count, uint32_t cap) { return next_patches(count, cap); }

extern "C" void stub_setup_shape(uint32_t n, uint32_t wave, uint32_t threads, uint32_t* batch, uint32_t* blocks)
{
  const SetupShape s = setup_shape(n, wave, threads);
  *batch = s.batch;
  *blocks = s.blocks;
}
