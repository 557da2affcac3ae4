// Prints what representative threads of one block of an attention kernel do: trace FORM TILES MODE STATE
//   FORM   pair, pieces (attn_kernel.cuh) or solo (attn_solo.cuh), with "8" behind it for E4M3 scores
//   MODE   steady, growing (the offset moves at every tile) or bounded
//   STATE  fresh, or carried (a running state comes in and goes out)
#include <string>
#include <vector>

#include "attn_solo.cuh"

Index3 threadIdx, blockIdx;

using namespace dtb;

int main(int argc, char** argv) {
  if (argc != 5) return 2;
  const std::string form = argv[1], mode = argv[3];
  const int n = std::atoi(argv[2]);
  const bool carried = argv[4] == std::string("carried"), solo = form.compare(0, 4, "solo") == 0, pieces = form == "pieces";
  const bool fp8 = form.back() == '8';
  constexpr int rows = kQTiles * kBlockM;
  std::vector<__nv_bfloat16> o(rows * kHeadDim);
  std::vector<float> acc(rows * (kHeadDim + 2));
  const float mk[2] = {0.f, 1.f};
  AttnKernelParams p = {};
  p.tmap_q.name = 'Q'; p.tmap_k.name = 'K'; p.tmap_v.name = 'V';
  p.o = o.data();
  p.o_stride_s = kHeadDim;
  p.acc_o = acc.data(); p.acc_m = acc.data() + rows * kHeadDim; p.acc_l = p.acc_m + rows;
  p.mk = mode == "bounded" ? mk : nullptr;
  p.B = p.Hq = p.Hkv = p.num_splits = 1;
  p.Sq = solo ? kBlockM : rows;
  p.Skv = (n + (pieces ? 2 : 0)) * kBlockN;
  p.acc_init = !carried;
  p.scale_log2 = 1.f;
  PieceTable tb = {};
  tb.n_pieces = tb.q_blocks = 1;
  tb.tile_begin[0] = 2;               // of the unit's n + 2 key tiles the piece takes the last n
  tb.tile_end[0] = static_cast<uint16_t>(n + 2);

  auto run = [&](const char* role, int thread) {
    std::memset(smem_raw, 0, sizeof(smem_raw));
    threadIdx = {static_cast<unsigned>(thread), 0, 0};
    growing = mode == "growing";
    tiles_read = 0;
    std::printf("thread %s\n", role);
    if (pieces) attn_fwd_pieces_kernel(p, tb);
    else if (solo && fp8) carried ? attn_solo_kernel<true, true>(p) : attn_solo_kernel<false, true>(p);
    else if (solo) carried ? attn_solo_kernel<true, false>(p) : attn_solo_kernel<false, false>(p);
    else if (fp8) carried ? attn_fwd_kernel<true, true>(p) : attn_fwd_kernel<false, true>(p);
    else carried ? attn_fwd_kernel<true, false>(p) : attn_fwd_kernel<false, false>(p);
  };
  run("load", kLoadWarp * 32);
  run("scores", kMmaWarp * 32);
  run("values", kPvWarp * 32);
  for (int group = 0; group < kQTiles; ++group)
    for (int w = 0; w < 2; ++w) {       // a thread of the group's first warp and one of its second
      const std::string role = "group" + std::to_string(group) + "." + std::to_string(w);
      run(role.c_str(), group * kBlockM + 32 * w);
    }

  auto name = [&](const char* what, const void* bar) { std::printf("name %u %s\n", smem_u32(bar), what); };
  auto names = [&](auto* b, int stages) {
    for (int i = 0; i < stages; ++i) { name("kv_full", &b->kv_full[i]); name("kv_empty", &b->kv_empty[i]); }
    for (int t = 0; t < kQTiles; ++t) {
      name("s_full", &b->s_full[t]); name("p_lo", &b->p_lo[t]); name("p_hi", &b->p_hi[t]); name("pv_done", &b->pv_done[t]);
    }
    name("s_free", &b->s_free);
  };
  if (solo) {
    auto* b = reinterpret_cast<SoloBarriers*>(smem_raw + kTileBytes + kSoloStages * kTileBytes);
    names(b, kSoloStages);
    name("q_full", &b->q_full[0]);
    name("solo_ready", &b->solo_ready);
  } else {
    auto* b = reinterpret_cast<PipelineBarriers*>(smem_raw + kQTiles * kTileBytes + kStages * kTileBytes);
    names(b, kStages);
    for (int t = 0; t < kQTiles; ++t) name("q_full", &b->q_full[t]);
  }
}
