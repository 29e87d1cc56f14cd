// Runs the plan build's host phases (spearfish_gb300/csrc/sf_plan.cu) without a GPU: reads a plan
// from the file named on the command line -- four 64-bit words (SMs, pool bytes, scores, jobs),
// the scores, the jobs -- and prints its description, each job's bucket and the sizes it takes.
#include "../spearfish_gb300/csrc/sf_plan.cu"

#include <cstdio>

using namespace sfe;

int main(int argc, char** argv) {
  FILE* f = std::fopen(argv[1], "rb");
  uint64_t head[4];
  if (!f || std::fread(head, 8, 4, f) != 4) return 2;
  std::vector<sf_affine_t> scores(head[2]);
  std::vector<sf_job_t> jobs(head[3]);
  if (std::fread(scores.data(), sizeof(sf_affine_t), scores.size(), f) != scores.size() ||
      std::fread(jobs.data(), sizeof(sf_job_t), jobs.size(), f) != jobs.size())
    return 2;
  std::fclose(f);
  sf_context ctx;
  ctx.sms = (int)head[0];
  sf_plan P;
  P.ctx = &ctx;
  P.shared = argc > 2;  // as a server's slot
  P.pool_bytes = head[1];
  P.scratch.reset(new BuildScratch);
  BuildScratch& S = *P.scratch;
  if (jobs_to_passes(jobs.data(), jobs.size(), scores.data(), (uint32_t)scores.size(), head[1], P.passes) ||
      build_sequences(&P, S)) {
    std::printf("%s\n", last_error().c_str());
    return 1;
  }
  // Each pass's sequences lie where its words begin.
  std::map<uint64_t, std::pair<uint64_t, uint32_t>> placed;
  for (size_t u = 0; u < P.seq_len.size(); ++u) placed[P.seq_woff[u]] = {P.seq_boff[u], P.seq_len[u]};
  for (size_t q = 0; q < jobs.size(); ++q) {
    const Pass& p = P.passes[q];
    if (placed[S.word_of[2 * q]] != std::make_pair(p.p_off, p.m) ||
        placed[S.word_of[2 * q + 1]] != std::make_pair(p.t_off, p.n))
      return 3;
  }
  choose_chains(&P, S, allow16());
  if (describe_passes(&P, S, allow16())) return 1;
  lay_out_outputs(&P, S);
  build_chains(&P, S);
  build_buckets(&P, S);
  describe_plan(&P, S);
  std::vector<uint32_t> at(jobs.size());
  if (plan_job_buckets(&P, at.data(), at.size())) return 1;
  std::printf("{\"plan\": %s, \"job_buckets\": [", P.desc.c_str());
  for (size_t q = 0; q < at.size(); ++q) std::printf("%s%d", q ? ", " : "", (int)at[q]);
  std::printf("], \"launches\": [");
  for (size_t q = 0; q < P.groups.size(); ++q)
    std::printf("%s{\"stream\": %d, \"lead\": %s, \"warps\": %d, \"tasks\": %u}", q ? ", " : "",
                P.groups[q].stream, P.groups[q].lead ? "true" : "false",
                P.groups[q].grid * P.groups[q].block / 32, P.groups[q].task_count);
  // The passes of each class in a plan of their own, as the autotuner times them: how many get
  // another class there.
  std::map<std::tuple<int, int, int, int, int>, std::vector<size_t>> alike;
  for (size_t q = 0; q < jobs.size(); ++q) {
    const BucketKey& k = S.per[q].first;
    alike[{k.kind, k.c, k.wide, k.tb, k.lanes}].push_back(q);
  }
  size_t strays = 0;
  for (const auto& g : alike) {
    sf_plan T;
    T.ctx = &ctx;
    T.pool_bytes = P.pool_bytes;
    T.scratch.reset(new BuildScratch);
    choose_as(&P, &T);
    for (size_t q : g.second) T.passes.push_back(P.passes[q]);
    if (build_sequences(&T, *T.scratch)) return 1;
    choose_chains(&T, *T.scratch, allow16());
    if (describe_passes(&T, *T.scratch, allow16())) return 1;
    for (const auto& it : T.scratch->per) strays += !(it.first == S.per[g.second[0]].first);
  }
  std::printf("], \"strays\": %zu, \"myers_kcut\": %s", strays, P.myers_kcut ? "true" : "false");
  // What upload_plan asks for, buffer by buffer.
  const uint64_t needs = P.pool_bytes + 4 * P.pool_words + 20 * P.seq_len.size() +
                         S.dj.size() * (sizeof(DJob) + sizeof(DParams) + sizeof(DRes) + sizeof(TJob) + sizeof(TRes)) +
                         S.mj.size() * (sizeof(MJob) + 4) + 4 * P.tb_words + 8 * P.ops_words + 12 * S.wlist.size() +
                         4 * S.order.size() + sizeof(uint2) * S.tasks.size() + 4 * P.buckets.size() +
                         4 * S.scratch_total + 14 * 64;
  std::printf(", \"tb_words\": %llu, \"pool_words\": %llu, \"sequences\": %zu, \"needs\": %llu, "
              "\"estimate\": %llu}\n",
              (unsigned long long)P.tb_words, (unsigned long long)P.pool_words, P.seq_len.size(),
              (unsigned long long)(needs + needs / 4 + 14 * 256),
              (unsigned long long)plan_bytes_estimate(P.passes, P.pool_bytes));
  return 0;
}
