// Which normalisation rows are held in registers by a cluster of CTAs (norm_resident.cuh) and which take the streaming kernels: host
// arithmetic on sizes only.
//
// A row that fits is not always better off resident: the CTAs of a cluster load, meet and store in step, and a new cluster starts only when
// as many slots as it has ranks are free.  Where planes are not whole 16-byte pieces the resident kernels also move one value at a time, four
// times the instructions a byte, and a forward pass of several waves of wide clusters then takes longer than the streaming form.
// Measured, resident over streaming time, medians over 700 random layers of up to 700 MB and a grid of ranks x waves x planes, three sets of
// tensors in turn.  Columns: ranks that the row needs; a wave is four CTAs on every SM.
//               waves:  up to 1                1 to 2                 2 to 4                 more
//               ranks:  1   2  3-4 5-8 9-16    1   2  3-4 5-8 9-16    1   2  3-4 5-8 9-16    1   2  3-4 5-8 9-16
//   batch norm, units of 16 bytes
//     forward          .47 .51 .53 .54 .60    .50 .69 .73 .84 .91    .65 .79 .76 .86 .97    .60 .69 .73 .78 .93
//     backward         .50 .50 .52 .50 .57    .55 .63 .69 .76 .89    .67 .68 .71 .79 .96     -  .67 .71 .73 .95
//   batch norm, single values
//     forward          .53 .54 .57 .64 .65    .75 .81 .88 .83 .98    .79 .98 .99 1.10 1.18  .69 .90 1.06 1.12 1.26
//       planes of 65 to 256 values, which the streaming form reads a value at a time too: .19 to 1.10, median .48, beyond one wave
//     backward         .52 .51 .51 .50 .55    .67 .72 .66 .71 .82    .66 .74 .71 .76 .91    .69 .73 .75 .77 .87
//   group norm, units of 16 bytes
//     forward          .79 .79 .67 .49 .41    .56 .88 .92 .82 .60    .49 .90 .99 .94 .91    .48 1.00 1.00 .92 .99
//     backward        1.05 .92 .81 .59 .40    .94 .77 1.04 .81 .66    -  .79 .91 .96 .85     -  .70 .98 .83 .91
//   group norm, single values
//     forward          .73 .74 .67 .55 .46    .69 .85 .95 1.11 .70   .41 .84 .97 1.08 .85   .41 .75 .96 1.13 1.03
//       three and four ranks, up to 444 rows (one wave of the streaming kernel): .79 to 1.59, planes of 225 to 361 values .79 to 1.09
//     backward        1.08 .93 .78 .57 .36   1.11 1.11 1.04 .82 .52  .51 1.01 .95 .96 .73   .49 .78 .93 .90 .76
#pragma once

namespace b200 {
namespace nres {

constexpr int PLAN_THREADS = 256, PLAN_MAX_RANKS = 16;

struct RankPlan {
  int ranks = 0;        // CTAs of a cluster, 0: the row does not fit
  int need = 0;         // of which the row needs so many
  double waves = 0;     // of all CTAs at four to an SM
};

// `units` of a row, of which a thread holds up to `most`.  As few ranks as hold the row (a wider exchange costs more than a fuller
// thread: 256 channels of 12544 values forward 9.5 us with 2 ranks of eight units a thread, 12.5 with 4 of four), then up to eight by doubling
// while all CTAs still run at once and a thread has more than two units (20 rows and fewer would leave most SMs idle).  Between nine and
// sixteen a cluster has what the row needs: with sixteen for all of them a row of nine took 1.7 times as long.
inline RankPlan plan_ranks(long long units, long long rows, int most, int sms) {
  RankPlan p;
  const long long holds = (long long)PLAN_THREADS * most, need = (units + holds - 1) / holds;
  if (need > PLAN_MAX_RANKS) return p;
  long long ranks = need;
  while (ranks <= 4 && rows * ranks * 2 <= 4ll * sms && units > ranks * PLAN_THREADS * 2) ranks *= 2;
  p.need = (int)need;
  p.ranks = (int)ranks;
  p.waves = (double)(rows * ranks) / (4.0 * sms);
  return p;
}

// Rows whose units wait in the shared memory of a cluster's CTAs, `unit_bytes` for each: as few ranks as hold the row with four CTAs to an SM
// (`quarter` bytes each), or sixteen with up to two to an SM.
constexpr int PLAN_STAGED_BYTES = 100 * 1024;
struct StagedPlan {
  int ranks = 0;        // 0: the row does not fit
  int units = 0;        // of a thread
};
inline StagedPlan plan_staged(long long units, int unit_bytes, int quarter) {
  StagedPlan p;
  const long long holds = (long long)PLAN_THREADS * (quarter / (PLAN_THREADS * unit_bytes)), need = (units + holds - 1) / holds;
  const long long ranks = need < PLAN_MAX_RANKS ? need : PLAN_MAX_RANKS, per = (units + ranks - 1) / ranks, mine = (per + PLAN_THREADS - 1) / PLAN_THREADS;
  if (mine * PLAN_THREADS * unit_bytes > PLAN_STAGED_BYTES) return p;
  p.ranks = (int)ranks;
  p.units = (int)mine;
  return p;
}

// The line through the table above, for rows beyond one wave; `plane`: values of a plane, `vec`: values of a unit.
inline bool batch_norm_resident(const RankPlan& p, int vec, long long plane, bool backward) {
  if (p.ranks == 0) return false;
  if (p.waves <= 2.0 || vec == 4 || backward) return true;
  return p.need <= 2 || (p.need <= 4 && p.waves <= 4.0) || (p.need <= 8 && plane > 64 && plane <= 256);
}
inline bool group_norm_resident(const RankPlan& p, int vec, long long plane, bool backward, bool stream_in_one_wave) {
  if (p.ranks == 0) return false;
  if (p.waves <= 1.0 || vec == 4 || backward) return true;
  if (p.need > 8) return p.waves <= 4.0;
  return p.need <= 2 || plane <= 256 || (p.need <= 4 && !stream_in_one_wave);
}

}  // namespace nres
}  // namespace b200
