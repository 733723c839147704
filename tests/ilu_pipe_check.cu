// Host-only check of the pipelined triangular solves' plan
// (tnl_b200/csrc/ilu_pipe.cuh): for grids, bands and random lower triangles
// over a range of sizes and part counts, every row has one packed position
// inside the plan, steps start at multiples of 4 and hold at most
// kPipeStepRows rows, and a run of the parts' steps, each step taken as soon
// as the waits of its external entries allow, finishes (no deadlock) with
// every entry reading the row it means: from the ring slot that holds it, or
// from a row its owner has finished -- for the part's own old rows so long
// ago that the stage's refill cannot overtake it.  And the choice of parts: a
// chain of rows up to 8M long, one or eight entries a row, is one part, as
// long as its steps one after the other, whatever parts it is cut into; grids
// keep their parts and are a fraction of their one-part length.  Prints one
// line "ok <entries>" or the first violation.
#include <cstdint>
#include <cstdio>
#include <random>
#include <vector>

#include "ilu_pipe.cuh"

using namespace tnlb;

namespace {

int64_t checked = 0;

int fail(const char* what, int32_t n, int32_t parts, int32_t i)
{
   std::printf("violation: %s (n=%d, parts=%d, row %d)\n", what, n, parts, i);
   return 1;
}

// rp/cols: strictly lower triangle (upper: strictly upper)
int check(const std::vector<int32_t>& rp, const std::vector<int32_t>& cols, bool upper, int32_t parts)
{
   const int32_t n = (int32_t)rp.size() - 1;
   std::vector<int32_t> lev(n, 0);
   int32_t lmax = 0;
   for (int32_t k = 0; k < n; k++) {
      const int32_t i = upper ? n - 1 - k : k;
      for (int32_t q = rp[i]; q < rp[i + 1]; q++) lev[i] = std::max(lev[i], lev[cols[q]] + 1);
      lmax = std::max(lmax, lev[i]);
   }
   const PipePlan P = pipe_plan(lev, lmax, parts);
   std::vector<int32_t> beg(rp.begin(), rp.end() - 1), end(rp.begin() + 1, rp.end());
   const PipeBuild b{P.rows_at.data(), P.pos.data(), P.step.data(), beg.data(), end.data(), cols.data(),
                     P.part_step.data(), P.steps.data(), P.npad, P.chunk, 0};
   if ((int32_t)P.part_step.size() != parts + 1) return fail("parts", n, parts, 0);
   int64_t rows = 0;
   int32_t at = 0;
   for (const PipeStep& s : P.steps) {
      if (s.t0 != at || s.t0 % 4 || s.rows < 1 || s.rows > kPipeStepRows) return fail("step", n, parts, s.t0);
      at += (s.rows + 3) / 4 * 4;
      rows += s.rows;
   }
   if (rows != n || at != P.npad) return fail("rows", n, parts, 0);
   for (int32_t i = 0; i < n; i++)
      if (P.pos[i] < 0 || P.pos[i] >= P.npad || P.rows_at[P.pos[i]] != i || P.pos[i] < P.steps[P.step[i]].t0 ||
          P.pos[i] >= P.steps[P.step[i]].t0 + P.steps[P.step[i]].rows || P.step[i] < P.part_step[i / P.chunk] ||
          P.step[i] >= P.part_step[i / P.chunk + 1])
         return fail("position", n, parts, i);
   std::vector<std::vector<int32_t>> ring(parts, std::vector<int32_t>(kPipeWindow, -1));
   std::vector<int32_t> done(parts, 0);
   int64_t left = (int64_t)P.steps.size();
   while (left > 0) {
      bool moved = false;
      for (int32_t p = parts - 1; p >= 0; p--) {
         const int32_t count = P.part_step[p + 1] - P.part_step[p];
         while (done[p] < count) {
            const PipeStep s = P.steps[P.part_step[p] + done[p]];
            const int32_t send = s.t0 + s.rows;
            bool ready = true;
            for (int32_t t = s.t0; t < send && ready; t++) {
               const int32_t i = P.rows_at[t];
               for (int32_t q = rp[i]; q < rp[i + 1]; q++) {
                  const int32_t col = cols[q], owner = col / P.chunk;
                  if (pipe_in_ring(b, i, col, send)) continue;
                  const int32_t need = owner == p ? 0 : P.step[col] - P.part_step[owner] + 1;
                  if (owner == p && P.step[col] - P.part_step[p] > done[p] - kPipeMaxStages)
                     return fail("own external entry too young", n, parts, i);
                  if (done[owner] < need) ready = false;
               }
            }
            if (!ready) break;
            for (int32_t t = s.t0; t < send; t++) {
               const int32_t i = P.rows_at[t];
               for (int32_t q = rp[i]; q < rp[i + 1]; q++, checked++)
                  if (pipe_in_ring(b, i, cols[q], send) && ring[p][P.pos[cols[q]] & (kPipeWindow - 1)] != cols[q])
                     return fail("ring slot", n, parts, i);
            }
            // a step's own writes must not reach a slot that the step reads: checked by reading after them too
            for (int32_t t = s.t0; t < send; t++) ring[p][t & (kPipeWindow - 1)] = P.rows_at[t];
            for (int32_t t = s.t0; t < send; t++) {
               const int32_t i = P.rows_at[t];
               for (int32_t q = rp[i]; q < rp[i + 1]; q++)
                  if (pipe_in_ring(b, i, cols[q], send) && ring[p][P.pos[cols[q]] & (kPipeWindow - 1)] != cols[q])
                     return fail("ring slot overwritten within the step", n, parts, i);
            }
            done[p]++;
            left--;
            moved = true;
         }
      }
      if (!moved) return fail("deadlock", n, parts, 0);
   }
   return 0;
}

void grid(int nx, int ny, int nz, bool upper, std::vector<int32_t>& rp, std::vector<int32_t>& cols)
{
   rp.assign(1, 0);
   cols.clear();
   for (int z = 0; z < nz; z++)
      for (int y = 0; y < ny; y++)
         for (int x = 0; x < nx; x++) {
            const int32_t i = (z * ny + y) * nx + x;
            if (!upper) {
               if (z > 0) cols.push_back(i - nx * ny);
               if (y > 0) cols.push_back(i - nx);
               if (x > 0) cols.push_back(i - 1);
            }
            else {
               if (x < nx - 1) cols.push_back(i + 1);
               if (y < ny - 1) cols.push_back(i + nx);
               if (z < nz - 1) cols.push_back(i + nx * ny);
            }
            rp.push_back((int32_t)cols.size());
         }
}

// every row depends on the `width` rows before it (upper: after it)
int check_chain(int32_t n, int32_t width, bool upper)
{
   std::vector<int32_t> beg(n), end(n), cols;
   cols.reserve((size_t)n * width);
   for (int32_t i = 0; i < n; i++) {
      beg[i] = (int32_t)cols.size();
      for (int32_t d = 1; d <= width; d++) {
         const int32_t c = upper ? i + d : i - d;
         if (c >= 0 && c < n) cols.push_back(c);
      }
      end[i] = (int32_t)cols.size();
   }
   std::vector<int32_t> lev(n), level(n + 1);
   for (int32_t i = 0; i < n; i++) lev[i] = upper ? n - 1 - i : i;
   for (int32_t i = 0; i <= n; i++) level[i] = i;
   const int32_t parts = pipe_parts(n, 148);
   double ns = 0;
   const PipePlan P = pipe_choose(lev, level, parts, beg, end, 0, cols, upper, &ns);
   if (P.parts != 1 || ns < kPipeStepNs * n) return fail("chain in several parts", n, P.parts, 0);
   const PipePlan Q = pipe_plan(lev, n - 1, parts);
   if (pipe_schedule_ns(Q, beg, end, 0, cols, upper) < kPipeStepNs * n) return fail("chain too short", n, parts, 0);
   return 0;
}

int check_grid_choice(int nx, int ny)
{
   std::vector<int32_t> rp, cols;
   grid(nx, ny, 1, false, rp, cols);
   const int32_t n = nx * ny, parts = pipe_parts(n, 148);
   std::vector<int32_t> lev(n), level(nx + ny, 0), beg(rp.begin(), rp.end() - 1), end(rp.begin() + 1, rp.end());
   for (int32_t i = 0; i < n; i++) level[(lev[i] = i % nx + i / nx) + 1]++;
   for (size_t l = 1; l < level.size(); l++) level[l] += level[l - 1];
   double ns = 0;
   const PipePlan P = pipe_choose(lev, level, parts, beg, end, 0, cols, false, &ns);
   double one = 0;
   for (size_t l = 0; l + 1 < level.size(); l++) one += kPipeStepNs * ((level[l + 1] - level[l] + 255) / 256);
   if (P.parts != parts || ns < kPipeStepNs * (nx + ny - 1) || ns > 0.7 * (one + kPipeRowNs * n))
      return fail("grid's choice", n, P.parts, 0);
   return 0;
}

}  // namespace

int main()
{
   for (bool upper : {false, true})
      for (int32_t n : {20000, 1000003, 4000000, 8000000})
         for (int32_t width : {1, 8})
            if ((int64_t)n * width <= 16000000 && check_chain(n, width, upper)) return 1;
   if (check_grid_choice(1000, 1024) || check_grid_choice(700, 1900)) return 1;
   std::mt19937 rng(1);
   std::vector<int32_t> rp, cols;
   const int sizes[][3] = {{1, 1, 1}, {5, 7, 1}, {300, 1, 1}, {257, 255, 1}, {1, 600, 1}, {31, 33, 29}, {700, 90, 1}};
   for (auto& g : sizes)
      for (int parts : {1, 2, 3, 7, 20})
         for (bool upper : {false, true}) {
            grid(g[0], g[1], g[2], upper, rp, cols);
            if (check(rp, cols, upper, parts)) return 1;
         }
   // random rows: up to 8 entries, anywhere or within a band (few long levels, many short ones, empty rows)
   for (int c = 0; c < 60; c++) {
      const int32_t n = 1 + (int32_t)(rng() % 20000), band = c % 3 == 0 ? n : 1 + (int32_t)(rng() % 9000);
      const bool upper = c & 1;
      rp.assign(1, 0);
      cols.clear();
      for (int32_t i = 0; i < n; i++) {
         const int32_t room = std::min(band, upper ? n - 1 - i : i), k = room > 0 ? (int32_t)(rng() % 9) : 0;
         std::vector<int32_t> row;
         for (int32_t q = 0; q < k; q++) {
            const int32_t d = 1 + (int32_t)(rng() % room);
            row.push_back(upper ? i + d : i - d);
         }
         std::sort(row.begin(), row.end());
         cols.insert(cols.end(), row.begin(), row.end());
         rp.push_back((int32_t)cols.size());
      }
      for (int parts : {1, 4, 15, 127})
         if (check(rp, cols, upper, parts)) return 1;
   }
   std::printf("ok %lld\n", (long long)checked);
   return 0;
}
