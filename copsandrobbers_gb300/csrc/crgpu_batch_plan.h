// crgpu_batch_plan.h - how a batch is split between teams of blocks and single blocks (host code only).
#pragma once
#include <algorithm>
#include <cstddef>
#include <functional>
#include <queue>
#include <vector>

namespace crgpu {

// order[0 .. count) goes to teams of `size` blocks, `teams` of them resident; a team has team_bytes of
// slot memory, a block of it solo_bytes once it goes on alone.
struct TeamPlan {
    int size = 1, teams = 0, count = 0;
    size_t team_bytes = 0, solo_bytes = 0;

    static TeamPlan alone(int blocks, size_t slot_bytes) { return TeamPlan{1, blocks, 0, slot_bytes, slot_bytes}; }
    int resident(int graphs) const { return std::max(1, std::min(graphs, teams)); }
    size_t bytes(int graphs) const { return (size_t)resident(graphs) * team_bytes; }
};

// Splits the batch between teams and single blocks.  Run time of a graph on one block: proportional
// to its configurations times vertices at the largest k, plus a constant for its launches' worth of
// barriers; a team of s blocks is worth a little less than s blocks (measured on 256 graphs of
// n = 128: 0.95, 0.88 and 0.78 of them for 2, 4 and 8).  Each split whose slots take less than
// `memory` bytes is played through the two queues, largest graph first, and the shortest run wins; a
// batch of more than 64 graphs per block needs no teams (the longest graph is then a small part of the
// run).  cost: of the graphs in descending order; blocks: that are resident alone; slot_bytes: of the
// largest graph; resident_teams(size): clusters of `size` blocks that are resident; solo_bytes(m): of
// the largest graph but the first m.
inline TeamPlan plan_teams(const std::vector<double>& cost, int blocks, size_t slot_bytes, size_t memory,
                           const std::function<int(int)>& resident_teams,
                           const std::function<size_t(int)>& solo_bytes) {
    const int count = (int)cost.size();
    TeamPlan best = TeamPlan::alone(blocks, slot_bytes);
    if (count > 64 * blocks) return best;
    const double fixed = 2.5e4;   // in the cost's unit
    double total = 0;
    for (double c : cost) total += c + fixed;
    auto play = [&](int size, int teams, double eff, int by_teams) {
        std::priority_queue<double, std::vector<double>, std::greater<double>> q;
        for (int t = 0; t < teams; ++t) q.push(0.0);
        double end = 0;
        for (int i = 0; i < by_teams; ++i) {
            const double t = q.top() + cost[i] / (size * eff) + 1.5 * fixed;
            q.pop();
            q.push(t);
            end = std::max(end, t);
        }
        std::vector<double> at;
        for (; !q.empty(); q.pop())
            for (int k = 0; k < size; ++k) at.push_back(q.top());
        std::priority_queue<double, std::vector<double>, std::greater<double>> r(std::greater<double>(), std::move(at));
        for (int i = by_teams; i < count; ++i) {
            const double t = r.top() + cost[i] + fixed;
            r.pop();
            r.push(t);
            end = std::max(end, t);
        }
        return end;
    };
    double shortest = play(1, blocks, 1.0, 0);
    const struct { int size; double eff; } kinds[] = {{2, 0.95}, {4, 0.88}, {8, 0.78}};
    for (const auto& k : kinds) {
        const int teams = resident_teams(k.size);
        if (teams <= 0) continue;
        int last = -1;
        for (double f = 2.0; f > 0.01; f /= 1.6) {
            // the graphs longer than a share f of the ideal run
            int m = 0;
            while (m < count && cost[m] > f * total / blocks) ++m;
            if (m == last || m == 0) continue;
            last = m;
            const size_t solo = solo_bytes(m);
            const TeamPlan plan{k.size, teams, m, std::max(slot_bytes, k.size * solo), solo};
            if (plan.bytes(count) >= memory) continue;
            const double t = play(k.size, teams, k.eff, m);
            if (t < 0.98 * shortest) {
                shortest = t;
                best = plan;
            }
        }
    }
    return best;
}

}  // namespace crgpu
