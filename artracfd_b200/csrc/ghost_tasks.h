// Copy tasks of the one-launch ghost fill (host code, no CUDA dependence
// beyond the int2/int4 vector types, so that a host-only test can compile it).
//
// The copies of a fill (destination, source node index) read only nodes the
// fill does not change, so their order is free.  Runs of copies whose
// destinations and sources both advance by one node (rows of a periodic or
// outflow ghost plane) become tasks, one warp or block each (ghost_program), a
// run longer than kGhostLong cut into pieces of at most that many.  A task is
// (first destination, source offset, length, 0).  The
// copies of runs shorter than kGhostMinRun are returned one by one (`single`, a
// thread each).
#pragma once

#include <algorithm>
#include <vector>

constexpr int kGhostLong = 2048;
constexpr int kGhostMinRun = 32;

template <class Int2, class Int4>
void ghost_copy_tasks_of(const std::vector<Int2> &pairs, std::vector<Int4> &tasks, std::vector<Int2> &single)
{
    auto task = [&](size_t q, size_t len) {
        Int4 t;
        t.x = pairs[q].x;
        t.y = pairs[q].y - pairs[q].x;
        t.z = (int)len;
        t.w = 0;
        tasks.push_back(t);
    };
    for (size_t i = 0; i < pairs.size();) {
        size_t j = i + 1;
        while (j < pairs.size() && pairs[j].x == pairs[j - 1].x + 1 && pairs[j].y == pairs[j - 1].y + 1) {
            ++j;
        }
        if (j - i < (size_t)kGhostMinRun) {
            single.insert(single.end(), pairs.begin() + i, pairs.begin() + j);
        } else {
            for (size_t q = i; q < j; q += kGhostLong) task(q, std::min<size_t>(kGhostLong, j - q));
        }
        i = j;
    }
}

// The copies of a fill on the grid whose axes 0 and 1 are exchanged: node
// (i, j, k) of a grid with n1 nodes along axis 1 and row pitch `pitch` is
// node (j, i, k) of the transposed grid (n0 rows of pitch `xpitch`); the
// copies come back in destination order.  For a fill of copies (periodic and
// outflow faces) this is the same fill of the transposed grid.
template <class Int2>
std::vector<Int2> transposed_copies_of(const std::vector<Int2> &pairs, int pitch, int n0, int n1, int xpitch)
{
    auto tr = [&](int q) {
        const unsigned row = (unsigned)q / (unsigned)pitch, k = row / (unsigned)n1;
        const unsigned i = (unsigned)q - row * (unsigned)pitch, j = row - k * (unsigned)n1;
        return (int)((k * (unsigned)n0 + i) * (unsigned)xpitch + j);
    };
    // destination order by a table of the sources (a destination has one source)
    int end = 0;
    std::vector<Int2> xc(pairs.size());
    for (size_t q = 0; q < xc.size(); ++q) {
        xc[q].x = tr(pairs[q].x);
        xc[q].y = tr(pairs[q].y);
        end = std::max(end, xc[q].x + 1);
    }
    std::vector<int> source((size_t)end, 0);  // source + 1, 0: no copy
    for (const Int2 &c : xc) source[(size_t)c.x] = c.y + 1;
    size_t n = 0;
    for (int q = 0; q < end; ++q) {
        if (source[(size_t)q] == 0) continue;
        xc[n].x = q;
        xc[n].y = source[(size_t)q] - 1;
        ++n;
    }
    return xc;
}

// The sweeps (bit s) whose stages read node q = (k * n1 + j) * pitch + i outside
// the computed range [lo, hi): along s the stencil reaches `half` nodes beyond
// it; a viscous flux also reads one node across, beside the nodes from the one
// before the range to the one after it.
struct GhostReads {
    int pitch, n1;
    int lo[3], hi[3];
    int half;
    bool viscous;
    // the row of the node asked for last and the answer inside the range along x
    // (nodes are asked for in order: one pair of divisions a row)
    int first = 0, last = -1, inside = 0;
    bool in[3], beside[3], near[3];

    GhostReads(int pitch_, int n1_, const int *lo_, const int *hi_, int half_, bool viscous_)
        : pitch(pitch_), n1(n1_), half(half_), viscous(viscous_)
    {
        for (int t = 0; t < 3; ++t) {
            lo[t] = lo_[t];
            hi[t] = hi_[t];
        }
    }
    void set(int t, int c)
    {
        in[t] = c >= lo[t] && c < hi[t];
        beside[t] = c == lo[t] - 1 || c == hi[t];
        near[t] = c >= lo[t] - half && c < hi[t] + half;
    }
    int operator()(int q)
    {
        if (q < first || q > last) {
            const int row = q / pitch, k = row / n1;
            first = row * pitch;
            last = first + pitch - 1;
            set(1, row - k * n1);
            set(2, k);
            inside = mask_at(lo[0]);
        }
        const int c = q - first;
        return c >= lo[0] && c < hi[0] ? inside : mask_at(c);
    }
    int mask_at(int c)
    {
        set(0, c);
        int mask = 0;
        for (int s = 0; s < 3; ++s) {
            const int a = s == 0 ? 1 : 0, b = s == 2 ? 1 : 2;
            const bool across = viscous && (in[s] || beside[s]) && ((beside[a] && in[b]) || (in[a] && beside[b]));
            if ((near[s] && in[a] && in[b]) || across) mask |= 1 << s;
        }
        return mask;
    }
};

#ifdef __CUDACC__
inline void ghost_copy_tasks(const std::vector<int2> &pairs, std::vector<int4> &tasks, std::vector<int2> &single)
{
    ghost_copy_tasks_of<int2, int4>(pairs, tasks, single);
}
#endif
