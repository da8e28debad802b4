// Checks on the CPU that the hand-over of the 2D strips (pfast_gb300/csrc/strip_sync.h) orders every
// lane's accesses before it in one warp ahead of every lane's accesses behind it in another, directly
// and through a chain of warps.  Its functions run over vector clocks: a fence acquires what the
// lane's loads have read and releases what the lane has seen, a barrier joins the lanes of a warp; a
// broadcast orders nothing.  Prints "ok <name>" or "FAIL <name>".
#include <algorithm>
#include <cstdio>
#include <map>
#include <vector>

#include "strip_sync.h"

using namespace pfast;

static const int kLanes = 8, kWarps = 4, kN = kLanes * kWarps;
typedef std::vector<unsigned> Clock;
static void join(Clock& a, const Clock& b) { for (int i = 0; i < kN; ++i) a[i] = std::max(a[i], b[i]); }

struct Machine {
    std::map<const volatile int*, Clock> word;
    std::vector<Clock> seen, released, read;
    Machine() : seen(kN, Clock(kN, 0)), released(seen), read(seen) {}
};

struct Warp {   // a whole warp; lane 0 leads
    Machine* m;
    int l0;
    bool leader() const { return true; }
    void barrier() const {
        Clock c(kN, 0);
        for (int l = 0; l < kLanes; ++l) join(c, m->seen[l0 + l]);
        for (int l = 0; l < kLanes; ++l) m->seen[l0 + l] = c;
    }
    void fence() const { join(m->seen[l0], m->read[l0]); m->released[l0] = m->seen[l0]; }
    void store(volatile int* p, int v) const { *p = v; m->word[p] = m->released[l0]; }
    int poll(volatile int* p, int want) const {
        if (m->word.count(p)) join(m->read[l0], m->word[p]);
        return *p >= want;
    }
    int broadcast(int v) const { return v; }
    void access() const { for (int l = 0; l < kLanes; ++l) ++m->seen[l0 + l][l0 + l]; }   // every lane
    bool sees(const Warp& o) const {
        for (int l = 0; l < kLanes; ++l)
            for (int k = 0; k < kLanes; ++k)
                if (m->seen[l0 + l][o.l0 + k] < m->seen[o.l0 + k][o.l0 + k]) return false;
        return true;
    }
};

static int bad = 0;
static void check(bool ok, const char* name) { std::printf("%s %s\n", ok ? "ok" : "FAIL", name); bad += !ok; }

int main() {
    Machine m;
    const Warp a{&m, 0}, b{&m, kLanes}, c{&m, 2 * kLanes};
    int ab = 0, bc = 0, ca = 0;
    a.access();
    strip_publish(a, &ab, 1);
    check(strip_wait(b, &ab, 1) && b.sees(a), "stores of a strip ahead of the loads of the next");
    b.access();
    strip_publish(b, &bc, 1);
    check(strip_wait(c, &bc, 1) && c.sees(b) && c.sees(a), "through a strip between them");
    c.access();
    strip_publish(c, &ca, 1);
    check(strip_wait(a, &ca, 1) && a.sees(b) && a.sees(c), "loads ahead of the stores of the next order");
    check(!strip_wait(a, &ca, 2), "given up");
    return bad ? 1 : 0;
}
