// Race detector of the lane-interleaving host build (tests/test_lane_races.py).
//
// csrc/lanesim.cpp is compiled with -fsanitize=thread and linked with this file
// in place of the sanitizer's runtime, so every load and store of the decoder
// calls one of the __tsan_ functions below.  Accesses to the decoder slot, the
// memory that a group's lanes share, are recorded byte by byte from one
// __syncwarp barrier to the next.  A byte is raced on when the outcome depends
// on how the lanes' accesses interleave:
//
//   * a lane read it before writing it itself, and another lane wrote a value
//     other than the one it had at the last barrier;
//   * a lane read it after writing it itself, and it was written by another lane
//     too and held more than one value in between;
//   * two lanes wrote it and left different values.
//
// Lanes that write the same single value, or the same values that nobody reads
// before the barrier, are in order: the decoder's redundant stretches do so.
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

namespace {

enum { LANES = 32, REPORTS = 20 };

struct Cell {
    uint32_t epoch;
    uint32_t wrote, changed;         // lanes that wrote; that wrote something else than `old`
    uint32_t read_first, read_own;   // lanes that read before / after writing it themselves
    uint8_t old, value, several;     // at the barrier; first value written; more than one was
    uint8_t last[LANES];
    void *reader, *writer;
};

struct Race {
    unsigned char *base = nullptr;
    size_t size = 0;
    Cell *cells = nullptr;
    uint32_t *touched = nullptr;
    size_t ntouched = 0;
    uint32_t epoch = 1;
    int lane = 0;
    size_t wr_at = 0, wr_n = 0;      // a store that has been announced; its value is read at the lane's next event
    void *wr_pc = nullptr;
    unsigned long long races = 0;
};
__thread Race *t_race;

Cell &touch(Race *r, size_t i)
{
    Cell &c = r->cells[i];
    if (c.epoch != r->epoch) {
        memset(&c, 0, sizeof c);
        c.epoch = r->epoch;
        c.old = r->base[i];
        r->touched[r->ntouched++] = (uint32_t)i;
    }
    return c;
}

void settle(Race *r)
{
    const uint32_t me = 1u << r->lane;
    for (size_t i = r->wr_at; i < r->wr_at + r->wr_n; i++) {
        Cell &c = r->cells[i];
        const uint8_t v = r->base[i];
        if (!c.wrote) c.value = v;
        else if (v != c.value) c.several = 1;
        c.wrote |= me;
        if (v != c.old) {
            c.changed |= me;
            c.writer = r->wr_pc;
        }
        c.last[r->lane] = v;
    }
    r->wr_n = 0;
}

void access(const void *p, size_t n, int write, void *pc)
{
    Race *r = t_race;
    if (!r) return;
    settle(r);
    const size_t at = (size_t)((const unsigned char *)p - r->base);
    if (at >= r->size || n > r->size - at) return;
    for (size_t i = at; i < at + n; i++) {
        Cell &c = touch(r, i);
        if (write) continue;
        (c.wrote >> r->lane & 1 ? c.read_own : c.read_first) |= 1u << r->lane;
        c.reader = pc;
    }
    if (write) {
        r->wr_at = at;
        r->wr_n = n;
        r->wr_pc = pc;
    }
}

bool others(uint32_t a, uint32_t b)   // a lane of a and a different lane of b
{
    return a && b && !(a == b && !(a & (a - 1)));
}

} // namespace

extern "C" {

void lanerace_begin(void *base, size_t size)
{
    Race *r = new Race();
    r->base = (unsigned char *)base;
    r->size = size;
    r->cells = (Cell *)calloc(size, sizeof(Cell));
    r->touched = (uint32_t *)malloc(size * sizeof(uint32_t));
    if (!r->cells || !r->touched) abort();
    t_race = r;
}

void lanerace_lane(int id)
{
    if (!t_race) return;
    settle(t_race);
    t_race->lane = id;
}

// All lanes have reached a barrier.
void lanerace_barrier()
{
    Race *r = t_race;
    if (!r) return;
    settle(r);
    for (size_t k = 0; k < r->ntouched; k++) {
        const Cell &c = r->cells[r->touched[k]];
        if (!c.wrote) continue;
        int differ = 0, first = -1;
        for (int l = 0; l < LANES; l++)
            if (c.wrote >> l & 1) {
                if (first < 0) first = l;
                else differ |= c.last[l] != c.last[first];
            }
        if (others(c.read_first, c.changed) || (c.several && others(c.read_own, c.wrote)) || differ) {
            if (r->races++ < REPORTS)
                fprintf(stderr, "lane race at slot+%u: written %#x read %#x / %#x%s, reader %p writer %p\n",
                        r->touched[k], c.wrote, c.read_first, c.read_own, differ ? ", left different" : "", c.reader,
                        c.writer);
        }
    }
    r->ntouched = 0;
    r->epoch++;
}

unsigned long long lanerace_end()
{
    Race *r = t_race;
    t_race = nullptr;
    unsigned long long n = r->races;
    free(r->cells);
    free(r->touched);
    delete r;
    return n;
}

#define HOOKS(n)                                                                                    \
    void __tsan_read##n(void *p) { access(p, n, 0, __builtin_return_address(0)); }                  \
    void __tsan_write##n(void *p) { access(p, n, 1, __builtin_return_address(0)); }                 \
    void __tsan_unaligned_read##n(void *p) { access(p, n, 0, __builtin_return_address(0)); }        \
    void __tsan_unaligned_write##n(void *p) { access(p, n, 1, __builtin_return_address(0)); }
HOOKS(1) HOOKS(2) HOOKS(4) HOOKS(8) HOOKS(16)
void __tsan_read_range(void *p, long n) { access(p, (size_t)n, 0, __builtin_return_address(0)); }
void __tsan_write_range(void *p, long n) { access(p, (size_t)n, 1, __builtin_return_address(0)); }
void __tsan_init() {}
void __tsan_func_entry(void *) {}
void __tsan_func_exit() {}
void __tsan_vptr_update(void *, void *) {}
void __tsan_vptr_read(void *) {}

// memset and memcpy are not instrumented; the decoder's are announced here
void *lanerace_memset(void *d, int v, size_t n)
{
    access(d, n, 1, __builtin_return_address(0));
    return memset(d, v, n);
}
void *lanerace_memcpy(void *d, const void *s, size_t n)
{
    access(s, n, 0, __builtin_return_address(0));
    access(d, n, 1, __builtin_return_address(0));
    return memcpy(d, s, n);
}

}
