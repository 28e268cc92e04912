// Drives the step control (csrc/common.cuh: ctl_begin, ctl_end, ctl_begin_t0) on
// the host. Compiled and run by test_control.py; prints "ok" or the first rule
// that does not hold.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include <cuda_runtime.h>

// the device functions that the header's inline functions name
static double __dmul_rn(double a, double b) { return a * b; }
static double __dadd_rn(double a, double b) { return a + b; }
static float __fmul_rn(float a, float b) { return a * b; }
static float __fsub_rn(float a, float b) { return a - b; }
static double __longlong_as_double(long long v) {
    double d;
    std::memcpy(&d, &v, sizeof d);
    return d;
}
static unsigned long long atomicMax(unsigned long long* a, unsigned long long v) {
    const unsigned long long o = *a;
    if (v > o) *a = v;
    return o;
}

#include "common.cuh"

#define CHECK(c)                                         \
    do {                                                 \
        if (!(c)) {                                      \
            std::printf("line %d: %s\n", __LINE__, #c);  \
            std::exit(1);                                \
        }                                                \
    } while (0)

using namespace slab;

static uint64_t bits(double v) {
    uint64_t b;
    std::memcpy(&b, &v, sizeof b);
    return b;
}

static constexpr int NX = 64, NY = 48;

static void box_to(Ctl& c, double x0, double x1, double y0, double y1) {
    const double b[4] = {x0, x1, y0, y1};
    for (int k = 0; k < 4; ++k) c.pos_acc[k] = bits(b[k]);
}
static bool box_is(const Ctl& c, int i0, int i1, int j0, int j1) {
    return c.box[0] == i0 && c.box[1] == i1 && c.box[2] == j0 && c.box[3] == j1;
}
// an advance call's start, as the two paths' control kernels make it
static void arm(Ctl& c, int64_t steps) {
    c.stop = 0;
    c.frame_hit = 0;
    c.steps_left = steps;
    c.stop_at_frame = 0;
    ctl_begin(&c, NX, NY);
}

int main() {
    Ctl c;
    std::memset(&c, 0, sizeof c);
    c.dx = 1.0;
    c.one_over_dx = 1.0;
    c.C_cfl = 0.5;
    c.dt_max = 0.01;
    c.output_dt = 1.0;
    c.total_time = 10.0;
    c.stop = 1;
    box_to(c, 10.5, 20.5, 8.5, 30.5);

    // the t = 0 pass leaves the box for the first step
    ctl_begin_t0(&c, NX, NY);
    CHECK(c.active && box_is(c, 9, 22, 7, 32));
    arm(c, 5);
    CHECK(c.active && box_is(c, 9, 22, 7, 32));

    // begun, not run, and begun again: the same step
    const double dt = c.dt, t1 = c.new_time;
    arm(c, 5);
    CHECK(c.active && !c.err && box_is(c, 9, 22, 7, 32) && c.dt == dt && c.new_time == t1);
    ctl_begin_t0(&c, NX, NY);
    CHECK(c.active && !c.err && box_is(c, 9, 22, 7, 32));
    arm(c, 2);

    // a step that runs moves the box
    box_to(c, 11.5, 21.5, 9.5, 31.5);
    c.vmax2_acc = bits(4.0);
    ctl_end(&c);
    ctl_begin(&c, NX, NY);
    CHECK(c.active && c.steps == 1 && box_is(c, 10, 23, 8, 33));
    box_to(c, 12.5, 22.5, 10.5, 32.5);
    ctl_end(&c);
    ctl_begin(&c, NX, NY);
    CHECK(!c.active && c.stop && c.steps == 2 && box_is(c, 10, 23, 8, 33));  // the budget: the box of the last step stays
    arm(c, 1);
    CHECK(c.active && box_is(c, 11, 24, 9, 34));

    // a box outside the terrain stops the run, and the grid keeps the box of its last step
    box_to(c, 12.5, 63.5, 10.5, 32.5);
    ctl_end(&c);
    arm(c, 1);
    CHECK(!c.active && c.stop && (c.err & ERR_DOMAIN));
    CHECK(box_is(c, 11, 24, 9, 34));
    ctl_begin_t0(&c, NX, NY);
    CHECK(!c.active && box_is(c, 11, 24, 9, 34));
    std::printf("ok\n");
    return 0;
}
