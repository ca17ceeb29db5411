// Applies the autotuners' rules (boids_engine.h) to times read from stdin:
// kTuneCount set times, the best set's time with the choice of kernels, and
// whether the flock has that choice.  Prints "set split" per line.
#include "boids_engine.h"

#include <cstdio>

int main()
{
    float ms[boidsgpu::kTuneCount], choice;
    int routed;
    for (;;) {
        for (float &m : ms)
            if (std::scanf("%f", &m) != 1) return 0;
        if (std::scanf("%f %d", &choice, &routed) != 2) return 1;
        const int c = boidsgpu::tune_choice(ms, routed != 0);
        std::printf("%d %d\n", c, c > 0 && boidsgpu::tune_splits(ms[c], routed ? choice : INFINITY));
    }
}
