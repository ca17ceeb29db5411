// Prints the all-pairs product filter's constants as the engine derives them:
// reads "radius field" lines, writes "filter_radius turn min pass pad" in full
// precision (pad: the half-precision word).
#include "boids_engine.h"

#include <cstdio>

int main()
{
    double radius, field;
    while (std::scanf("%lf %lf", &radius, &field) == 2) {
        const double rf = boidsgpu::filter_radius(boidsgpu::f_up(radius), (float)field);
        const boidsgpu::ApFilter f = boidsgpu::ap_filter(rf, field);
        std::printf("%.17g %.9g %.9g %.9g %u\n", rf, f.turn, f.min, boidsgpu::kApPass, boidsgpu::kApPad);
    }
}
