// Prints the pairs a boid from which and up to which a flock goes a warp per
// boid (boids_engine.h): reads "even seen n kind" lines (kind: 0 a handle, 1 the
// allocation-free step, 2 an ensemble), writes "line top".
#include "boids_engine.h"

#include <cstdio>

int main()
{
    double even, seen, n;
    int kind;
    while (std::scanf("%lf %lf %lf %d", &even, &seen, &n, &kind) == 4)
        std::printf("%.9g %.9g\n", boidsgpu::crowd_line(even, n, (boidsgpu::CrowdKind)kind), boidsgpu::crowd_top(even, seen, n, (boidsgpu::CrowdKind)kind));
}
