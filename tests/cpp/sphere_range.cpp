// Host check of the sphere test's early answer (beyondRange in
// albedo_b200/csrc/kernels/traverse.cuh): whenever it says that a sphere seen
// from outside has no root in (tmin, tmax), the whole test, restated here in
// host arithmetic (built with -ffp-contract=off, as the device's _rn
// operations round), finds none.
//
// Arguments: "float" or "double". Prints one line per category: tests, early
// answers, hits of the whole test, and early answers it contradicts.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>

namespace {

template <typename T>
T dot3(const T* a, const T* b)
{
    return (a[0] * b[0] + a[1] * b[1]) + a[2] * b[2];
}

template <typename T>
bool beyondRange(T a, T h, T c, T oc2, T tmin, T tmax)
{
    if (h > T(0)) {
        return tmin >= T(0);
    }
    return h * h >= T(0.01) * (a * oc2) && c > (T(-2.01) * h) * tmax;
}

// sphereRoot without the early answer; `far_only` is its kSphereFarOnly mode.
template <typename T>
bool wholeTest(const T* o, const T* d, const T* center, T radius, T tmin, T tmax, bool far_only, bool& early)
{
    T oc[3];
    for (int i = 0; i < 3; ++i) {
        oc[i] = o[i] - center[i];
    }
    const T a = dot3(d, d);
    const T h = dot3(d, oc);
    const T r2 = radius * radius;
    const T oc2 = dot3(oc, oc);
    const T c = oc2 - r2;
    early = c > T(0) && beyondRange(a, h, c, oc2, tmin, tmax);
    const T k = h / a;
    T l[3];
    for (int i = 0; i < 3; ++i) {
        l[i] = oc[i] - d[i] * k;
    }
    const T disc = a * (r2 - dot3(l, l));
    if (disc < T(0)) {
        return false;
    }
    const T q = -(h + std::copysign(std::sqrt(disc), h));
    T near_root = T(0);
    T far_root = T(0);
    if (q != T(0)) {
        near_root = q / a;
        far_root = c / q;
        if (near_root > far_root) {
            std::swap(near_root, far_root);
        }
    }
    const auto inside = [&](T t) { return tmin < t && t < tmax; };
    return (!far_only && inside(near_root)) || inside(far_root);
}

template <typename T>
void check()
{
    std::mt19937_64 rng(7);
    std::uniform_real_distribution<double> unit(0.0, 1.0);
    std::normal_distribution<double> normal;
    const char* categories[] = {"room", "small", "grazing", "touching", "scaled"};
    for (const char* category : categories) {
        long tests = 0;
        long answered = 0;
        long hits = 0;
        long wrong = 0;
        const bool room = std::strcmp(category, "room") == 0;
        for (int i = 0; i < 1'000'000; ++i) {
            const double radius = room ? 1e4 : std::pow(10.0, -3.0 + 4.0 * unit(rng));
            double u[3];
            double d[3];
            double nu = 0.0;
            double nd = 0.0;
            for (int k = 0; k < 3; ++k) {
                u[k] = normal(rng);
                d[k] = normal(rng);
                nu += u[k] * u[k];
                nd += d[k] * d[k];
            }
            // Origins from on the surface (a few ulps either side) to far away.
            double height = radius * std::pow(10.0, -7.0 + 9.0 * unit(rng));
            if (room) {
                height = std::pow(10.0, -4.0 + 5.0 * unit(rng));
            } else if (std::strcmp(category, "touching") == 0) {
                height = radius * 1e-7 * (unit(rng) - 0.5);
            }
            const double scale = std::strcmp(category, "scaled") == 0 ? std::pow(10.0, -3.0 + 6.0 * unit(rng)) : 1.0;
            if (std::strcmp(category, "grazing") == 0) {
                // Aimed at the sphere's rim.
                double along = 0.0;
                for (int k = 0; k < 3; ++k) {
                    along += d[k] * u[k] / std::sqrt(nu);
                }
                nd = 0.0;
                const double distance = radius + height;
                double side = 0.0;
                for (int k = 0; k < 3; ++k) {
                    d[k] -= along * u[k] / std::sqrt(nu);
                    side += d[k] * d[k];
                }
                const double rim = radius * (1.0 + 1e-5 * (unit(rng) - 0.5));
                for (int k = 0; k < 3; ++k) {
                    d[k] = d[k] / std::sqrt(side) * rim - u[k] / std::sqrt(nu) * distance;
                    nd += d[k] * d[k];
                }
            }
            T o[3];
            T dir[3];
            T center[3];
            for (int k = 0; k < 3; ++k) {
                const double c = room ? (k == 0 ? -10003.0 : 0.0) : 4.0 * (unit(rng) - 0.5);
                center[k] = static_cast<T>(static_cast<float>(c));
                o[k] = static_cast<T>(static_cast<float>(c + u[k] / std::sqrt(nu) * (radius + height)));
                dir[k] = static_cast<T>(static_cast<float>(d[k] / std::sqrt(nd) * scale));
            }
            const T tmins[] = {T(0), T(0), T(0), static_cast<T>(unit(rng) - 0.5)};
            const T tmax = unit(rng) < 0.3 ? std::numeric_limits<T>::infinity()
                                           : static_cast<T>(static_cast<float>((height + radius * unit(rng)) *
                                                                               std::pow(10.0, 2.0 * unit(rng) - 1.0)));
            bool early = false;
            const bool hit = wholeTest<T>(o, dir, center, static_cast<T>(static_cast<float>(radius)), tmins[i & 3],
                                          tmax, (i & 16) != 0, early);
            ++tests;
            answered += early ? 1 : 0;
            hits += hit ? 1 : 0;
            wrong += early && hit ? 1 : 0;
        }
        std::printf("%s tests=%ld early=%ld hits=%ld wrong=%ld\n", category, tests, answered, hits, wrong);
    }
}

} // namespace

int main(int argc, char** argv)
{
    if (argc > 1 && std::strcmp(argv[1], "double") == 0) {
        check<double>();
    } else {
        check<float>();
    }
    return 0;
}
