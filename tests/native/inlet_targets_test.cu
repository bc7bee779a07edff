// The absorbing layers' targets formed on the host against the same sums and
// products rounded one by one (the device's form); prints the number of values
// that differ, for binary32 and binary64.
#include <cstdio>
#include <cstring>
#include <random>

#include "kernels3d.cuh"

template <class A> A once(A a) {
    volatile A kept = a;   // a rounded value, which no later operation is contracted with
    return kept;
}

template <class A> A target(int i, const A* u) {
    namespace d3 = orr::d3;
    const A cu = once(once(once(A(d3::cx(i)) * u[0]) + once(A(d3::cy(i)) * u[1])) + once(A(d3::cz(i)) * u[2]));
    const A uu = once(once(once(u[0] * u[0]) + once(u[1] * u[1])) + once(u[2] * u[2]));
    const A square = once(once(A(4.5) * cu) * cu), speed = once(A(1.5) * uu);
    const A w = static_cast<A>(d3::w(i));
    if (sizeof(A) == 4) {
        return once(w * once(once(once(A(3) * cu) + square) - speed));
    }
    return once(w * once(once(once(A(1) + once(A(3) * cu)) + square) - speed));
}

template <class A> int differing() {
    std::mt19937_64 random(11);
    std::uniform_real_distribution<double> speed(-0.12, 0.12);
    int count = 0;
    for (int k = 0; k < 500; ++k) {
        const double v[3] = {speed(random), speed(random), speed(random)};
        A values[orr::kInletValues];
        orr::fill_inlet(values, v);
        for (int i = 0; i < orr::d3::Q; ++i) {
            const A want = target<A>(i, values);
            count += std::memcmp(&want, &values[orr::kInletTargets + i], sizeof(A)) != 0;
        }
    }
    return count;
}

int main() { std::printf("%d %d\n", differing<float>(), differing<double>()); }
