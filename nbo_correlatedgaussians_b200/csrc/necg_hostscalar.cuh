// necg_hostscalar.cuh -- a value-carrying FP64 scalar that also counts the
// operations applied to it, and host accessors for bra/ket records.  Used to
// instantiate the term templates of necg_math.cuh on the host: by the FLOP
// counter (necg_count.cu) and by the test emulator of the kernels.
#pragma once
#include <math.h>
#include <stddef.h>

#include "necg_math.cuh"

namespace necg {

struct CountCtx {
    long long flops = 0, special = 0;
};
inline CountCtx &count_ctx() {
    static thread_local CountCtx c;
    return c;
}

// (Host and device for the templates' sake, which are: only the host runs them.)
struct CD {
    double v;
    NECG_HD CD() : v(0.0) {}
    NECG_HD CD(double x) : v(x) {}
    NECG_HD CD &operator+=(const CD &o) { v += o.v; return flop(); }
    NECG_HD CD &operator-=(const CD &o) { v -= o.v; return flop(); }
    NECG_HD CD &operator*=(const CD &o) { v *= o.v; return flop(); }
#pragma nv_exec_check_disable
    NECG_HD CD &flop() { ++count_ctx().flops; return *this; }
#pragma nv_exec_check_disable
    NECG_HD CD &spec() { ++count_ctx().special; return *this; }
};
NECG_HD CD operator+(CD a, CD b) { return CD(a.v + b.v).flop(); }
NECG_HD CD operator-(CD a, CD b) { return CD(a.v - b.v).flop(); }
NECG_HD CD operator*(CD a, CD b) { return CD(a.v * b.v).flop(); }
NECG_HD CD operator/(CD a, CD b) { return CD(a.v / b.v).spec(); }
NECG_HD CD operator+(double a, CD b) { return CD(a) + b; }
NECG_HD CD operator+(CD a, double b) { return a + CD(b); }
NECG_HD CD operator-(double a, CD b) { return CD(a) - b; }
NECG_HD CD operator-(CD a, double b) { return a - CD(b); }
NECG_HD CD operator*(double a, CD b) { return CD(a) * b; }
NECG_HD CD operator*(CD a, double b) { return a * CD(b); }
NECG_HD CD operator-(CD a) { return CD(-a.v); }
NECG_HD bool operator>(CD a, double b) { return a.v > b; }
NECG_HD bool operator<=(CD a, double b) { return a.v <= b; }
NECG_HD bool operator<=(CD a, CD b) { return a.v <= b.v; }
NECG_HD CD rsq(CD a) { return CD(1.0 / ::sqrt(a.v)).spec(); }
NECG_HD CD rcp(CD a) { return CD(1.0) / a; }
NECG_HD CD exp(CD a) { return CD(::exp(a.v)).spec(); }
NECG_HD double val(CD x) { return x.v; }

// bra record field f of basis k in a structure-of-arrays buffer
struct HostBra {
    const double *p;  // bra + k
    size_t K;
    NECG_HD CD operator()(int f) const { return CD(p[(size_t)f * K]); }
};
struct HostKet {
    const double *p;
    NECG_HD CD operator[](int i) const { return CD(p[i]); }
};
struct HostKetBase {
    const double *p;
    NECG_HD HostKet at(size_t off) const { return HostKet{p + off}; }
};

}  // namespace necg
