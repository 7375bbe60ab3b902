// The block tables that k_orbit_tables makes (csrc/chaos_perturb.cu, included here with its orbit code) against their
// definition evaluated on the host, at every index: (P, Q) of the 16- and 64-step blocks for both difference types and
// the exponent limits.  Arguments: centre x, centre y, bits, then iteration limits.  Prints "ok <limits set>" a limit.
#include <cstdarg>
#include <cstdio>
#include <cstdlib>

#include "../chaos-ultra_gb300/csrc/chaos_perturb.cu"

namespace chaos {
int api_fail(int code, const char *fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    std::vprintf(fmt, ap);
    va_end(ap);
    return code;
}
// (frames are not rendered here)
int api_device_counter(cudaStream_t, bool, WorkCounter *, int *) { return -1; }
void api_device_counter_done(const WorkCounter &) {}
int api_device_status(const WorkCounter &, cudaStream_t, uint32_t **) { return -1; }
bool api_budget(double, unsigned long long *) { return false; }
int api_read_status(const uint32_t *, cudaStream_t, double) { return -1; }
}  // namespace chaos

template <class T> static std::vector<T> fetch(const T *dev, size_t n)
{
    std::vector<T> v(n);
    if (cudaMemcpy(v.data(), dev, n * sizeof(T), cudaMemcpyDeviceToHost) != cudaSuccess) std::exit(3);
    return v;
}

struct Map {
    double px, py, qx, qy;
};

// The block of `length` steps from m, and its limit (LIN_NONE where it may not start); near: the limit's logarithm is
// within 1e-9 of a whole number.  bound_q: the majorant of |Q| (the same recurrence on moduli).
static int block(const std::vector<double2> &z, const std::vector<char> &ev, uint32_t m, uint32_t length, double slack,
                 Map &map, double &bound_q, bool &near)
{
    const uint32_t last = (uint32_t)z.size() - 1u;
    near = false;
    auto zz = [&](uint32_t j) { return z[j].x * z[j].x + z[j].y * z[j].y; };
    if (!(m + length < last) || !(zz(m) > 0.0)) return LIN_NONE;
    double px = 1, py = 0, qx = 0, qy = 0, rho = INFINITY, norm = 0;
    bound_q = 0;
    for (uint32_t j = m;; j++) {
        if (j > m && ev[j]) return LIN_NONE;
        norm = 2.0 * (px * px + py * py + qx * qx + qy * qy);
        rho = std::min(rho, zz(j) / norm);
        if (j == m + length) break;
        const double ax = 2.0 * z[j].x, ay = 2.0 * z[j].y;
        const double npx = ax * px - ay * py, npy = ax * py + ay * px;
        const double nqx = ax * qx - ay * qy + 1.0, nqy = ax * qy + ay * qx;
        px = npx, py = npy, qx = nqx, qy = nqy;
        bound_q = std::hypot(ax, ay) * bound_q + 1.0;
    }
    map = Map{px, py, qx, qy};
    if (length == 64u && !(norm <= 0x1p200)) return LIN_NONE;
    if (!(rho > 0.0) || !std::isfinite(rho)) return LIN_NONE;
    const double l = 0.5 * std::log2(rho) - slack, f = std::floor(l);
    near = std::fabs(l - std::round(l)) < 1e-9;
    return f < -127.0 ? (int)LIN_NONE : (int)std::min(127.0, f);
}

static long check(const std::vector<double2> &z, const std::vector<char> &ev, double slack, const std::vector<Map> &b16,
                  const std::vector<Map> &b64, const std::vector<char2> &lim, double stored)
{
    long set = 0;
    for (uint32_t m = 0; m < z.size(); m++)
        for (uint32_t length = 16; length <= 64; length += 48) {
            Map want{};
            double bound_q = 0;
            bool near;
            const int l = block(z, ev, m, length, slack, want, bound_q, near);
            const int have = length == 16 ? lim[m].x : lim[m].y;
            const bool off_by_one = near && l != LIN_NONE && have != LIN_NONE && std::abs(l - have) == 1;
            if (have != l && !off_by_one) return std::printf("limit %d, not %d, at %u + %u\n", have, l, m, length), -1;
            if (have == LIN_NONE) continue;
            set++;
            // `length` complex products (and sums) of at most eight roundings each, then the table's own
            const Map &got = length == 16 ? b16[m] : b64[m];
            const double u = 8.0 * length * 0x1p-53, p = std::hypot(want.px, want.py), q = std::hypot(want.qx, want.qy);
            if (!(std::hypot(got.px - want.px, got.py - want.py) <= u * p + stored * p) ||
                !(std::hypot(got.qx - want.qx, got.qy - want.qy) <= u * bound_q + stored * q))
                return std::printf("block at %u + %u\n", m, length), -1;
        }
    return set;
}

int main(int argc, char **argv)
{
    for (int a = 4; a < argc; a++) {
        chaos_orbit *o = nullptr;
        if (chaos_orbit_create(argv[1], argv[2], (uint32_t)std::atoi(argv[3]), (uint32_t)std::atoi(argv[a]), &o)) return 2;
        const size_t n = o->last + 1u;
        const std::vector<double2> z = fetch(o->z64, n);
        std::vector<double2> z32(n);
        std::vector<char> ev(n), ev32(n);
        const std::vector<float2> f = fetch(o->z32, n), f2 = fetch(o->z2, n);
        for (size_t j = 0; j < n; j++) {
            if (f[j].x != (float)z[j].x || f[j].y != (float)z[j].y || f2[j].x != 2.f * f[j].x || f2[j].y != 2.f * f[j].y)
                return std::printf("binary32 orbit at %zu\n", j), 1;
            z32[j] = make_double2(f[j].x, f[j].y);
            const double r2 = std::fma(z[j].x, z[j].x, z[j].y * z[j].y);
            const float r2f = std::fmaf(f[j].x, f[j].x, f[j].y * f[j].y);
            ev[j] = !(r2 < 3.99) || r2 < 0x1p-98;
            ev32[j] = !(r2f < 3.99f) || r2f < 0x1p-98f;
        }
        std::vector<Map> b16(n), b64(n);
        const std::vector<float4> s16 = fetch(o->bla16, n), s64 = fetch(o->bla64, n);
        for (size_t j = 0; j < n; j++) {
            b16[j] = Map{s16[j].x, s16[j].y, s16[j].z, s16[j].w};
            b64[j] = Map{s64[j].x, s64[j].y, s64[j].z, s64[j].w};
        }
        const long set32 = check(z32, ev32, 25.5, b16, b64, fetch(o->lin_lim, n), 0x1p-23);
        const std::vector<double2> d16 = fetch(o->bla16d, 2 * n), d64 = fetch(o->bla64d, 2 * n);
        for (size_t j = 0; j < n; j++) {
            b16[j] = Map{d16[2 * j].x, d16[2 * j].y, d16[2 * j + 1].x, d16[2 * j + 1].y};
            b64[j] = Map{d64[2 * j].x, d64[2 * j].y, d64[2 * j + 1].x, d64[2 * j + 1].y};
        }
        const long set64 = check(z, ev, 54.5, b16, b64, fetch(o->lin_limd, n), 0.0);
        if (set32 < 0 || set64 < 0) return 1;
        std::printf("ok %ld %ld\n", set32, set64);
        chaos_orbit_destroy(o);
    }
    return 0;
}
