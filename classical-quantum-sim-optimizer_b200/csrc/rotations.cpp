// Host planner of Pauli-rotation passes: gates -> relabellings, phases and
// rotations -> phases of four register directions.
#include "rotations.hpp"

#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>

namespace dq {

namespace {

constexpr long double kPiL = 3.14159265358979323846264338327950288L;
// Angles and moduli are kept with 64-bit mantissas: what the gates' entries say
// is then lost only where a factor is rounded for the kernel.
using ld = long double;
// Most an entry may differ from the unitary matrix (times a scale) that the
// rotations apply in its place: the rounding of the entries and of products of
// matrices (largest of 10^6 U3 2.1e-16, of products of twelve 8.1e-16, of forty 1.3e-15).
// Others, such as a U3 of an angle of 1e5, whose sums of angles are rounded to
// 1e-11, run in register phases, which apply the entries as they are.
constexpr ld kUnitaryTol = 2e-15L;
constexpr ld kScaleTol = 1e-12L;  // a scale further from one is no rounding
// No turn, or a quarter turn, to the rounding of the product of matrices that gives it.
constexpr ld kAngleTol = 1.2e-16L;
constexpr ld kExactTol = 1e-18L;  // the same, to the rounding of the numbers here
constexpr int kMaxDiagQubits = 6;

int parity64(uint64_t x) { return __builtin_parityll(x); }
int parity(uint32_t x) { return __builtin_parity(x); }  // (of directions and what lies on them: tile bits)

struct Item {
    bool rot = false;
    bool imag = false;   // rotation without the factor i (mu & v even)
    uint32_t v = 0;      // rotation: direction (tile-local place bits)
    uint64_t mask = 0;   // parity mask over place bits (tile-local below m, tile index above)
    double t = 0.0;      // rotation: signed tangent
    ld a = 0.0;          // phase: angle
    ld b = 0.0;          // phase: logarithm of its modulus (factors e^(+-(b + ia)))
};

struct Unsupported {};

struct Complex {
    ld re, im;
    Complex(ld r = 0.0L, ld i = 0.0L) : re(r), im(i) {}
    Complex(cplx z) : re(z.re), im(z.im) {}
    Complex conj() const { return {re, -im}; }
    Complex operator*(ld g) const { return {re * g, im * g}; }
};
Complex operator*(Complex x, Complex y) { return {x.re * y.re - x.im * y.im, x.re * y.im + x.im * y.re}; }
Complex operator+(Complex x, Complex y) { return {x.re + y.re, x.im + y.im}; }
Complex operator-(Complex x, Complex y) { return {x.re - y.re, x.im - y.im}; }

ld arg(Complex z) {
    if (z.im == 0.0L) return z.re < 0 ? kPiL : 0.0L;
    return std::atan2(z.im, z.re);
}
ld norm2(Complex z) { return z.re * z.re + z.im * z.im; }

// The unitary matrix [[x, y], [z, w]] nearest to a one-qubit matrix, times e^scale.
// With the arguments of one entry each, 20 layers of U3 brickwork on 12 qubits were 2.2e-15
// off the product of the entries, from the nearest matrix 1.1e-15; without the
// scale 2,400 H gates 1.7e-13.
struct Polar {
    Complex x, y, z, w;
    ld c, s;  // moduli of x and z
    ld scale;
};

// False where the entries are not those of a unitary matrix to their rounding.
bool polar(const Mat2& u, Polar& p) {
    const Complex a = u[0][0], b = u[0][1], c = u[1][0], d = u[1][1];
    // The polar factor of a 2x2 matrix u is u + (det u / |det u|) adj(u)^H, up to a scale.
    const Complex det = a * d - b * c;
    const ld size = std::sqrt(norm2(det));
    if (!(std::fabs(size - 1.0L) <= 2 * kScaleTol)) return false;
    const Complex f = det.im == 0.0L ? Complex(det.re < 0 ? -1.0L : 1.0L, 0.0L) : det * (1.0L / size);
    p.x = a + f * d.conj();
    p.y = b - f * c.conj();
    p.z = c - f * b.conj();
    p.w = d + f * a.conj();
    const ld x2 = norm2(p.x), z2 = norm2(p.z), r = std::sqrt(x2 + z2);
    p.c = std::sqrt(x2) / r;
    p.s = std::sqrt(z2) / r;
    p.scale = 0.5L * (size - 1.0L);  // (its logarithm: the square is below 1e-24)
    const ld g = (1.0L + p.scale) / r;
    const Complex off[4] = {a - p.x * g, b - p.y * g, c - p.z * g, d - p.w * g};
    for (const Complex& e : off)
        if (!(norm2(e) <= kUnitaryTol * kUnitaryTol)) return false;
    return true;
}

// The mean logarithm of a diagonal's moduli; false where one differs from it by
// more than rounding.
bool mean_modulus(const std::vector<cplx>& values, ld& mean) {
    mean = 0.0L;
    for (cplx d : values) mean += 0.5L * (norm2(d) - 1.0L);  // (each its logarithm, as above)
    mean /= ld(values.size());
    if (!(std::fabs(mean) <= kScaleTol)) return false;
    for (cplx d : values)
        if (!(std::fabs(0.5L * (norm2(d) - 1.0L) - mean) <= kUnitaryTol)) return false;
    return true;
}

// x + a, kept below a turn: a sum of 1,000 angles would lose 2e-14 to its own size.
void turn(ld& x, ld a) {
    x += a;
    if (std::fabs(x) > kPiL) x = std::remainder(x, 2 * kPiL);
}

// The gates of a pass as items, with the frame that relabels places.
class Lowering {
  public:
    Lowering(const std::vector<int>& tile, int n) : m_(int(tile.size())) {
        mask_.resize(size_t(n));
        cons_.assign(size_t(n), 0);
        dir_.assign(size_t(n), 0);
        int outer = 0;
        for (int q = 0, l = 0; q < n; q++) {
            if (l < m_ && tile[size_t(l)] == q) {
                mask_[size_t(q)] = uint64_t(1) << l;
                dir_[size_t(q)] = 1u << l;
                l++;
            } else {
                mask_[size_t(q)] = uint64_t(1) << (m_ + outer++);
            }
        }
    }

    void add(const Operation& op) {
        switch (op.type) {
            case Operation::One: one(op.target, op.m, op.controls); break;
            case Operation::X: x(op.target, op.controls); break;
            case Operation::Swap: swap(op.a, op.b, op.controls); break;
            case Operation::Diagonal: diagonal(op); break;
            case Operation::Dense: dense(op); break;
            default: throw Unsupported{};
        }
    }

    std::vector<Item> items;
    ld global = 0.0;           // phase of the whole state
    ld norm = 0.0;             // logarithm of a modulus of the whole state
    uint64_t sign = 0;         // Z^sign still to be applied

    const std::vector<uint64_t>& masks() const { return mask_; }
    const std::vector<int>& consts() const { return cons_; }
    const std::vector<uint32_t>& dirs() const { return dir_; }

  private:
    int m_;
    std::vector<uint64_t> mask_;
    std::vector<int> cons_;
    std::vector<uint32_t> dir_;
    struct Open {
        uint64_t mask;
        size_t item;
    };
    std::vector<Open> open_;  // phases that every later rotation commutes with

    // exp(i a Z^mask (-1)^cons); `tol`: what an angle may be off a multiple of pi/2 and count as one.
    void phase(uint64_t mask, int cons, ld a, ld tol = kExactTol) {
        if (cons) a = -a;
        if (mask == 0) {
            turn(global, a);
            return;
        }
        if (std::fabs(a) > kPiL / 2) {
            const ld r = std::nearbyint(a / kPiL);
            a -= r * kPiL;
            if (std::fmod(r, 2.0L) != 0.0L) turn(global, kPiL);
        }
        if (std::fabs(a) <= tol) return;
        if (std::fabs(std::fabs(a) - kPiL / 2) <= tol) {  // +-i Z^mask
            turn(global, a > 0 ? kPiL / 2 : -kPiL / 2);
            sign ^= mask;
            return;
        }
        for (const Open& o : open_)
            if (o.mask == mask) {
                turn(items[o.item].a, a);
                return;
            }
        Item it;
        it.mask = mask;
        it.a = a;
        open_.push_back({mask, items.size()});
        items.push_back(it);
    }

    // exp(-i theta/2 P) with (c, s) = (cos, sin)(theta/2), P the product over the
    // qubits of X (bit of xs), Z (of zs) or Y (both).
    void rotation(std::initializer_list<uint64_t> xs, std::initializer_list<uint64_t> zs, ld c, ld s) {
        rotation_of<std::initializer_list<uint64_t>>(xs, zs, c, s);
    }
    template <class Qubits>
    void rotation_of(const Qubits& xs, const Qubits& zs, ld c, ld s) {
        uint32_t v = 0;
        uint64_t mask = 0;
        int cons = 0, ny = 0;
        for (uint64_t q : xs) {
            if (dir_[size_t(q)] == 0) throw Unsupported{};  // a rotated qubit outside the tile
            v ^= dir_[size_t(q)];
        }
        for (uint64_t q : zs) {
            mask ^= mask_[size_t(q)];
            cons ^= cons_[size_t(q)];
            if (std::find(xs.begin(), xs.end(), q) != xs.end()) ny++;
        }
        const bool imag = ny % 2 == 0;
        if ((ny / 2) % 2) cons ^= 1;  // i^ny = +-1 or +-i
        if (c < 0) {
            turn(global, kPiL);
            c = -c;
            s = -s;
        }
        if (s == 0.0) return;
        if (cons) s = -s;  // from here P = (i) X^v Z^mask
        if (std::fabs(s) > c) {
            // c - i s P = (-i P) (s + i c P): rotate by the complement, then apply P
            // (the phases and rotations before see the place, so P comes last).
            ld c2 = s, s2 = -c;
            if (c2 < 0) {
                turn(global, kPiL);
                c2 = -c2;
                s2 = -s2;
            }
            if (s2 != 0.0) emit(v, mask, imag, c2, s2);
            if (imag) turn(global, -(kPiL / 2));
            sign ^= mask;
            for (size_t q = 0; q < mask_.size(); q++) cons_[q] ^= parity64(mask_[q] & v);
            return;
        }
        emit(v, mask, imag, c, s);
    }

    void emit(uint32_t v, uint64_t mask, bool imag, ld c, ld s) {
        Item it;
        it.rot = true;
        it.imag = imag;
        it.v = v;
        it.mask = mask;
        it.t = double(s / c);
        norm += 0.5L * (c * c + s * s - 1.0L);  // (an RXX's entries as they are rounded)
        if (parity64(sign & v)) it.t = -it.t;
        open_.erase(std::remove_if(open_.begin(), open_.end(),
                                   [&](const Open& o) { return parity(uint32_t(o.mask) & v) != 0; }),
                    open_.end());
        items.push_back(it);
    }

    // Phases phi[j] by the qubits' values (qubits[0] the MSB of j).
    void phases(const std::vector<uint64_t>& qubits, std::vector<ld> phi) {
        const size_t k = qubits.size();
        if (k > size_t(kMaxDiagQubits)) throw Unsupported{};
        const size_t D = size_t(1) << k;
        for (size_t h = 1; h < D; h <<= 1)
            for (size_t i = 0; i < D; i++)
                if (!(i & h)) {
                    const ld x = phi[i], y = phi[i | h];
                    phi[i] = x + y;
                    phi[i | h] = x - y;
                }
        for (size_t S = 0; S < D; S++) {
            uint64_t mask = 0;
            int cons = 0;
            for (size_t b = 0; b < k; b++)
                if ((S >> (k - 1 - b)) & 1) {
                    mask ^= mask_[size_t(qubits[b])];
                    cons ^= cons_[size_t(qubits[b])];
                }
            const ld a = phi[S] / ld(D);
            if (a != 0.0) phase(mask, cons, a);
        }
    }

    static void pattern(const std::vector<Control>& controls, std::vector<uint64_t>& qubits, size_t& index) {
        index = 0;
        for (const Control& c : controls) {
            qubits.push_back(c.qubit);
            index = (index << 1) | size_t(c.value);
        }
    }

    // -1 where every control holds and `target` is 1.
    void controlled_z(const std::vector<Control>& controls, uint64_t target) {
        std::vector<uint64_t> q;
        size_t j;
        pattern(controls, q, j);
        q.push_back(target);
        std::vector<ld> phi(size_t(1) << q.size(), 0.0);
        phi[(j << 1) | 1] = kPiL;
        phases(q, phi);
    }

    void one(uint64_t target, const Mat2& u, const std::vector<Control>& controls) {
        // u = e^{i alpha} RZ(beta) RY(theta) RZ(gamma)
        Polar p;
        if (!polar(u, p)) throw Unsupported{};
        const ld c = p.c, s = p.s;
        // Arguments of u00, u10 and u11; the fourth entry's follows from
        // unitarity, so the smaller pair gives one argument only.
        ld A, B, D;
        if (c >= s) {
            A = arg(p.x);
            D = arg(p.w);
            B = s > 0 ? arg(p.z) : A;
        } else {
            B = arg(p.z);
            const ld C = arg(p.y * -1.0L);
            A = c > 0 ? arg(p.x) : B;
            D = B + C - A;
        }
        const ld beta = B - A, gamma = D - B, alpha = A + (beta + gamma) / 2;
        norm += p.scale / ld(size_t(1) << controls.size());  // where controls hold only: its mean
        if (controls.empty()) {
            turn(global, alpha);
            // RZ(-+pi/2) RY(theta) RZ(+-pi/2) = RX(+-theta)
            const ld turns = std::fabs(beta + gamma) < kPiL ? 0.0L : std::nearbyint((beta + gamma) / (2 * kPiL));
            if (s > 0 && std::fabs(beta + gamma - turns * 2 * kPiL) <= kAngleTol &&
                std::fabs(std::fabs(std::remainder(beta, 2 * kPiL)) - kPiL / 2) <= kAngleTol) {
                // RZ(gamma) = RZ(-beta) (-1)^turns; beta = +-pi/2 up to whole turns, which cancel in the pair.
                if (std::fmod(std::fabs(turns), 2.0L) == 1.0L) turn(global, kPiL);
                rotation({target}, {}, c, std::remainder(beta, 2 * kPiL) < 0 ? s : -s);
                return;
            }
            phase(mask_[size_t(target)], cons_[size_t(target)], -gamma / 2, kAngleTol);
            rotation({target}, {target}, c, s);
            phase(mask_[size_t(target)], cons_[size_t(target)], -beta / 2, kAngleTol);
            return;
        }
        std::vector<uint64_t> q;
        size_t j;
        pattern(controls, q, j);
        const size_t nc = q.size();
        std::vector<uint64_t> qt = q;
        qt.push_back(target);
        auto crz = [&](ld angle) {
            std::vector<ld> phi(size_t(2) << nc, 0.0);
            phi[j << 1] = -angle / 2;
            phi[(j << 1) | 1] = angle / 2;
            phases(qt, phi);
        };
        const ld half = std::atan2(s, c) / 2;  // theta / 4
        crz(gamma);
        if (nc == 1) {
            // CZ RY CZ is the rotation about Z Y (its negative where the control holds at 0): no phases.
            rotation({target}, {target, q[0]}, std::cos(half), controls[0].value ? -std::sin(half) : std::sin(half));
        } else {
            controlled_z(controls, target);
            rotation({target}, {target}, std::cos(half), -std::sin(half));
            controlled_z(controls, target);
        }
        rotation({target}, {target}, std::cos(half), std::sin(half));
        crz(beta);
        std::vector<ld> phi(size_t(1) << nc, 0.0);
        phi[j] = alpha;
        phases(q, phi);
    }

    void cx(uint64_t c, bool value, uint64_t t) {
        if (dir_[size_t(t)] == 0) throw Unsupported{};
        mask_[size_t(t)] ^= mask_[size_t(c)];
        cons_[size_t(t)] ^= cons_[size_t(c)] ^ (value ? 0 : 1);
        if (dir_[size_t(c)]) dir_[size_t(c)] ^= dir_[size_t(t)];
    }

    void x(uint64_t target, const std::vector<Control>& controls) {
        if (dir_[size_t(target)] == 0) throw Unsupported{};
        if (controls.empty()) {
            cons_[size_t(target)] ^= 1;
        } else if (controls.size() == 1) {
            cx(controls[0].qubit, controls[0].value, target);
        } else {
            const ld r = std::sqrt(0.5L);
            auto h = [&] {  // H = RY(pi/2) Z
                phase(mask_[size_t(target)], cons_[size_t(target)], -kPiL / 2);  // -i Z
                turn(global, kPiL / 2);
                rotation({target}, {target}, r, r);
            };
            h();
            controlled_z(controls, target);
            h();
        }
    }

    void swap(uint64_t a, uint64_t b, const std::vector<Control>& controls) {
        if (controls.empty()) {
            if (dir_[size_t(a)] == 0 || dir_[size_t(b)] == 0) throw Unsupported{};
            std::swap(mask_[size_t(a)], mask_[size_t(b)]);
            std::swap(cons_[size_t(a)], cons_[size_t(b)]);
            std::swap(dir_[size_t(a)], dir_[size_t(b)]);
            return;
        }
        cx(b, true, a);
        std::vector<Control> both = controls;
        both.push_back({a, true});
        x(b, both);
        cx(b, true, a);
    }

    void diagonal(const Operation& op) {
        ld mean;
        if (!mean_modulus(op.values, mean)) throw Unsupported{};
        norm += mean;
        std::vector<ld> phi;
        for (cplx d : op.values) phi.push_back(arg(d));
        phases(op.qubits, phi);
    }

    // A one-qubit matrix, or cos I - i sin P for a two-qubit Pauli matrix P.
    void dense(const Operation& op) {
        if (op.qubits.size() == 1) {
            Mat2 u;
            for (int r = 0; r < 2; r++)
                for (int c = 0; c < 2; c++) u[size_t(r)][size_t(c)] = op.values[size_t(2 * r + c)];
            one(op.qubits[0], u, {});
            return;
        }
        if (op.qubits.size() != 2) throw Unsupported{};
        const uint64_t hi = op.qubits[0], lo = op.qubits[1];
        for (int X = 1; X < 4; X++)      // bit 1: hi, bit 0: lo
            for (int Z = 0; Z < 4; Z++) {
                // P|j> = i^ny (-1)^{Z.j} |j ^ X>; entry (j ^ X, j) of the matrix is -i s times that.
                const int ny = __builtin_popcount(unsigned(X & Z));
                const double c = op.values[0].re;
                auto factor = [&](int j) {  // -i i^ny (-1)^{Z.j}
                    cplx f(0, -1);
                    for (int y = 0; y < ny; y++) f = f * cplx(0, 1);
                    return __builtin_parity(unsigned(Z & j)) ? -f : f;
                };
                const cplx f0 = factor(0), e0 = op.values[size_t(X * 4)];
                const double s = e0.re * f0.re + e0.im * f0.im;
                bool ok = std::fabs(c * c + s * s - 1.0) <= double(kScaleTol);
                for (int r = 0; r < 4 && ok; r++)
                    for (int j = 0; j < 4 && ok; j++) {
                        cplx want(0);
                        if (r == j) want = cplx(c);
                        if (r == (j ^ X)) want = factor(j) * cplx(s);
                        const cplx got = op.values[size_t(r * 4 + j)];
                        ok = std::fabs(got.re - want.re) <= 1e-15 && std::fabs(got.im - want.im) <= 1e-15;
                    }
                if (!ok) continue;
                std::vector<uint64_t> xs, zs;
                if (X & 2) xs.push_back(hi);
                if (X & 1) xs.push_back(lo);
                if (Z & 2) zs.push_back(hi);
                if (Z & 1) zs.push_back(lo);
                rotation_of(xs, zs, c, s);
                return;
            }
        throw Unsupported{};
    }
};

// A subspace of places in echelon form (each vector's top bit in no other).
struct Span {
    uint32_t basis[kRotRegBits] = {};
    int dim = 0;
    uint32_t reduce(uint32_t v) const {
        for (int i = 0; i < dim; i++)
            if (v & (uint32_t(1) << (31 - __builtin_clz(basis[i])))) v ^= basis[i];
        return v;
    }
    bool add(uint32_t v) {
        v = reduce(v);
        if (!v || dim == kRotRegBits) return false;
        const uint32_t top = uint32_t(1) << (31 - __builtin_clz(v));
        for (int i = 0; i < dim; i++)
            if (basis[i] & top) basis[i] ^= v;
        basis[dim++] = v;
        return true;
    }
};

constexpr ld kMaxOwed = 200.0L;  // rotations may leave amplitudes e^200 too large before a table
constexpr int kWindow = 128;  // items a phase chooses among
// Rotations a phase may hold: its words then fit a launch argument whatever the
// circuit. A rotation takes at most 20 (its own two, a step, a table before it
// with another), each other item of the window 6 (an angle and a modulus of a slot: a mask
// word, a factor and a step each), the phase itself 56 (its head, three more tables, two to fetch ahead).
constexpr int kPhaseRotations = 82;
static_assert(20 * kPhaseRotations + 6 * (kWindow - kPhaseRotations) + 56 <= kRotParamWords);
// Below this many qubits half of them: planning then takes a third less time,
// where it is most of a call, for at most 3 % longer programs (either way).
constexpr int kWideQubits = 20;
constexpr int kPinnedLow = 2, kPinnedQubits = 20, kPinnedTile = 12;
struct Bits {
    uint64_t w[2] = {0, 0};
    void set(int i) { w[i >> 6] |= uint64_t(1) << (i & 63); }
    bool get(int i) const { return (w[i >> 6] >> (i & 63)) & 1; }
    bool within(const Bits& o) const { return !((w[0] & ~o.w[0]) | (w[1] & ~o.w[1])); }
    bool any() const { return (w[0] | w[1]) != 0; }
    int count() const { return __builtin_popcountll(w[0]) + __builtin_popcountll(w[1]); }
    // f(i) for every member in order.
    template <class F>
    void each(F&& f) const {
        for (int k = 0; k < 2; k++)
            for (uint64_t r = w[k]; r; r &= r - 1) f(64 * k + __builtin_ctzll(r));
    }
};
Bits operator&(const Bits& a, const Bits& b) { return {{a.w[0] & b.w[0], a.w[1] & b.w[1]}}; }
Bits operator|(const Bits& a, const Bits& b) { return {{a.w[0] | b.w[0], a.w[1] | b.w[1]}}; }
Bits operator^(const Bits& a, const Bits& b) { return {{a.w[0] ^ b.w[0], a.w[1] ^ b.w[1]}}; }
Bits without(const Bits& a, const Bits& b) { return {{a.w[0] & ~b.w[0], a.w[1] & ~b.w[1]}}; }

uint4 word(uint32_t x, uint32_t y, uint32_t z, uint32_t w) { return make_uint4(x, y, z, w); }
uint4 word(double a, double b) {
    uint4 u;
    double d[2] = {a, b};
    std::memcpy(&u, d, sizeof u);
    return u;
}

// A factor as doubles.  Entries recur (a CZ's are e^{+-i pi/4}), so the rounding
// of their modulus would add up: of the nearest pairs the one closest in modulus.
// `off` gains the logarithm of the modulus, and the angle, by which it misses.
struct Factor {
    ld re = 1.0L, im = 0.0L;
    void times(const Factor& f) {
        const ld r = re * f.re - im * f.im;
        im = re * f.im + im * f.re;
        re = r;
    }
};

// e^{ia} for |a| <= 2 pi: of the nearest multiple of pi/64, from a table, times
// that of the rest, below pi/128, by the power series to its 10th term (1e-23).
Factor turned(ld a) {
    static const std::vector<Factor> table = [] {
        std::vector<Factor> t;
        for (int k = -129; k <= 129; k++) t.push_back({std::cos(ld(k) * kPiL / 64), std::sin(ld(k) * kPiL / 64)});
        return t;
    }();
    const int k = int(std::lrint(double(a) * (64 / 3.14159265358979323846)));
    const ld x = a - ld(k) * (kPiL / 64), y = x * x;
    Factor f{1.0L - y / 2 * (1.0L - y / 12 * (1.0L - y / 30 * (1.0L - y / 56 * (1.0L - y / 90)))),
             x * (1.0L - y / 6 * (1.0L - y / 20 * (1.0L - y / 42 * (1.0L - y / 72))))};
    f.times(table[size_t(k + 129)]);
    return f;
}

ld grown(ld b) { return std::fabs(b) < 1e-10L ? 1.0L + b : std::exp(b); }

// The neighbours of a double away from zero and towards it (zero has none).
double outward(double x) {
    if (x == 0.0) return x;
    uint64_t u;
    std::memcpy(&u, &x, 8);
    u++;
    std::memcpy(&x, &u, 8);
    return x;
}
double inward(double x) {
    if (x == 0.0) return x;
    uint64_t u;
    std::memcpy(&u, &x, 8);
    u--;
    std::memcpy(&x, &u, 8);
    return x;
}

uint4 factor_word(const Factor& f, ld off[2]) {
    const ld re = f.re, im = f.im, S2 = re * re + im * im;
    const double x = double(re), y = double(im);
    double best[2] = {x, y};
    const ld x2 = ld(x) * x, y2 = ld(y) * y;
    ld miss = std::fabs(x2 + y2 - S2);
    const double tries[4][2] = {{outward(x), y}, {inward(x), y}, {x, outward(y)}, {x, inward(y)}};
    for (int i = 0; i < 4; i++) {
        const double* t = tries[i];
        const ld m = std::fabs(i < 2 ? ld(t[0]) * t[0] + y2 - S2 : x2 + ld(t[1]) * t[1] - S2);
        if (m < miss) {
            miss = m;
            best[0] = t[0];
            best[1] = t[1];
        }
    }
    const ld dx = best[0] - re, dy = best[1] - im, inv = 1.0L / S2;
    off[0] += (dx * re + dy * im) * inv;
    off[1] += (dy * re - dx * im) * inv;
    return word(best[0], best[1]);
}

// The phase after which a team's fetch counts as done (RotProgram::tell), by the
// SM cycles of a 12-qubit tile's phases as measured step by step.
int teller(const RotProgram& p) {
    const double rotation[4] = {0, 135, 300, 340};
    std::vector<double> upto;  // the work up to each phase's end
    for (int ph = 0; ph < p.nphases; ph++) {
        const uint4 head = p.words[size_t(3 * ph)];
        double cycles = 1100;
        for (uint32_t i = 0; i < head.y; i++) {
            const uint4 s = p.words[head.x + i];
            cycles += 75 + (s.x & 0xF00u ? 300 : 0) + (s.x & kRotTable ? 300 : 0);
            for (int j = 0; j < 4; j++) cycles += rotation[(s.x >> (2 * j)) & 3u];
            if (s.x & (kRotSlots | kRotSlotModuli)) cycles += 370 + 73.0 * double(s.w & 0xFFFFu);
        }
        upto.push_back((upto.empty() ? 0.0 : upto.back()) + cycles);
    }
    if (upto.empty()) return -1;
    const double half = 0.55 * (upto.back() + 3000.0);  // (the rest: stores and fetches)
    int tell = std::min(1, (p.nphases - 1) / 2);
    while (tell >= 0 && upto[size_t(tell)] > half) tell--;
    return tell;
}

class Scheduler {
  public:
    Scheduler(std::vector<Item> items, int m, int n, Lowering& lw, RotProgram& out)
        : items_(std::move(items)), m_(m), window_(n < kWideQubits ? kWindow / 2 : kWindow), lw_(lw), out_(out) {}

    void run() {
        for (size_t i = 0; i < items_.size(); i++)
            if (items_[i].rot || items_[i].a != 0.0) active_.push_back(int(i));
        struct Ph {
            uint4 head[3];
            std::vector<uint4> steps, rots;
        };
        std::vector<Ph> phases;
        std::vector<int> data_at;
        do {
            Ph p;
            data_at.push_back(int(tables_.size()));
            one_phase(p.head);
            pack(p.steps, p.rots);
            phases.push_back(std::move(p));
        } while (!active_.empty());
        if (phases.size() == 1 && phases[0].steps.empty()) {  // relabellings only
            phases.clear();
            data_at.clear();
        }
        size_t step_at = phases.size() * 3, rot_at = step_at;
        for (const Ph& p : phases) rot_at += p.steps.size();
        out_.words.clear();
        for (Ph& p : phases) {
            p.head[0].x = uint32_t(step_at);
            p.head[0].y = uint32_t(p.steps.size());
            p.head[2].y = uint32_t(rot_at);
            out_.words.insert(out_.words.end(), p.head, p.head + 3);
            step_at += p.steps.size();
            rot_at += p.rots.size();
        }
        for (const Ph& p : phases) out_.words.insert(out_.words.end(), p.steps.begin(), p.steps.end());
        for (const Ph& p : phases) out_.words.insert(out_.words.end(), p.rots.begin(), p.rots.end());
        out_.data = int(out_.words.size());
        out_.words.insert(out_.words.end(), tables_.begin(), tables_.end());
        // The kernel fetches a step and a rotation ahead.
        out_.words.insert(out_.words.end(), 2, make_uint4(0, 0, 0, 0));
        out_.nphases = int(phases.size());
        out_.phase_data = data_at;
        out_.tell = teller(out_);
    }

  private:
    std::vector<Item> items_;
    int m_, window_;
    Lowering& lw_;
    RotProgram& out_;
    std::vector<int> active_;  // items not applied yet, in order
    double fma_ = 0;

    // One part of a step, in the order the kernel applies a step's parts.
    struct Part {
        int place = 0;     // 0-3: rotation on register bit `place`; 4: other rotations; 5: table; 6: slot phases or moduli
        uint32_t d = 0, kind = 0, signs = 0, mask = 0, data = 0, count = 0;
        double t = 0.0, u = 0.0;
    };
    std::vector<Part> parts_;

    // Consecutive parts share a step as long as their places ascend: a step's
    // fixed cost (its branches fetch instructions the other warps are not
    // running) is about that of a rotation.
    void pack(std::vector<uint4>& steps, std::vector<uint4>& rots) {
        int last = 99;
        for (const Part& p : parts_) {
            if (p.place <= last) steps.push_back(make_uint4(0, 0, 0, 0));
            last = p.place;
            uint4& s = steps.back();
            if (p.place <= 4) {
                s.x |= p.place < 4 ? (p.kind + 1) << (2 * p.place) : (p.d | p.kind << 4) << 8;
                rots.push_back(word(p.t, p.u));
                if (p.kind != kRotPlain) rots.push_back(make_uint4(p.signs, p.mask, 0, 0));
            } else if (p.place == 5) {
                s.x |= kRotTable;
                s.y = p.data;
            } else {
                s.x |= p.kind;
                s.z = p.data;
                s.w = p.count | p.signs << 16;
            }
        }
        parts_.clear();
    }

    void one_phase(uint4 head[3]) {
        const int W = int(std::min<size_t>(active_.size(), size_t(window_)));
        std::vector<const Item*> it(static_cast<size_t>(W));
        for (int i = 0; i < W; i++) it[size_t(i)] = &items_[size_t(active_[size_t(i)])];
        // Earlier items an item does not commute with: by the parity of one's mask on
        // the other's direction, both ways (phases have no direction), a tile bit for
        // all items at a time.
        Bits pred[kWindow], all, rot_bits;
        uint32_t dir[kWindow];
        {
            Bits mask_has[kRotMaxTile], dir_has[kRotMaxTile];
            const uint32_t local = (1u << m_) - 1;
            for (int j = 0; j < W; j++) {
                const Item& x = *it[size_t(j)];
                dir[j] = x.v;
                Bits sum;
                for (uint32_t r = x.v; r; r &= r - 1) sum = sum ^ mask_has[__builtin_ctz(r)];
                for (uint32_t r = uint32_t(x.mask) & local; r; r &= r - 1) sum = sum ^ dir_has[__builtin_ctz(r)];
                pred[j] = sum;
                for (uint32_t r = x.v; r; r &= r - 1) dir_has[__builtin_ctz(r)].set(j);
                for (uint32_t r = uint32_t(x.mask) & local; r; r &= r - 1) mask_has[__builtin_ctz(r)].set(j);
                all.set(j);
                if (x.rot) rot_bits.set(j);
            }
        }
        // Directions modulo V: a rotation can run when its own is 0, or the one
        // direction `more` that V is tried with.
        Span V;
        uint32_t red[kWindow];
        for (int i = 0; i < W; i++) red[i] = dir[i];
        auto widen = [&](uint32_t v) {  // v into V, and its top bit out of the directions
            v = V.reduce(v);
            if (!V.add(v)) return;
            const uint32_t top = uint32_t(1) << (31 - __builtin_clz(v));
            for (int i = 0; i < W; i++)
                if (red[i] & top) red[i] ^= v;
        };
        // `exec` and what can run after it among `some`.
        auto closure = [&](const Bits& some, Bits exec) {
            int rots = (exec & rot_bits).count();
            without(some, exec).each([&](int i) {
                if (!pred[i].within(exec) || (dir[i] && rots == kPhaseRotations)) return;
                rots += dir[i] ? 1 : 0;
                exec.set(i);
            });
            return exec;
        };
        // Directions one at a time: the one that lets the most rotations in,
        // among those of the first rotations that only lack their direction.
        Bits inside = without(all, rot_bits);  // items without a direction outside V
        Bits exec = closure(inside, Bits{});
        while (V.dim < kRotRegBits) {
            uint32_t cand[8];
            Bits has[8];
            int count = 0;
            const Bits waiting = without(rot_bits, exec);
            waiting.each([&](int i) {
                if (count < 8 && red[i] && pred[i].within(exec) && std::find(cand, cand + count, red[i]) == cand + count)
                    cand[count++] = red[i];
            });
            waiting.each([&](int i) {
                const int k = int(std::find(cand, cand + count, red[i]) - cand);
                if (k < count) has[k].set(i);
            });
            if (count == 0) break;
            int best = -1, take = 0;
            Bits bestE;
            for (int k = 0; k < count; k++) {
                const Bits e = closure(inside | has[k], exec);
                const int r = (e & rot_bits).count();
                if (r > best) {
                    best = r;
                    take = k;
                    bestE = e;
                }
            }
            widen(cand[take]);
            inside = inside | has[take];
            exec = bestE;
        }
        for (int b = m_ - 1; b >= 0 && V.dim < kRotRegBits; b--) widen(1u << b);
        for (int i = 0; i < W; i++)
            if (!red[i]) inside.set(i);
        exec = closure(inside, exec);
        const bool last = int(active_.size()) == W && rot_bits.within(exec);

        // Order: rotations as far as they go, then the phases that hold the
        // next ones back, and so on.  `flush[f]` comes before the rotations of group f.
        std::vector<std::vector<int>> groups, flush;
        Bits done;
        while (true) {
            std::vector<int> g;
            without(rot_bits & exec, done).each([&](int i) {
                if (!pred[i].within(done)) return;
                done.set(i);
                g.push_back(i);
            });
            groups.push_back(std::move(g));
            Bits needed;
            without(rot_bits & exec, done).each([&](int j) {
                // Held back by phases only?
                const Bits missing = without(pred[j], done);
                if (!(missing & rot_bits).any()) needed = needed | missing;
            });
            if (!needed.any()) break;
            std::vector<int> ready;
            needed.each([&](int i) {
                if (pred[i].within(done)) ready.push_back(i);
            });
            for (int i : ready) done.set(i);
            flush.push_back(std::move(ready));
        }
        // V's basis: the directions of the first rotations, whose signs then
        // follow their own register bit where they commute.
        uint32_t basis[kRotRegBits];
        {
            Span got;
            auto want = [&](uint32_t v) {
                const int at = got.dim;
                if (got.add(v)) basis[at] = v;
            };
            for (auto& g : groups)
                for (int i : g) want(it[size_t(i)]->v);
            for (int j = 0; j < kRotRegBits; j++) want(V.basis[j]);
        }
        // After the last rotation every phase left; also those of a window without rotations.
        std::vector<int> tail;
        if (last || std::all_of(groups.begin(), groups.end(), [](const std::vector<int>& g) { return g.empty(); }))
            for (int i = 0; i < W; i++)
                if (!it[size_t(i)]->rot && !done.get(i) && pred[i].within(done)) tail.push_back(i);

        // The slots' places: the complement of V in which the parities of up to
        // four of those phases vanish (their factors then depend on the
        // register entry alone).
        const uint64_t local = (uint64_t(1) << m_) - 1;
        uint32_t M[kRotRegBits], R[kRotRegBits];  // masks and their parities on V's basis
        int nm = 0;
        auto on_V = [&](uint64_t mask) {
            uint32_t r = 0;
            for (int j = 0; j < kRotRegBits; j++) r |= uint32_t(parity(uint32_t(mask) & basis[j])) << j;
            return r;
        };
        uint32_t ech[kRotRegBits] = {};
        auto take = [&](uint64_t mask) {
            if (nm == kRotRegBits) return;
            uint32_t r = on_V(mask), red = r;
            for (int j = 0; j < kRotRegBits; j++)  // ech[j]: a vector whose top bit is j
                if (ech[kRotRegBits - 1 - j] && ((red >> (kRotRegBits - 1 - j)) & 1)) red ^= ech[kRotRegBits - 1 - j];
            if (!red) return;
            ech[31 - __builtin_clz(red)] = red;
            M[nm] = uint32_t(mask & local);
            R[nm++] = r;
        };
        for (auto& f : flush)
            for (int i : f)
                if (!(it[size_t(i)]->mask & ~local)) take(it[size_t(i)]->mask);
        for (int i : tail)
            if (!(it[size_t(i)]->mask & ~local)) take(it[size_t(i)]->mask);
        for (int i = 0; i < W; i++)
            if (!it[size_t(i)]->rot && pred[i].within(done) && !(it[size_t(i)]->mask & ~local))
                take(it[size_t(i)]->mask);
        for (int b = 0; b < m_; b++) take(uint64_t(1) << b);
        // Place p shifted within its coset so that every M vanishes: solve
        // sum_j x_j R[i]_j = M[i].p for x (R is invertible).
        uint32_t inv[kRotRegBits] = {};  // bit i of inv[j]: x_j takes M[i].p
        {
            uint32_t rows[kRotRegBits], id[kRotRegBits];
            for (int i = 0; i < kRotRegBits; i++) {
                rows[i] = R[i];
                id[i] = 1u << i;
            }
            for (int c = 0; c < kRotRegBits; c++) {
                int p = c;
                while (p < kRotRegBits && !((rows[p] >> c) & 1)) p++;
                std::swap(rows[c], rows[p]);
                std::swap(id[c], id[p]);
                for (int i = 0; i < kRotRegBits; i++)
                    if (i != c && ((rows[i] >> c) & 1)) {
                        rows[i] ^= rows[c];
                        id[i] ^= id[c];
                    }
            }
            for (int j = 0; j < kRotRegBits; j++) inv[j] = id[j];
        }
        auto project = [&](uint32_t p) {
            uint32_t mp = 0;
            for (int i = 0; i < kRotRegBits; i++) mp |= uint32_t(__builtin_parity(M[i] & p)) << i;
            for (int j = 0; j < kRotRegBits; j++)
                if (__builtin_parity(inv[j] & mp)) p ^= basis[j];
            return p;
        };
        // A basis of that complement; the first three (lanes 0-7 of a 16-byte
        // shared-memory wavefront) on distinct bank groups where it has such vectors.
        std::vector<uint32_t> U;
        {
            std::vector<uint32_t> red;
            auto independent = [&](uint32_t p, bool keep) {
                for (uint32_t r : red)
                    if (p & (uint32_t(1) << (31 - __builtin_clz(r)))) p ^= r;
                if (!p) return false;
                if (keep) {
                    const uint32_t top = uint32_t(1) << (31 - __builtin_clz(p));
                    for (uint32_t& r : red)
                        if (r & top) r ^= p;
                    red.push_back(p);
                }
                return true;
            };
            std::vector<uint32_t> unit;
            for (int b = 0; b < m_; b++) unit.push_back(project(1u << b));
            uint32_t banks[3] = {}, nb = 0;
            auto lane = [&](uint32_t p) {
                if (nb == 3 || int(U.size()) == m_ - kRotRegBits) return;
                uint32_t l = rot_swizzle(p) & 7u;
                for (uint32_t i = 0; i < nb; i++)
                    if (l & (1u << (31 - __builtin_clz(banks[i])))) l ^= banks[i];
                if (!p || !l || !independent(p, true)) return;
                const uint32_t top = 1u << (31 - __builtin_clz(l));
                for (uint32_t i = 0; i < nb; i++)
                    if (banks[i] & top) banks[i] ^= l;
                banks[nb++] = l;
                U.push_back(p);
            };
            for (uint32_t p : unit) lane(p);
            for (int i = 0; i < m_ && nb < 3; i++)
                for (int j = 0; j < i; j++) lane(unit[size_t(i)] ^ unit[size_t(j)]);
            for (uint32_t p : unit)
                if (int(U.size()) < m_ - kRotRegBits && p && independent(p, true)) U.push_back(p);
        }
        uint32_t slots_of[kWindow];
        Bits slots_known;
        auto slots = [&](int item) {  // kernel parity mask
            if (!slots_known.get(item)) {
                const uint64_t mask = it[size_t(item)]->mask;
                uint32_t s = uint32_t(mask >> m_) << kRotSlotBits;
                for (size_t i = 0; i < U.size(); i++) s |= uint32_t(parity(uint32_t(mask) & U[i])) << i;
                slots_of[item] = s;
                slots_known.set(item);
            }
            return slots_of[item];
        };
        static const std::array<uint32_t, kRotEntries> sign_bits = [] {
            std::array<uint32_t, kRotEntries> all{};
            for (uint32_t r = 0; r < uint32_t(kRotEntries); r++)
                for (uint32_t v = 0; v < uint32_t(kRotEntries); v++) all[r] |= uint32_t(parity(r & v)) << v;
            return all;
        }();
        auto signs = [&](uint32_t r) { return sign_bits[r]; };
        uint32_t combined[kRotEntries] = {};  // the places of the register entries
        for (uint32_t d = 1; d < uint32_t(kRotEntries); d++)
            combined[d] = combined[d & (d - 1)] ^ basis[__builtin_ctz(d)];
        uint32_t on_basis[kWindow];  // directions on the basis
        (rot_bits & exec).each([&](int i) {
            uint32_t d = 1;
            while (d < uint32_t(kRotEntries) && combined[d] != dir[i]) d++;
            on_basis[i] = d & uint32_t(kRotEntries - 1);
        });

        // Emission.  pend[j]: logarithm of the factor still owed by the entries
        // with register bit j clear (the others owe its negative).
        ld pend[kRotRegBits] = {};
        // A table: the phases `f` (none needs a slot parity), what the entries and
        // the state are owed, and the angle G.
        auto emit_table = [&](const std::vector<int>& f, ld G) {
            Part part;
            part.place = 5;
            part.data = uint32_t(tables_.size());
            parts_.push_back(part);
            Factor T[kRotEntries];
            ld g[kRotEntries];
            T[0] = turned(std::remainder(G, 2 * kPiL));
            g[0] = grown(uniform_);
            for (int v = 1; v < kRotEntries; v++) {
                T[v] = T[0];
                g[v] = g[0];
            }
            auto grow = [&](uint32_t r, ld b) {  // e^b, inverted by the parity of r
                const ld up = grown(b), down = 1.0L / up;
                for (uint32_t v = 0; v < uint32_t(kRotEntries); v++) g[v] *= __builtin_parity(r & v) ? down : up;
            };
            for (int j = 0; j < kRotRegBits; j++)
                if (pend[j] != 0.0L) grow(1u << j, pend[j]);
            for (int i : f) {
                const Item& x = *it[size_t(i)];
                const uint32_t r = on_V(x.mask);
                if (x.a != 0.0L) {
                    const Factor plus = turned(x.a), minus{plus.re, -plus.im};
                    for (uint32_t v = 0; v < uint32_t(kRotEntries); v++) T[v].times(__builtin_parity(r & v) ? minus : plus);
                }
                if (x.b != 0.0L) grow(r, x.b);
            }
            for (int v = 0; v < kRotEntries; v++) {
                T[v].re *= g[v];
                T[v].im *= g[v];
            }
            ld off[2] = {};
            for (const Factor& t : T) tables_.push_back(factor_word(t, off));
            for (ld& p : pend) p = 0.0;
            // What the table misses on average is owed to the next ones.
            uniform_ = -off[0] / kRotEntries;
            lw_.global -= off[1] / kRotEntries;
            out_.tables++;
            fma_ += 6.0;
        };
        // Rotations of a group in an order that fills steps: places ascending,
        // earlier ones that do not commute first.
        for (auto& g : groups) {
            std::vector<int> left = g, order;
            int at = -1;
            while (!left.empty()) {
                size_t pick = left.size();
                int place = 99;
                for (size_t i = 0; i < left.size(); i++) {
                    bool free = true;
                    for (size_t j = 0; j < i && free; j++) free = !pred[size_t(left[i])].get(left[j]);
                    if (!free) continue;
                    const uint32_t d = on_basis[left[i]];
                    const int p = (d & (d - 1)) == 0 && !it[size_t(left[i])]->imag ? __builtin_ctz(d) : 4;
                    if (p > at && p < place) {
                        place = p;
                        pick = i;
                    }
                }
                if (pick == left.size()) {
                    at = -1;
                    continue;
                }
                at = place;
                order.push_back(left[pick]);
                left.erase(left.begin() + long(pick));
            }
            g = order;
        }
        auto emit_flush = [&](std::vector<int> f, bool final) {
            // Phases that need no slot parity come along for nothing.
            bool free_table = final;
            for (int i : f) free_table = free_table || slots(i) == 0;
            if (free_table) {
                Bits listed = done | rot_bits;
                for (int i : f) listed.set(i);
                without(all, listed).each([&](int i) {
                    if (!pred[i].within(applied_) || slots(i) != 0) return;
                    f.push_back(i);
                    done.set(i);
                });
            }
            std::vector<std::pair<uint32_t, std::vector<int>>> by;  // register parity -> phases
            std::vector<int> here;  // of the table
            bool table = false;
            for (int i : f) {
                const Item& x = *it[size_t(i)];
                if (applied_.get(i)) continue;
                applied_.set(i);
                const uint32_t r = on_V(x.mask);
                if (slots(i) == 0) {
                    table = true;
                    here.push_back(i);
                    continue;
                }
                auto b = std::find_if(by.begin(), by.end(), [&](auto& e) { return e.first == r; });
                if (b == by.end()) {
                    by.push_back({r, {}});
                    b = by.end() - 1;
                }
                b->second.push_back(i);
            }
            // The slots' data first: what its rounding misses on average is settled by the table.
            struct SlotStep {
                uint32_t parity, kind;
                std::vector<int> terms;
                std::vector<uint4> factors;
            };
            std::vector<SlotStep> steps;
            for (auto& b : by) {
                SlotStep angles{b.first, kRotSlots, {}, {}}, moduli{b.first, kRotSlotModuli, {}, {}};
                for (int i : b.second) {
                    const Item& x = *it[size_t(i)];
                    if (x.a != 0.0) {
                        ld off[2] = {};
                        angles.terms.push_back(i);
                        angles.factors.push_back(factor_word(turned(x.a), off));
                        uniform_ -= off[0];
                    }
                    if (x.b != 0.0) {
                        const ld up = grown(x.b), down = 1.0L / up;
                        moduli.terms.push_back(i);
                        moduli.factors.push_back(word(double(up), double(down)));
                        uniform_ -= 0.5L * ((double(up) - up) / up + (double(down) - down) / down);
                    }
                }
                if (!angles.terms.empty()) steps.push_back(std::move(angles));
                if (!moduli.terms.empty()) steps.push_back(std::move(moduli));
            }
            ld G = 0.0;
            if (final) {
                G = std::remainder(lw_.global, 2 * kPiL);
                uniform_ += lw_.norm;
                table = table || G != 0.0;
                for (ld p : pend) table = table || p != 0.0;
                table = table || uniform_ != 0.0;
            }
            if (table) emit_table(here, G);
            for (const SlotStep& step : steps) {
                const size_t count = step.terms.size();
                Part part;
                part.place = 6;
                part.kind = step.kind;
                part.signs = signs(step.parity);
                part.data = uint32_t(tables_.size());
                part.count = uint32_t(count);
                parts_.push_back(part);
                for (size_t i = 0; i < count; i += 4) {
                    uint32_t m4[4] = {};
                    for (size_t j = i; j < std::min(count, i + 4); j++) m4[j - i] = slots(step.terms[j]);
                    tables_.push_back(word(m4[0], m4[1], m4[2], m4[3]));
                }
                tables_.insert(tables_.end(), step.factors.begin(), step.factors.end());
                out_.slot_phases++;
                const double each = step.kind == kRotSlots ? 6.0 : 2.0;
                fma_ += each + each * double(count) / kRotEntries;
            }
        };
        // The coordinate functional of register bit j: a mask that vanishes on the slots.
        auto functional = [&](int j) {
            uint64_t f = 0;
            for (int i = 0; i < kRotRegBits; i++)
                if ((inv[j] >> i) & 1) f ^= M[i];
            return f;
        };
        applied_ = Bits{};
        // The next table after each group (groups.size(): none in this phase).
        std::vector<size_t> table_at(groups.size() + 1, groups.size());
        for (size_t g = groups.size(); g-- > 0;) {
            bool table = g + 1 == groups.size() && last;
            if (g < flush.size())
                for (int i : flush[g]) table = table || slots(i) == 0;
            table_at[g] = table ? g : table_at[g + 1];
        }
        for (size_t g = 0; g < groups.size(); g++) {
            for (size_t gi = 0; gi < groups[g].size(); gi++) {
                const int i = groups[g][gi];
                const Item& x = *it[size_t(i)];
                const uint32_t d = on_basis[i], r = on_V(x.mask);
                const int low = __builtin_ctz(d);
                // In place where a table comes before the next rotation that mixes
                // this register bit, or where the factors owed can join a phase
                // that waits with the same mask.
                bool in_place = table_at[g] < groups.size();
                for (size_t h = g; h < groups.size() && h <= table_at[g] && in_place; h++)
                    for (size_t hi = h == g ? gi + 1 : 0; hi < groups[h].size() && in_place; hi++)
                        in_place = !((on_basis[groups[h][hi]] >> low) & 1);
                if (!in_place && table_at[g] == groups.size()) {
                    const uint64_t f = functional(low);
                    for (int j = 0; j < W && !in_place; j++)
                        in_place = !it[size_t(j)]->rot && !done.get(j) && it[size_t(j)]->mask == f &&
                                   pred[j].within(done);
                    for (size_t h = g; h < groups.size() && in_place; h++)
                        for (size_t hi = h == g ? gi + 1 : 0; hi < groups[h].size() && in_place; hi++)
                            in_place = !((on_basis[groups[h][hi]] >> low) & 1);
                }
                const ld lost = 0.5L * std::log1p(ld(x.t) * x.t);
                Part part;
                part.place = (d & (d - 1)) == 0 && !x.imag ? low : 4;
                part.d = d;
                part.kind = x.imag ? kRotImag : !in_place ? kRotKept
                            : part.place < 4 && r == (1u << low) && slots(i) == 0 ? kRotPlain : kRotSigned;
                part.signs = signs(r);
                part.mask = slots(i);
                part.t = x.t;
                part.u = double(ld(x.t) / (1.0L + ld(x.t) * x.t));
                // Entries that owe different factors must not mix, whatever the kind: those
                // without the factor i are in place without the look-ahead above.
                for (int j = 0; j < kRotRegBits; j++)
                    if (((d >> j) & 1) && pend[j] != 0.0) {
                        emit_table({}, 0.0);
                        break;
                    }
                if (part.kind == kRotKept) {
                    part.u = double(1.0L + ld(x.t) * x.t);
                    uniform_ -= lost + 0.5L * (part.u / (1.0L + ld(x.t) * x.t) - 1.0L);  // the determinant as it is rounded
                } else {
                    pend[low] -= lost;
                }
                parts_.push_back(part);
                applied_.set(i);
                out_.rotations++;
                fma_ += 4.0;
            }
            if (g < flush.size()) emit_flush(flush[g], false);
        }
        if (last || !tail.empty()) emit_flush(tail, last);
        if (!last && uniform_ < -kMaxOwed) {  // a circuit without phases: keep the amplitudes in range
            emit_table({}, 0.0);
        }
        // Factors still owed become phases of the register bits' parities (the
        // coordinate functionals), for later phases of the pass.
        std::vector<Item> owed;
        for (int j = 0; j < kRotRegBits; j++) {
            if (pend[j] == 0.0) continue;
            Item f;
            f.mask = functional(j);
            f.b = pend[j];
            owed.push_back(f);
        }
        head[0] = word(0, 0, rot_swizzle(basis[0]) | rot_swizzle(basis[1]) << 16,
                       rot_swizzle(basis[2]) | rot_swizzle(basis[3]) << 16);
        uint32_t b[12] = {};
        for (size_t i = 0; i < U.size(); i++) b[i] = rot_swizzle(U[i]);
        head[1] = word(b[0] | b[1] << 16, b[2] | b[3] << 16, b[4] | b[5] << 16, b[6] | b[7] << 16);
        head[2] = word(b[8], 0, 0, 0);
        std::vector<int> left;
        for (const Item& f : owed) {
            // Joined with a phase of the same mask that is ready, else first in line.
            bool joined = false;
            for (int i = 0; i < W && !joined; i++) {
                Item& x = items_[size_t(active_[size_t(i)])];
                if (x.rot || applied_.get(i) || x.mask != f.mask || !pred[i].within(applied_)) continue;
                x.b += f.b;
                joined = true;
            }
            if (joined) continue;
            left.push_back(int(items_.size()));
            items_.push_back(f);
        }
        for (int i = 0; i < int(active_.size()); i++)
            if (i >= W || !applied_.get(i)) left.push_back(active_[size_t(i)]);
        active_ = std::move(left);
        out_.flops_per_amp = fma_;
    }

    Bits applied_;
    ld uniform_ = 0.0;  // logarithm of a factor all amplitudes are owed
    std::vector<uint4> tables_;  // data of the tables and slot phases
};

}  // namespace

namespace {

// Whether an operation has a rotation form.
bool rotation_form(const Operation& op) {
    switch (op.type) {
        case Operation::One: {
            Polar p;
            return op.controls.size() < size_t(kMaxDiagQubits) && polar(op.m, p);
        }
        case Operation::X: return op.controls.size() < size_t(kMaxDiagQubits);
        case Operation::Swap: return op.controls.size() + 1 < size_t(kMaxDiagQubits);
        case Operation::Diagonal: {
            ld mean;
            return op.qubits.size() <= size_t(kMaxDiagQubits) && mean_modulus(op.values, mean);
        }
        default: break;
    }
    std::vector<uint64_t> q = op.touched();
    std::sort(q.begin(), q.end());
    auto local = [&](uint64_t x) { return uint64_t(std::lower_bound(q.begin(), q.end(), x) - q.begin()); };
    Operation l = op;
    l.target = local(op.target);
    l.a = local(op.a);
    l.b = local(op.b);
    for (Control& c : l.controls) c.qubit = local(c.qubit);
    for (uint64_t& x : l.qubits) x = local(x);
    std::vector<int> tile;
    for (size_t i = 0; i < q.size(); i++) tile.push_back(int(i));
    try {
        Lowering(tile, int(tile.size())).add(l);
    } catch (const Unsupported&) {
        return false;
    }
    return true;
}

}  // namespace

bool rotation_targets_only(const std::vector<Operation>& ops, size_t begin, size_t end, int n, int m) {
    m = std::min(m, n);
    if (m < kRotMinTile || m > kRotMaxTile || n - m > kRotMaxOuter || n == m) return false;
    bool wide = false;
    for (size_t i = begin; i < end; i++) wide = wide || (ops[i].type == Operation::Diagonal && ops[i].qubits.size() > 1);
    for (size_t i = begin; wide && i < end; i++) wide = rotation_form(ops[i]);
    return wide;
}

int rotation_pinned_low(const std::vector<Operation>& ops, size_t begin, size_t end, int n, int m) {
    if (n < kPinnedQubits || m < kPinnedTile) return 0;
    for (size_t i = begin; i < end; i++)
        if (!rotation_form(ops[i]) || int(ops[i].touched().size()) + kPinnedLow > m) return 0;
    return kPinnedLow;
}

bool register_phases_quicker(const std::vector<Operation>& ops, size_t begin, size_t end, int n) {
    if (n > 11) return false;
    // Microseconds of both forms beyond a launch, fitted to the device times of 18
    // families of circuits (5 to 11 qubits, 10 and 30 layers, one B200).
    double rotations = 0.0, ones = 0.0, multi = 0.0, size = 0.0;
    std::vector<size_t> last(size_t(n), end);  // the last many-qubit operation on each qubit
    for (size_t i = begin; i < end; i++) {
        const Operation& op = ops[i];
        const size_t nc = std::min<size_t>(op.controls.size(), 4);
        switch (op.type) {
            case Operation::One: {
                if (nc > 0) {
                    rotations += 0.8 * double(nc);
                    break;
                }
                // Z rotations on both sides of the Y rotation, or one.
                const cplx left = op.m[0][0] * cplx(op.m[1][0].re, -op.m[1][0].im);
                const cplx right = op.m[0][0] * cplx(op.m[0][1].re, -op.m[0][1].im);
                rotations += std::fabs(left.im) > 1e-15 && std::fabs(right.im) > 1e-15 ? 0.31 : 0.2;
                break;
            }
            case Operation::X: {
                const double by_controls[5] = {0.0, 0.0, 0.55, 1.7, 3.7};
                rotations += by_controls[nc];
                break;
            }
            case Operation::Swap: rotations += nc == 0 ? 0.0 : nc == 1 ? 0.65 : 1.7; break;
            case Operation::Diagonal: rotations += 0.06 * double(op.qubits.size()); break;
            default: rotations += 0.4; break;
        }
        const std::vector<uint64_t> qubits = op.touched();
        size += double(qubits.size());
        if (qubits.size() <= 1) {
            ones += double(qubits.size());
            continue;
        }
        // (one on the qubits of the one before is fused with it)
        const size_t before = last[size_t(qubits[0])];
        bool same = before != end && ops[before].touched().size() == qubits.size();
        for (uint64_t q : qubits) same = same && last[size_t(q)] == before;
        if (!same) multi += 1.0;
        for (uint64_t q : qubits) last[size_t(q)] = i;
    }
    // Phases larger than a launch argument are read from device memory.
    const double phases = (0.4 * multi + 0.12 * ones) * (size > 410.0 ? 1.75 : 1.0);
    const double share = n <= 7 ? 0.86 : n <= 9 ? 0.9 : n == 10 ? 1.04 : 1.35;  // matrices take longer as the tile grows
    return rotations > share * phases;
}

bool build_rotation_pass(const std::vector<Operation>& ops, const std::vector<int>& tile_qubits, int n,
                         RotProgram& out) {
    const int m = int(tile_qubits.size());
    if (m < kRotMinTile || m > kRotMaxTile || n - m > kRotMaxOuter) return false;
    Lowering lw(tile_qubits, n);
    try {
        for (const Operation& op : ops) lw.add(op);
    } catch (const Unsupported&) {
        return false;
    }
    out = RotProgram{};
    out.m = m;
    Scheduler s(lw.items, m, n, lw, out);
    s.run();
    // Place of tile index e: sum over q of (e_q ^ const_q ^ outer part) v_q.
    uint32_t c = 0;
    for (int q = 0; q < m; q++) {
        const size_t g = size_t(tile_qubits[size_t(q)]);
        const uint32_t v = lw.dirs()[g];
        out.out_dir[q] = uint16_t(rot_swizzle(v));
        if (lw.consts()[g]) c ^= v;
        for (int j = 0; j < n - m; j++)
            if ((lw.masks()[g] >> (m + j)) & 1) out.out_outer[j] = uint16_t(out.out_outer[j] ^ rot_swizzle(v));
        if (parity64(lw.sign & v)) out.sign_local |= 1u << q;
    }
    out.out_const = uint16_t(rot_swizzle(c));
    // sign . p over p(e): on e through sign.v_q, on the tile index through its
    // own bits and through the places' outer part.
    out.sign_const = parity64(lw.sign & c);
    for (int j = 0; j < n - m; j++) {
        int bit = int((lw.sign >> (m + j)) & 1);
        for (int q = 0; q < m; q++) {
            const size_t g = size_t(tile_qubits[size_t(q)]);
            if ((lw.masks()[g] >> (m + j)) & 1) bit ^= parity64(lw.sign & lw.dirs()[g]);
        }
        if (bit) out.sign_outer |= 1u << j;
    }
    return true;
}

std::vector<RotProgram> split_rotation_pass(RotProgram&& p, size_t most) {
    std::vector<RotProgram> parts;
    if (p.words.size() <= most) {
        parts.push_back(std::move(p));
        return parts;
    }
    const int end = int(p.words.size()) - 2 - p.data;
    auto rots_end = [&](int ph) { return ph + 1 < p.nphases ? p.words[size_t(3 * ph + 5)].y : uint32_t(p.data); };
    auto data_end = [&](int ph) { return ph + 1 < p.nphases ? p.phase_data[size_t(ph + 1)] : end; };
    auto size = [&](int ph) {
        const uint4 *h = &p.words[size_t(3 * ph)];
        return size_t(3 + h[0].y + rots_end(ph) - h[2].y) + size_t(data_end(ph) - p.phase_data[size_t(ph)]);
    };
    for (int first = 0; first < p.nphases;) {
        int last = first;
        for (size_t total = 2 + size(first); last + 1 < p.nphases; last++) {
            total += size(last + 1);
            if (total > most) break;
        }
        RotProgram part;
        part.m = p.m;
        part.nphases = last + 1 - first;
        const int base = p.phase_data[size_t(first)];
        uint32_t step_at = uint32_t(3 * part.nphases), rot_at = step_at;
        for (int ph = first; ph <= last; ph++) rot_at += p.words[size_t(3 * ph)].y;
        for (int ph = first; ph <= last; ph++) {
            const uint4 *h = &p.words[size_t(3 * ph)];
            part.words.insert(part.words.end(), h, h + 3);
            uint4* own = &part.words[part.words.size() - 3];
            own[0].x = step_at;
            own[2].y = rot_at;
            step_at += h[0].y;
            rot_at += rots_end(ph) - h[2].y;
        }
        for (int ph = first; ph <= last; ph++) {
            const uint4 head = p.words[size_t(3 * ph)];
            for (uint32_t i = 0; i < head.y; i++) {
                uint4 s = p.words[head.x + i];
                if (s.x & kRotTable) s.y -= uint32_t(base);
                if (s.x & (kRotSlots | kRotSlotModuli)) s.z -= uint32_t(base);
                part.words.push_back(s);
            }
        }
        auto take = [&](size_t from, size_t to) {
            part.words.insert(part.words.end(), p.words.begin() + long(from), p.words.begin() + long(to));
        };
        take(p.words[size_t(3 * first + 2)].y, rots_end(last));
        part.data = int(part.words.size());
        take(size_t(p.data + base), size_t(p.data + data_end(last)));
        part.words.insert(part.words.end(), 2, make_uint4(0, 0, 0, 0));
        part.tell = teller(part);
        // Places stay as they are between the parts; the last one leaves the frame.
        for (int q = 0; q < p.m; q++) part.out_dir[q] = uint16_t(rot_swizzle(1u << q));
        parts.push_back(std::move(part));
        first = last + 1;
    }
    RotProgram& out = parts.back();
    std::copy(std::begin(p.out_dir), std::end(p.out_dir), out.out_dir);
    std::copy(std::begin(p.out_outer), std::end(p.out_outer), out.out_outer);
    out.out_const = p.out_const;
    out.sign_local = p.sign_local;
    out.sign_outer = p.sign_outer;
    out.sign_const = p.sign_const;
    out.flops_per_amp = p.flops_per_amp;
    out.rotations = p.rotations;
    out.tables = p.tables;
    out.slot_phases = p.slot_phases;
    return parts;
}

}  // namespace dq
