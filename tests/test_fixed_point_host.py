"""The reduction's fixed-point arithmetic on the CPU (csrc/fixp.cuh compiles for both).

Running sums: a lane's 128 products at order 4096, with every low limb at its largest and of
one sign, against exact integers; one unit for the rounding of the sum and one for the
parts carried on.

The whole reduction (host/reduction.cu has its steps): random positive semidefinite matrices
with sectors, zeros, rank deficiency, grading and rounding-size entries keep a backward error
of 64 n 2^-53 and stay within the range of their integers."""

import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "tensornetworks.jl_gb300", "csrc")

SOURCE = r"""
#include "fixp.cuh"
using namespace tn::fixp;
int main() {
    int bad = 0;
    unsigned long long r = 88172645463325252ull;
    auto rnd = [&] { r ^= r << 13; r ^= r >> 7; r ^= r << 17; return r; };
    for (int trial = 0; trial < 2000; ++trial) {
        Dot s{0, 0, 0, 0, 0, 0};
        i128 ex = 0, ey = 0;
        const ll al = trial % 3 == 0 ? (1ll << 28) - 1 : trial % 3 == 1 ? -(1ll << 28) : (ll)(rnd() >> 36) - (1ll << 27);
        for (int t = 0; t < 128; ++t) {
            const ll hi = (ll)(rnd() >> 40) - (1ll << 23), vh = (ll)(rnd() >> 43) - (1ll << 20);
            // entries in units of 2^-61 (their limbs hold the upper 61 bits but three), v 2^-56
            const zint a{((hi << 29) + al) * 8, ((vh << 29) + al) * 8}, v{(vh << 29) + al, (hi % 1048576 << 29) - al};
            dot_add(s, a, limbs29(v));
            if ((t & 31) == 31) dot_carry(s);
            ex += (i128)a.x * v.x - (i128)a.y * v.y;
            ey += (i128)a.x * v.y + (i128)a.y * v.x;
        }
        const zint p = dot_value(s);
        const i128 dx = ((i128)p.x << 56) - ex, dy = ((i128)p.y << 56) - ey, tol = (i128)2 << 56;
        bad += dx > tol || dx < -tol || dy > tol || dy < -tol;
    }
    printf("%d\n", bad);
    return 0;
}
"""


def build(src, exe):
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    subprocess.run([nvcc, "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-I", CSRC, str(src), "-o", str(exe)],
                   check=True, capture_output=True)


def test_low_limbs_of_one_sign(tmp_path):
    src, exe = tmp_path / "dot.cu", tmp_path / "dot"
    src.write_text(SOURCE)
    build(src, exe)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout == "0\n"


@pytest.fixture(scope="module")
def reduction(tmp_path_factory):
    exe = tmp_path_factory.mktemp("reduction") / "reduction"
    build(os.path.join(os.path.dirname(os.path.abspath(__file__)), "host", "reduction.cu"), exe)
    return exe


@pytest.mark.parametrize("count,order,flat", [(150000, 6, 0), (150000, 12, 1), (1500, 60, 1), (40, 300, 1)])
def test_backward_error(reduction, count, order, flat):
    out = subprocess.run([str(reduction), "1", str(count), str(order), str(flat)], check=True, capture_output=True, text=True)
    assert out.stdout.startswith("0 of "), out.stdout


@pytest.mark.parametrize("n", [3, 8, 40, 150, 300])
def test_equal_rows(reduction, n):
    """Rows that are all alike below a larger one: the norm of what is left is the sum of its
    diagonal, while every row's exponent goes by its own."""
    out = subprocess.run([str(reduction), str(n)], check=True, capture_output=True, text=True)
    assert out.stdout == "0 of 7\n"


def test_products_of_rows_left_small(reduction):
    """A 12-row matrix whose update raises a row's products by more than |w|^2 says: they
    have to stay within their range of four (4.004 where the exponents minded |w|^2 once)."""
    case = os.path.join(os.path.dirname(os.path.abspath(__file__)), "host", "lifted_products.txt")
    out = subprocess.run([str(reduction), "file", case], check=True, capture_output=True, text=True)
    assert out.stdout.startswith("0 of 1"), out.stdout


def test_scale_of_a_product_that_rounds_to_zero(tmp_path):
    """q_exponent from v^H A v known to two units a row: the root of the true value, and so the
    update vectors, stay within a factor of two of the scale."""
    src, exe = tmp_path / "q.cu", tmp_path / "q"
    src.write_text(r"""
#include "fixp.cuh"
using namespace tn::fixp;
int main() {
    int bad = 0;
    for (int n = 2; n <= 4096; n = 2 * n - 1)
        for (int k = 0; k < 62; ++k)
            for (ll off = -2; off <= 2; ++off) {
                const ll q = k ? 1ll << (k - 1) : 0;
                const int h = q_exponent(q + off * n, -1000, 0, n);
                bad += ldexp((double)q, -60) > 4.0 * ldexp(1.0, 2 * h);
            }
    printf("%d\n", bad);
    return 0;
}
""")
    build(src, exe)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout == "0\n"


def test_a_limb_that_has_no_negative(tmp_path):
    """make_w with the lower limb of tau's imaginary part at -2^31, against exact integers."""
    src, exe = tmp_path / "w.cu", tmp_path / "w"
    src.write_text(r"""
#include "fixp.cuh"
using namespace tn::fixp;
int main() {
    const zint tau{(1ll << 60) - 12345, (1ll << 60) - (1ll << 31)}, p{(3ll << 55) + 77, (1ll << 57) + 5}, v{1ll << 49, 3ll << 48};
    const ll al = (1ll << 58) + 9;
    const zint w = make_w(tau, p, al, v);
    const i128 x = (i128)tau.x * p.x - (i128)tau.y * p.y, y = (i128)tau.x * p.y + (i128)tau.y * p.x;
    const ll wx = (ll)(x >> 63) - (ll)((i128)al * v.x >> 56), wy = (ll)(y >> 63) - (ll)((i128)al * v.y >> 56);
    printf("%d\n", llabs(w.x - wx) <= 4 && llabs(w.y - wy) <= 4);
    return 0;
}
""")
    build(src, exe)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout == "1\n"
