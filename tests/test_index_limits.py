"""Sizes at which 32-bit positions end, checked on the host alone."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mops_b200", "csrc")


def test_positions_and_what_the_walks_look_ahead_fit_an_int(tmp_path):
    """The walks form positions up to 102 behind the last entry in an int."""
    source = tmp_path / "limits.cpp"
    source.write_text("""
        #include "checks.hpp"
        using mops_b200::positions_fit_int;
        constexpr int64_t most = INT32_MAX;
        static_assert(!positions_fit_int(most + 1) && !positions_fit_int(most) && !positions_fit_int(most - 101), "");
        static_assert(positions_fit_int(most - 1000) && positions_fit_int(0), "");
        int main() {}
    """)
    subprocess.run(["g++", "-std=c++17", "-fsyntax-only", "-I", CSRC, str(source)], check=True)
