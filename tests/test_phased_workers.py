"""The host threads of large ray batches (csrc/phased_workers.hpp): phases in order, all work done however many
threads the system gives, and failures that end the call without a hang."""
import os
import subprocess
import textwrap

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "optical-pathtracer_b200", "csrc")

PROGRAM = textwrap.dedent(r"""
    #include "phased_workers.hpp"
    #include <atomic>
    #include <cstdio>
    #include <cstdlib>
    #include <stdexcept>
    #include <system_error>
    // a thread that the system refuses once `given` of them exist
    static int given;
    struct Counted {
        std::thread t;
        template <class F> explicit Counted(F&& f) {
            if (given-- <= 0) throw std::system_error(std::make_error_code(std::errc::resource_unavailable_try_again));
            t = std::thread(std::forward<F>(f));
        }
        Counted(Counted&&) = default;
        void join() { t.join(); }
    };
    int main(int argc, char** argv) {
        const int wanted = std::atoi(argv[1]), fail = std::atoi(argv[3]);  // 0 none, 1 first phase, 2 second
        given = std::atoi(argv[2]);
        const int expect = 1 + (given < wanted - 1 ? given : wanted - 1);
        for (int rep = 0; rep < 200; ++rep) {
            given = std::atoi(argv[2]);
            std::atomic<int> up{0}, down{0}, upDone{0}, downDone{0};
            bool order = true;
            owec::PhasedWorkersOf<Counted> gang(wanted);
            bool threw = false;
            try {
                gang.run([&](int k) { for (int i; (i = up++) < 1000;) { if (fail == 1 && i == 500) throw std::runtime_error("up"); ++upDone; } (void)k; },
                         [&](int k) { if (k >= expect || upDone != 1000) order = false; for (int i; (i = down++) < 1000;) { if (fail == 2 && i == 500) throw std::runtime_error("down"); ++downDone; } });
            } catch (const std::runtime_error&) { threw = true; }
            if (!order) { std::puts("order"); return 1; }
            if (threw != (fail != 0)) { std::puts("exception"); return 1; }
            if (fail == 0 && (upDone != 1000 || downDone != 1000)) { std::puts("work"); return 1; }
            if (fail == 1 && downDone != 0) { std::puts("went on"); return 1; }
        }
        std::puts("ok");
        return 0;
    }
""")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("phased")
    (d / "p.cpp").write_text(PROGRAM)
    exe = str(d / "p")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(d / "p.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("failing_phase", [0, 1, 2])
@pytest.mark.parametrize("wanted,given", [(1, 0), (4, 3), (4, 2), (4, 0), (9, 8)])
def test_phases_with_the_threads_there_are(program, wanted, given, failing_phase):
    r = subprocess.run([program, str(wanted), str(given), str(failing_phase)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
