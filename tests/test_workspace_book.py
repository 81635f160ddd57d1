"""CPU: the book of the contexts' workspaces (csrc/cas_workspace.h).

The header compiles as plain C++; a harness built here runs it with a counting allocator: growth to the last product's
need, products over the limit between small ones, the limit over several contexts, allocations that fail, what can be
taken back and what cannot, and threads that begin and end products while another takes back what is idle.
"""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "contention-aware-spgemm_b200", "csrc")

HARNESS = r"""
#include "cas_workspace.h"
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <thread>

#define EXPECT(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
constexpr size_t MB = size_t(1) << 20;
std::atomic<int> allocs{0}, frees{0};
std::atomic<bool> fail{false};
char* get(size_t n) {
  if (fail) return nullptr;
  ++allocs;
  return static_cast<char*>(malloc(n));
}
void put(char* p) { ++frees; free(p); }

// a product that asks for n bytes in two parts; how many of them fitted
int product(cas::WorkspaceBook& book, cas::Workspace& w, size_t limit, size_t n) {
  book.begin(w, limit, get, put);
  char *a = w.take(n / 2), *b = w.take(n - n / 2);
  if (a) memset(a, 1, n / 2);
  if (b) memset(b, 2, n - n / 2);
  if (a && b && (a[0] != 1 || a[n / 2 - 1] != 1)) return -1;
  book.end(w);
  return (a != nullptr) + (b != nullptr);
}

int sizes() {
  cas::WorkspaceBook book;
  cas::Workspace w;
  book.join(w);
  EXPECT(product(book, w, 64 * MB, 10 * MB) == 0);  // the first finds none
  for (int i = 0; i < 20; ++i) EXPECT(product(book, w, 64 * MB, (i % 2 ? 10 : 3) * MB) == 2);
  EXPECT(allocs == 1 && frees == 0);
  // a product over the limit between small ones: the workspace stays
  for (int i = 0; i < 20; ++i) {
    EXPECT(product(book, w, 64 * MB, 200 * MB) == 0);
    EXPECT(product(book, w, 64 * MB, 10 * MB) == 2);
  }
  EXPECT(allocs == 1 && frees == 0 && book.held() == w.cap && w.cap >= 10 * MB);
  EXPECT(product(book, w, 64 * MB, 30 * MB) < 2);
  EXPECT(product(book, w, 64 * MB, 30 * MB) == 2);
  EXPECT(allocs == 2 && frees == 1);
  book.leave(w, put);
  EXPECT(frees == 2 && book.held() == 0 && !w.mem);
  return 0;
}

int limit() {
  cas::WorkspaceBook book;
  cas::Workspace a, b;
  book.join(a);
  book.join(b);
  product(book, a, 32 * MB, 20 * MB);
  EXPECT(product(book, a, 32 * MB, 20 * MB) == 2);
  product(book, b, 32 * MB, 20 * MB);
  EXPECT(product(book, b, 32 * MB, 20 * MB) == 0 && b.cap == 0);  // 40 MB would be over the limit
  EXPECT(product(book, b, 32 * MB, 8 * MB) == 0);
  EXPECT(product(book, b, 32 * MB, 8 * MB) == 2);
  EXPECT(book.held() <= 32 * MB && book.held() == a.cap + b.cap);
  book.leave(a, put);
  product(book, b, 32 * MB, 20 * MB);
  EXPECT(product(book, b, 32 * MB, 20 * MB) == 2);
  // an allocation that fails leaves nothing on the book
  product(book, b, 32 * MB, 28 * MB);
  fail = true;
  EXPECT(product(book, b, 32 * MB, 28 * MB) == 0 && b.cap == 0 && book.held() == 0);
  fail = false;
  EXPECT(product(book, b, 32 * MB, 28 * MB) == 2);
  book.leave(b, put);
  EXPECT(book.held() == 0);
  return 0;
}

int reclaim() {
  cas::WorkspaceBook book;
  cas::Workspace a, b;
  book.join(a);
  book.join(b);
  for (int i = 0; i < 2; ++i) { product(book, a, 64 * MB, 8 * MB); product(book, b, 64 * MB, 8 * MB); }
  book.begin(a, 64 * MB, get, put);  // a product runs in a
  char* p = a.take(MB);
  EXPECT(p && a.mem && b.mem);
  book.reclaim(put);
  EXPECT(a.mem && !b.mem && b.cap == 0 && book.held() == a.cap);
  memset(p, 3, MB);
  book.end(a);
  book.reclaim(put);
  EXPECT(!a.mem && book.held() == 0);
  EXPECT(product(book, b, 64 * MB, 8 * MB) == 2);  // and grows again
  book.leave(a, put);
  book.leave(b, put);
  return 0;
}

int threads() {
  cas::WorkspaceBook book;
  std::atomic<int> bad{0}, left{4};
  std::thread ts[5];
  for (int t = 0; t < 4; ++t)
    ts[t] = std::thread([&, t] {
      cas::Workspace w;
      book.join(w);
      for (int i = 0; i < 2000; ++i)
        if (product(book, w, 3 * 4 * MB, size_t(1 + (i + t) % 4) * MB) < 0) ++bad;
      book.leave(w, put);
      --left;
    });
  ts[4] = std::thread([&] {
    while (left > 0) {
      book.reclaim(put);
      if (book.held() > 3 * 4 * MB) ++bad;
      std::this_thread::yield();
    }
  });
  for (auto& t : ts) t.join();
  EXPECT(bad == 0 && book.held() == 0);
  return 0;
}

int main(int, char** argv) {
  const int rc = !strcmp(argv[1], "sizes") ? sizes() : !strcmp(argv[1], "limit") ? limit()
               : !strcmp(argv[1], "reclaim") ? reclaim() : threads();
  if (rc == 0 && allocs != frees) { printf("%d allocations, %d freed\n", allocs.load(), frees.load()); return 1; }
  return rc;
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("workspace")
    (d / "t.cpp").write_text(HARNESS)
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O1", "-g", "-Wall", "-Wextra", "-pthread", "-I", CSRC, "-o",
                    str(d / "t"), str(d / "t.cpp")], check=True)
    return str(d / "t")


@pytest.mark.parametrize("what", ["sizes", "limit", "reclaim", "threads"])
def test_book(harness, what):
    p = subprocess.run([harness, what], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0, p.stdout + p.stderr
