// host_readable.h against memory that can and cannot be read: pages without read
// permission, unmapped ones, a read-only file map and the pages behind its end;
// rows with unreadable pages between them; more pages than one system call takes.
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <sys/mman.h>

#include "../../mosaic-art-rust_gb300/csrc/host_readable.h"

static int bad = 0;
static void expect(mg::ReadProbe& p, bool want, const char* what) {
  const bool got = p.end();
  if (got != want || (!want && p.error() != EFAULT)) {
    printf("%s: %d, expected %d, error %d\n", what, (int)got, (int)want, p.error());
    bad = 1;
  }
}

int main() {
  const size_t page = (size_t)sysconf(_SC_PAGESIZE);
  mg::ReadProbe p;
  auto check = [&](bool want, const char* what, const void* at, size_t bytes, size_t rows, size_t stride) {
    if (!p.begin()) abort();
    p.add(at, bytes, rows, stride);
    expect(p, want, what);
  };
  const size_t n = 3000;
  char* m = (char*)mmap(nullptr, n * page, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  check(true, "fresh pages", m, n * page, 1, n * page);
  check(true, "inside a page", m + 5, 7, 1, 7);
  check(true, "nothing", nullptr, 0, 5, 9);
  mprotect(m + (n - 1) * page, page, PROT_NONE);
  check(true, "up to the last byte", m, (n - 1) * page, 1, (n - 1) * page);
  check(false, "one byte more", m, (n - 1) * page + 1, 1, (n - 1) * page + 1);
  check(false, "that byte alone", m + (n - 1) * page, 1, 1, 1);
  mprotect(m + 2 * page, page, PROT_NONE);
  check(false, "the third page", m, (n - 1) * page, 1, (n - 1) * page);
  check(true, "rows on either side of it", m + 2 * page - 100, 100, 2, page + 100);
  check(false, "rows with a byte in it", m + 2 * page - 100, 101, 2, page + 100);
  munmap(m + 4 * page, page);
  check(false, "an unmapped page", m + 3 * page, 2 * page, 1, 2 * page);
  check(false, "null", nullptr, 1, 1, 1);
  check(true, "after all these", m, page, 1, page);
  if (!p.begin()) abort();
  p.add(m, 10, 1, 10);
  p.add(m + 2 * page, 10, 1, 10);
  p.add(m, 10, 1, 10);
  expect(p, false, "one of three");

  char name[] = "/tmp/host_readable_XXXXXX";
  const int fd = mkstemp(name);
  unlink(name);
  if (fd < 0 || ftruncate(fd, (off_t)(4 * page)) != 0) abort();
  char* f = (char*)mmap(nullptr, 4 * page, PROT_READ, MAP_SHARED, fd, 0);
  check(true, "a read-only file map", f, 4 * page, 1, 4 * page);
  if (ftruncate(fd, (off_t)(2 * page)) != 0) abort();
  check(true, "what is left of the file", f, 2 * page, 1, 2 * page);
  check(false, "behind its end", f, 4 * page, 1, 4 * page);
  printf(bad ? "failed\n" : "ok\n");
  return bad;
}
