// host_readable.h -- whether memory of this process can be read, found out
// without reading it from here: host code, no CUDA.
//
// A kernel that reads the caller's memory in place (mg_generate) faults on the GPU
// where a page cannot be read -- unmapped, without read permission, beyond the end
// of a file that was truncated -- and that ends the context for all its users.  So
// the operating system is asked first, by a write of one byte of every page to a
// pipe, which fails (EFAULT) where a read would fault.  It also maps pages that
// were not touched yet, which the host does faster than the GPU's faults.  It costs
// mg_generate 4 us of 207 for 33 small materials and 18 of 691 for 25 MB in pages of
// 64 KB (400 pieces, one call; 28 without the prefetch, 20 by populating the page
// tables instead, MADV_POPULATE_READ, which takes 30 times that in pages of 4 KB).
#pragma once
#include <errno.h>
#include <fcntl.h>
#include <stdint.h>
#include <sys/uio.h>
#include <unistd.h>

#include <vector>

namespace mg {

class ReadProbe {
 public:
  ReadProbe() = default;
  ReadProbe(const ReadProbe&) = delete;
  ReadProbe& operator=(const ReadProbe&) = delete;
  ~ReadProbe() {
    if (fd_[0] >= 0) close(fd_[0]);
    if (fd_[1] >= 0) close(fd_[1]);
  }

  // Starts over.  False: there is no pipe to be had, nothing can be told.
  bool begin() {
    pieces_.clear();
    last_ = 0;
    ok_ = true;
    error_ = 0;
    if (fd_[0] < 0 && pipe2(fd_, O_CLOEXEC | O_NONBLOCK) != 0) {
      fd_[0] = fd_[1] = -1;
      return false;
    }
    if (page_ == 0) page_ = (uintptr_t)sysconf(_SC_PAGESIZE);
    return true;
  }

  // `rows` rows of `bytes` bytes, `stride` (>= bytes) apart.  Bytes between rows are not looked at.
  void add(const void* p, size_t bytes, size_t rows, size_t stride) {
    const uintptr_t a = (uintptr_t)p;
    if (bytes == 0 || rows == 0) return;
    if (stride - bytes < page_) {  // no page lies between two rows
      range(a, a + stride * (rows - 1) + bytes);
    } else {
      for (size_t r = 0; r < rows; ++r) range(a + stride * r, a + stride * r + bytes);
    }
  }

  // Whether everything added since begin() can be read.
  bool end() {
    send();
    return ok_;
  }
  // After a false end(): the error it came from (EFAULT: memory that cannot be read).
  int error() const { return error_; }

 private:
  static constexpr size_t kPieces = 1024;  // IOV_MAX

  void range(uintptr_t lo, uintptr_t hi) {
    for (uintptr_t at = lo; at < hi && ok_; at = (at / page_ + 1) * page_) {
      const uintptr_t page = at / page_ + 1;
      if (page == last_) continue;
      last_ = page;
      __builtin_prefetch((const void*)at);  // (never faults) the write then misses no cache
      pieces_.push_back(iovec{(void*)at, 1});
      if (pieces_.size() == kPieces) send();
    }
  }

  void send() {
    if (pieces_.empty() || !ok_) return;
    ssize_t n;
    do n = writev(fd_[1], pieces_.data(), (int)pieces_.size());
    while (n < 0 && errno == EINTR);
    ok_ = n == (ssize_t)pieces_.size();
    if (!ok_) error_ = n < 0 ? errno : EFAULT;
    char sink[kPieces];
    while (n > 0) {
      const ssize_t got = read(fd_[0], sink, sizeof sink);
      if (got <= 0 && errno != EINTR) break;
      if (got > 0) n -= got;
    }
    pieces_.clear();
  }

  int fd_[2] = {-1, -1};
  uintptr_t page_ = 0, last_ = 0;  // last_: 1 + the page looked at last
  std::vector<iovec> pieces_;
  bool ok_ = true;
  int error_ = 0;
};

}  // namespace mg
