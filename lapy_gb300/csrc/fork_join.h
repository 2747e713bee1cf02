// Work begun on several streams and joined to the caller's (host logic only).
#pragma once

namespace lapy {

// begin(i) starts piece i; join(i) makes the caller wait for what piece i
// started.  Pieces are begun in order until one fails, and every piece that was
// begun is joined, the failed one too: it may have started a part of its work,
// and memory it uses goes back to the caller when this returns.  The first
// status that is not zero is returned.
template <class Begin, class Join>
int fork_join(int n, Begin begin, Join join) {
  int status = 0, begun = 0;
  while (begun < n && status == 0) status = begin(begun++);
  for (int i = 0; i < begun; ++i) {
    const int s = join(i);
    if (status == 0) status = s;
  }
  return status;
}

}  // namespace lapy
