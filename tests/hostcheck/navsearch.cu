// navsearch.cu -- test infrastructure: what the tests of the navigator's searches call on
// the host, in one library.
#include "cellgrids.cu"
#include "refinenav.cu"
#include "widesearch.cu"
