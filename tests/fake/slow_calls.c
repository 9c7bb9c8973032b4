/* Stand-ins for the library's entry points that the native calls bind: nothing needs scratch, and every call takes its time, as a
 * launch into a full queue does. */
#include <stddef.h>
#include <unistd.h>

int needs_none(const void* params, size_t* bytes) {
  (void)params;
  *bytes = 0;
  return 0;
}

int slow(void) {
  usleep(300000);
  return 0;
}
